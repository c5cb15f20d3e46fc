"""The CIC paint's forms: pairs of cells by vector atomics (rows of whole groups of
four cells, mesh 16-byte aligned), the segment walk of large meshes, and the general kernel. Large
meshes against sums in torch, small ones against the oracle.

Tolerance as the paint's parity test: 1e-6 relative L2 (FP32 weights, atomics in any order)."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from jfli_b200 import ops
from oracle import pm as opm
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


def positions(lead, shape, kind):
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    if kind == "uniform":  # absolute, some of them outside the box
        n = torch.tensor([float(v) for v in shape], device="cuda")
        return (torch.rand(*lead, *shape, 3, generator=g, device="cuda") * 1.2 - 0.1) * n
    if kind == "apart":
        return torch.randn(*lead, *shape, 3, generator=g, device="cuda") * 1.5
    x = [torch.arange(n, device="cuda") * (6.2831853 / n) for n in shape]  # neighbours move together
    wave = torch.sin(x[0])[:, None, None] + torch.cos(x[1])[:, None] + torch.sin(x[2])
    return torch.stack([1.3 * wave, 0.7 - wave, 0.4 + 0.9 * wave], -1).expand(*lead, *shape, 3).contiguous()


def unaligned(shape):
    return torch.zeros(int(np.prod(shape)) + 1, device="cuda")[1:].view(shape)


def in_torch(pos, absolute, weights, weight):
    """The paint in FP64 from single-precision corner weights, formed as the kernel forms them."""
    shape = pos.shape[-4:-1]
    out = torch.zeros(pos.shape[:-1], device="cuda", dtype=torch.float64)
    f = torch.floor(pos)
    w1 = pos - f
    w = [(1.0 - w1[..., a], w1[..., a]) for a in range(3)]
    at = []
    for a in range(3):
        i = f[..., a].long()
        if not absolute:
            i = i + torch.arange(shape[a], device="cuda").view([-1 if c == a else 1 for c in range(3)])
        i = torch.remainder(i, shape[a])
        at.append((i, torch.remainder(i + 1, shape[a])))
    scale = weight if weights is None else weights * weight
    cells = out.view(-1, shape[0] * shape[1] * shape[2])
    for cx in range(2):
        for cy in range(2):
            for cz in range(2):
                cell = (at[0][cx] * shape[1] + at[1][cy]) * shape[2] + at[2][cz]
                v = w[0][cx] * scale * w[1][cy] * w[2][cz]
                cells.scatter_add_(1, cell.reshape(cells.shape[0], -1), v.double().reshape(cells.shape[0], -1))
    return out


@pytest.mark.parametrize("lead, shape", [((), (200, 180, 176)), ((), (257, 101, 252)), ((2,), (150, 145, 148)),
                                         ((), (1, 2048, 3072)), ((), (64, 512, 192)),
                                         ((), (200, 180, 175))])
@pytest.mark.parametrize("kind", ["uniform", "apart", "together"])
def test_large_meshes(lead, shape, kind):
    pos = positions(lead, shape, kind)
    w = torch.rand(pos.shape[:-1], generator=torch.Generator(device="cuda").manual_seed(1), device="cuda") + 0.5
    for weights, weight in ((None, 1.0), (w, 0.5)):
        want = in_torch(pos, kind == "uniform", weights, weight)
        for mesh in (None, unaligned(pos.shape[:-1])):
            got = ops.paint_cic(pos, absolute=kind == "uniform", weights=weights, weight=weight, out=mesh).double()
            assert float((got - want).norm() / want.norm()) < 1e-6


@pytest.mark.parametrize("shape", [(1, 1, 4), (2, 1, 8), (9, 5, 12), (3, 4, 20), (7, 9, 28), (16, 16, 16), (5, 6, 64)])
@pytest.mark.parametrize("kind", ["uniform", "apart", "together"])
def test_small_meshes(shape, kind):
    pos = positions((2,), shape, kind)
    for mesh in (None, unaligned(pos.shape[:-1])):
        got = ops.paint_cic(pos, absolute=kind == "uniform", out=mesh)
        for b in range(2):
            ref = opm.cic_paint(pos[b].cpu().numpy().astype(np.float64), absolute=kind == "uniform")
            assert rel_l2(got[b].cpu().numpy(), ref) < 1e-6
