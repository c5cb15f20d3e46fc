"""CIC paint and force readout over mesh shapes at the edges of the segment walk: rows that do
and do not fill their segments, a number of y rows that is not a multiple of a CTA's eight, the
smallest axes, batches, weights, absolute positions outside the box.

Tolerances as the parity tests: paint 1e-6 relative L2 (FP32 weights, atomics in any order),
forces 1e-5."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from jfli_b200 import ops
from jfli_b200._lib import call, ptr, query, stream_ptr
from oracle import pm as opm
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.as_tensor(np.ascontiguousarray(a, np.float32), device="cuda")


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 3, 23), (5, 1, 24), (17, 9, 31), (3, 7, 32), (16, 8, 33), (33, 10, 48),
                                   (4, 5, 65), (7, 16, 96), (2, 2, 200), (40, 24, 56)])
@pytest.mark.parametrize("sigma", [0.3, 5.0])
def test_paint(shape, sigma):
    rng = np.random.default_rng(sum(shape))
    disp = rng.normal(0, sigma, (2, *shape, 3)).astype(np.float32)
    disp += np.float32(0.4 * sigma)  # neighbours that move together, so that the merges take place
    w = rng.uniform(0.5, 2.0, (2, *shape)).astype(np.float32)
    rel = ops.paint_cic(dev(disp), weights=dev(w), weight=0.5).cpu().numpy()
    grid = np.stack(np.meshgrid(*[np.arange(n) for n in shape], indexing="ij"), -1)
    pos = (disp + grid).astype(np.float32)
    absolute = ops.paint_cic(dev(pos), absolute=True).cpu().numpy()
    for b in range(2):
        assert rel_l2(rel[b], opm.cic_paint(disp[b].astype(np.float64), weight=0.5 * w[b].astype(np.float64))) < 1e-6
        assert rel_l2(absolute[b], opm.cic_paint(pos[b].astype(np.float64), absolute=True)) < 1e-6


@pytest.mark.parametrize("shape", [(8, 9, 16), (12, 18, 54), (16, 8, 32), (9, 4, 96), (32, 24, 36)])
@pytest.mark.parametrize("absolute", [False, True])
def test_forces_with_and_without_force_mesh(shape, absolute):
    rng = np.random.default_rng(sum(shape))
    pos = rng.normal(0, 1.5, (*shape, 3)).astype(np.float32)
    grid = np.stack(np.meshgrid(*[np.arange(n, dtype=np.float32) for n in shape], indexing="ij"), -1)
    if absolute:
        pos += grid
    t = dev(pos)
    ref = 1.5 * opm.pm_forces(pos.astype(np.float64) - (grid if absolute else 0.0))  # the oracle takes displacements
    full = ops.pm_forces(t, absolute=absolute, scale=1.5)
    assert rel_l2(full.cpu().numpy(), ref) < 1e-5
    nb = query("jfli_pm_step_workspace_bytes", *shape, 1)  # no room for the force mesh
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    out = torch.empty_like(t)
    call("jfli_pm_forces", stream_ptr(), ptr(t), int(absolute), 1.5, ptr(out), ptr(ws), nb, *shape, 1)
    assert rel_l2(out.cpu().numpy(), ref) < 1e-5
