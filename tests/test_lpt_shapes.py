"""LPT over mesh shapes at the edges of its kernels: the smallest axes, partial last warps (4
cells per thread), z lengths that take the scalar kernels (nz % 4 != 0, nz < 8), batches and
buffers that are not 16-byte aligned. Tolerance as the LPT parity tests: 1e-5 relative L2 of
FP32 kernels against the FP64 oracle."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from jfli_b200 import ops
from oracle import pm as opm
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu

C = (0.13, -0.0071, 0.056, 0.11)


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("shape", [(4, 4, 8), (6, 4, 12), (16, 24, 36), (8, 9, 6), (12, 8, 4), (4, 18, 54), (64, 32, 96)])
def test_lpt_matches_oracle(shape, order):
    ic = (0.7 * np.random.default_rng(sum(shape)).standard_normal((2, *shape))).astype(np.float32)
    t = torch.as_tensor(ic, device="cuda")
    dx, p = ops.lpt(t, order, *C)
    for b in range(2):
        rdx, rp = opm.lpt(ic[b].astype(np.float64), *C, order=order)
        assert rel_l2(dx[b].cpu().numpy(), rdx) < 1e-5
        assert rel_l2(p[b].cpu().numpy(), rp) < 1e-5


@pytest.mark.parametrize("order", [1, 2])
def test_unaligned_output(order):
    """dx and p one float off a 16-byte boundary: the scalar kernels, the same field."""
    shape = (16, 12, 24)
    ic = torch.randn(shape, generator=torch.Generator().manual_seed(1)).cuda()
    n = ic.numel() * 3
    dx = torch.empty(n + 4, device="cuda")[1:n + 1].view(*shape, 3)
    p = torch.empty(n + 4, device="cuda")[1:n + 1].view(*shape, 3)
    ops.lpt(ic, order, *C, dx=dx, p=p)
    rdx, rp = ops.lpt(ic, order, *C)
    assert rel_l2(dx.cpu().numpy(), rdx.cpu().numpy()) < 1e-6
    assert rel_l2(p.cpu().numpy(), rp.cpu().numpy()) < 1e-6
