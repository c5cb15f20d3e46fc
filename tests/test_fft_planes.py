"""The z and y passes of square planes in one kernel: every size, few planes and a batch, transforms
against NumPy in FP64 (2e-6 relative L2, the FFT parity tests' bound for FP32) and, as the
arithmetic is that of the separate passes, bit for bit the potential's forward half against them,
which an oblong mesh of the same rows takes. A cleared input and a subtracted mean."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from jfli_b200 import ops
from oracle import pm as opm
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu

SIZES = [32, 36, 48, 54, 64, 72, 96, 108, 128, 144]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("nx, batch", [(6, 1), (4, 3)])
def test_transforms(n, nx, batch):
    x = np.random.default_rng(n).standard_normal((batch, nx, n, n)).astype(np.float32)
    spec = ops.rfft3d(torch.as_tensor(x, device="cuda"))
    ref = np.fft.rfftn(x.astype(np.float64), axes=(1, 2, 3))
    assert rel_l2(spec.cpu().numpy(), ref) < 2e-6
    back = ops.irfft3d(torch.as_tensor(ref.astype(np.complex64), device="cuda"), n)
    assert rel_l2(back.cpu().numpy(), x) < 2e-6


@pytest.mark.parametrize("n", SIZES)
def test_rows_have_the_bits_of_the_separate_passes(n):
    # rows that only differ from 0 in the first plane line: the transform along y of a row at y = 0 is
    # the row itself at every ky, so both meshes give the z pass's bits
    row = torch.randn(6, 1, n, device="cuda")
    square = torch.zeros(6, n, n, device="cuda")
    oblong = torch.zeros(6, 2 * n if n < 128 else n // 2, n, device="cuda")
    square[:, :1], oblong[:, :1] = row, row
    a, b = ops.rfft3d(square), ops.rfft3d(oblong)
    assert torch.equal(a[:, 0], b[:, 0])


@pytest.mark.parametrize("n", SIZES)
def test_cleared_density(n):
    rho = 1.0 + 0.3 * np.random.default_rng(n).standard_normal((6, n, n))
    t = torch.as_tensor(rho.astype(np.float32), device="cuda")
    pot = torch.empty_like(t)
    ops.poisson_force(t, 1.0, pot=pot, clear=True)
    assert not t.any()
    assert rel_l2(pot.cpu().numpy(), opm.potential_real(rho.astype(np.float32).astype(np.float64))) < 1e-5
