"""Register passes of the mixed lengths 2^a 3^b: every length on each axis once, with partial
last tiles and rows, odd spectra and batches. Transforms against NumPy in FP64 (2e-6 relative
L2, the FFT parity tests' bound for FP32), potentials and initial conditions against the FP64
oracle (1e-5)."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from jfli_b200 import ops
from oracle import pm as opm
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu

LENGTHS = [18, 27, 36, 54, 72, 81, 108, 144, 162, 216, 243, 288, 324, 432, 486, 576, 648]


@pytest.mark.parametrize("n", LENGTHS)
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_transform_along_each_axis(n, axis):
    shape = [6, 9, 8]
    shape[axis] = 2 * n if axis == 2 else n
    x = np.random.default_rng(n).standard_normal((2, *shape)).astype(np.float32)
    spec = ops.rfft3d(torch.as_tensor(x, device="cuda"))
    ref = np.fft.rfftn(x.astype(np.float64), axes=(1, 2, 3))
    assert rel_l2(spec.cpu().numpy(), ref) < 2e-6
    back = ops.irfft3d(torch.as_tensor(ref.astype(np.complex64), device="cuda"), shape[2])
    assert rel_l2(back.cpu().numpy(), x) < 2e-6


@pytest.mark.parametrize("n", LENGTHS)
def test_poisson_and_initial_conditions(n):
    shape = (n, 6, 18)
    rng = np.random.default_rng(n)
    rho = 1.0 + 0.3 * rng.standard_normal(shape)
    pot = ops.poisson_potential(torch.as_tensor(rho.astype(np.float32), device="cuda"), 1.0).cpu().numpy()
    assert rel_l2(pot, opm.potential_real(rho.astype(np.float32).astype(np.float64))) < 1e-5
    k = np.logspace(-3, 1, 64)
    pk = 1e4 * k / (1.0 + (k / 0.02) ** 2) ** 1.2
    box = tuple(3.0 * v for v in shape)
    noise = rng.standard_normal(shape).astype(np.float32)
    dev = lambda a: torch.as_tensor(np.asarray(a, np.float32), device="cuda")
    ic = ops.ic_filter(dev(noise), dev(k), dev(pk), box).cpu().numpy()
    assert rel_l2(ic, opm.ic_filter(noise.astype(np.float64), box, k, pk)) < 1e-5
