"""The kernels that take a small square plane through its z and y transforms at once, bit for bit against
the separate passes. A mesh [8][n][n] whose only plane of data is x = 0 goes through them and a
transform along x that copies; a mesh [n][8][n] whose only data is at y = 0 goes through the separate
z pass, a transform along y that copies, and along x the column pass that the y transform of the
plane restates. The inverse the same way around. Copies are exact: the other terms are zeros."""

from __future__ import annotations

import pytest
import torch

from jfli_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [32, 36, 48, 54, 64, 72, 96, 108, 128, 144])
def test_planes_have_the_bits_of_the_separate_passes(n):
    g = torch.Generator(device="cuda").manual_seed(n)
    data = torch.randn(n, n, generator=g, device="cuda")
    plane, apart = torch.zeros(8, n, n, device="cuda"), torch.zeros(n, 8, n, device="cuda")
    plane[0], apart[:, 0] = data, data
    a, b = ops.rfft3d(plane)[0], ops.rfft3d(apart)[:, 0]
    assert float(a.abs().max()) > 1.0 and torch.equal(a, b)
    spec = torch.randn(n, n // 2 + 1, 2, generator=g, device="cuda")
    spec = torch.view_as_complex(spec)
    plane, apart = (torch.zeros(*s, n // 2 + 1, dtype=torch.complex64, device="cuda") for s in ((8, n), (n, 8)))
    plane[0], apart[:, 0] = spec, spec
    a, b = ops.irfft3d(plane, n)[0], ops.irfft3d(apart, n)[:, 0]
    assert float(a.abs().max()) > 0.0 and torch.equal(a, b)
