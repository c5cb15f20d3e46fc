"""Binned spectrum kernels at the edges of their ranges: odd and tiny x axes, tiles that cross
rows of the spectrum, lengths with and without a register transform, histograms of many and
of one column, batches.

Tolerances: mode counts and mean |k| are sums of the same FP32 |k| in FP64 (1e-12 relative,
exact for the counts). Power: FP32 transforms are within 2e-6 relative L2 of FP64 over the
field (the parity tests' bound), so a bin's sum of squares, which holds at least one mode
pair of comparable power, is within 2e-5 relative of the FP64 sum.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from jfli_b200 import ops
from jfli_b200.power import power_poles
from oracle import pm as opm

pytestmark = pytest.mark.gpu


def grid_sums(x, box, edges):
    """(power, count, |k|) per digitize bin over the full grid, FP64, |k| in FP32."""
    shape = x.shape
    f = np.fft.fftn(x.astype(np.float64))
    kv = []
    for a, (n, length) in enumerate(zip(shape, box)):
        i = np.rint(np.fft.fftfreq(n) * n).astype(np.float32)
        sh = [1, 1, 1]
        sh[a] = n
        c = np.float32(2.0 * np.pi / float(np.float32(length)))  # the C-ABI takes FP32 box sides
        kv.append((c * i).reshape(sh))
    k = np.sqrt((kv[0] * kv[0] + kv[1] * kv[1] + kv[2] * kv[2]).astype(np.float32))
    k = np.broadcast_to(k, shape).reshape(-1)
    b = np.digitize(k, edges)
    n = edges.size + 1
    p = (np.abs(f) ** 2).reshape(-1) / x.size
    return np.stack([np.bincount(b, p, n), np.bincount(b, minlength=n), np.bincount(b, k.astype(np.float64), n)])


@pytest.mark.parametrize("shape,nedges,batch", [
    ((27, 16, 32), 7, 2), ((2, 6, 4), 3, 1), ((3, 4, 8), 1, 1), ((64, 48, 18), 40, 1), ((72, 9, 36), 2048, 1),
    ((512, 4, 6), 33, 1), ((1024, 3, 4), 300, 1), ((128, 64, 64), 33, 3), ((81, 2, 4), 12, 1), ((256, 24, 16), 700, 1),
])
def test_power_sums_match_full_grid(shape, nedges, batch):
    rng = np.random.default_rng(sum(shape) + nedges)
    x = (1.0 + rng.standard_normal((batch, *shape))).astype(np.float32)
    box = tuple(3.1 * n for n in shape)
    edges = np.linspace(0.013, 1.7, nedges).astype(np.float32)
    got = ops.power_sums(torch.as_tensor(x, device="cuda"), torch.as_tensor(edges, device="cuda"), box).cpu().numpy()
    for b in range(batch):
        ref = grid_sums(x[b], box, edges)
        np.testing.assert_array_equal(got[b, 1], ref[1])
        np.testing.assert_allclose(got[b, 2], ref[2], rtol=1e-12)
        np.testing.assert_allclose(got[b, 0], ref[0], rtol=2e-5)


@pytest.mark.parametrize("shape,poles,cross,nedges", [
    ((32, 24, 36), (0, 1, 2, 3, 4, 5, 6, 7), True, 9), ((27, 18, 16), (3,), False, 5), ((16, 16, 16), (0, 2, 4), True, 60),
    ((6, 81, 8), (1, 2), True, 4), ((64, 64, 12), (16, 0), False, 12), ((2, 4, 64), (2, 1, 0), True, 500),
])
def test_power_poles_match_oracle(shape, poles, cross, nedges):
    """Every multipole count, odd and Nyquist-plane modes, an oblique line of sight. FP32 mu and
    L_l weights (up to (2l + 1) |L_l| rounding, 2e-6 at l = 16) on FP32 transforms: 1e-4 of the
    bin's monopole, the parity tests' bound."""
    rng = np.random.default_rng(sum(shape))
    a = rng.standard_normal(shape).astype(np.float32)
    b = (0.5 * a + rng.standard_normal(shape)).astype(np.float32) if cross else None
    box = tuple(2.7 * n for n in shape)
    edges = np.linspace(0.037, 1.9, nedges)
    los = (0.3, -0.5, 0.8)
    k, pk = power_poles(torch.as_tensor(a, device="cuda"), None if b is None else torch.as_tensor(b, device="cuda"),
                           box, edges, poles, los)
    kr, pr = opm.power_poles(a, b, box, edges, poles, los)
    scale = np.abs(opm.power_poles(a, None, box, edges, 0)[1])
    if cross:
        scale = np.maximum(scale, np.abs(opm.power_poles(b, None, box, edges, 0)[1]))
    np.testing.assert_allclose(k.cpu().numpy(), kr, rtol=1e-6)
    assert np.all(np.abs(np.atleast_2d(pk.cpu().numpy()) - np.atleast_2d(pr)) <= 1e-4 * scale)
