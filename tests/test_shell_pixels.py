"""Bilinear shell painting at the directions and map sizes where its table lookups and small
angles can go wrong: pole caps and the poles themselves, the axes and diagonals (ring starts,
the cap / belt border), maps from one base pixel row (large angles) to fine ones, overlapping
shells, batches.

Tolerance: a deposit is one FP32 rounding of an FP64 weight (6e-8), a pixel sums at most a few
thousand of them in FP32: 1e-5 of the map's largest value."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from jfli_b200 import ops
from oracle import healpix as oh

pytestmark = pytest.mark.gpu


def directions(rng, n):
    v = rng.standard_normal((n, 3))
    v[: n // 4] *= [1e-3, 1e-3, 1.0]  # near the poles
    v[n // 4 : n // 4 + 200, 2] = np.sqrt((v[n // 4 : n // 4 + 200, :2] ** 2).sum(-1) * 0.8)  # z = 2/3
    s = [[a, b, c] for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1) if (a, b, c) != (0, 0, 0)]
    v[-len(s):] = s
    return v / np.linalg.norm(v, axis=1, keepdims=True)


@pytest.mark.parametrize("nside", [1, 2, 3, 8, 40, 64, 100, 1024])
def test_bilinear_pixels(nside):
    n, box, obs = 16, 64.0, (32.0, 32.0, 32.0)
    rng = np.random.default_rng(nside)
    v = directions(rng, n**3) * rng.uniform(4.0, 28.0, (n**3, 1))
    v[-26:] = np.sign(v[-26:]) * 8.0 * (np.abs(v[-26:]) > 1e-9)  # exactly on the axes and diagonals
    pos = ((v + 32.0) * (n / box)).astype(np.float32).reshape(n, n, n, 3)
    t = torch.as_tensor(pos, device="cuda")
    x = pos.astype(np.float64) * (box / n)
    rmin, rmax = np.array([3.0, 10.0, 12.0]), np.array([11.0, 20.0, 40.0])  # overlapping
    out = ops.healpix_paint_shells(t, nside, (box,) * 3, obs, rmin, rmax, [1.0, 2.0, 0.5], absolute=True).cpu().numpy()
    for s, scale in enumerate((1.0, 2.0, 0.5)):
        ref = oh.paint_shell(x, obs, rmin[s], rmax[s], nside) * scale
        assert np.abs(out[s] - ref).max() <= 1e-5 * ref.max()
    two = torch.stack([t, t.flip(0)])
    one = ops.healpix_paint(two, nside, (box,) * 3, obs, -1.0, 25.0, absolute=True).cpu().numpy()
    for b in range(2):
        ref = oh.paint_shell(x, obs, -1.0, 25.0, nside)
        assert np.abs(one[b] - ref).max() <= 1e-5 * ref.max()


def test_shell_bounds_are_exact():
    """Particles whose distance equals an edge bit for bit: outside at rmin, inside at rmax."""
    n, box = 4, 4.0
    pos = np.zeros((n, n, n, 3), np.float32)
    r = np.float32(1.2345678) * np.arange(1, n**3 + 1, dtype=np.float32)
    pos[..., 0] = r.reshape(n, n, n)
    rd = r.astype(np.float64)
    t = torch.as_tensor(pos, device="cuda")
    out = ops.healpix_paint_shells(t, 4, (box,) * 3, (0.0, 0.0, 0.0), rd[:-1], rd[1:], np.ones(n**3 - 1),
                                   absolute=True).sum(1).cpu().numpy()
    np.testing.assert_allclose(out, 1.0, rtol=1e-6)
