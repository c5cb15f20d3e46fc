"""Bilinear shell painting of particles without a direction: one exactly at the observer (a shell
with a negative inner radius takes it), one at an infinite distance (a shell without an outer
radius takes it). Both go where the clamped angles put them: the south pole, and for an
infinity along one axis that axis.

Tolerance: single deposits of FP64 weights rounded to FP32 (6e-8), beside at most a handful of
neighbours: 1e-6."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from jfli_b200 import ops
from oracle import healpix as oh

pytestmark = pytest.mark.gpu


def at_direction(nside, theta, phi):
    pix, w = oh.get_interp_weights(nside, np.array([theta]), np.array([phi]))
    m = np.zeros(12 * nside * nside)
    np.add.at(m, np.asarray(pix).reshape(-1), np.asarray(w).reshape(-1))
    return m


@pytest.mark.parametrize("nside", [1, 2, 16, 100, 1024])
def test_particle_at_the_observer(nside):
    n, box, obs = 4, 4.0, (2.0, 2.0, 2.0)  # an undisplaced lattice: particle (2, 2, 2) is the observer
    x = torch.zeros(n, n, n, 3, device="cuda")
    lattice = np.stack(np.meshgrid(*[np.arange(n, dtype=np.float64)] * 3, indexing="ij"), -1)
    south = at_direction(nside, np.pi, 0.0)
    rmin, rmax = [-1.0, -1.0, -0.5], [0.5, 1.2, 0.0]  # overlapping: the general shell search
    out = ops.healpix_paint_shells(x, nside, (box,) * 3, obs, rmin, rmax, [1.0, 2.0, 4.0]).cpu().numpy()
    around = oh.paint_shell(lattice, obs, 0.5, 1.2, nside)
    for m, ref in zip(out, (south, 2.0 * (south + around), 4.0 * south)):
        assert np.abs(m - ref).max() <= 1e-6 * ref.max()
    one = ops.healpix_paint(x, nside, (box,) * 3, obs, -1.0, 0.5).cpu().numpy()
    assert np.abs(one - south).max() <= 1e-6
    tiled = ops.healpix_paint_tiled(x, nside, (box,) * 3, obs, -1.0, 0.5, np.eye(3)[None], np.zeros((1, 3)))
    assert np.abs(tiled.cpu().numpy() - south).max() <= 1e-6


@pytest.mark.parametrize("nside", [2, 64])
@pytest.mark.parametrize("axis, sign, theta, phi", [(0, 1, np.pi / 2, 0.0), (1, 1, np.pi / 2, np.pi / 2),
                                                     (0, -1, np.pi / 2, np.pi)])
def test_particle_at_infinity(nside, axis, sign, theta, phi):
    x = torch.full((2, 2, 2, 3), 1.0, device="cuda")
    x[0, 0, 0, axis] = sign * float("inf")
    obs = (0.0, 1.0, 1.0) if axis == 0 else (1.0, 0.0, 1.0)  # the others at distance 1
    out = ops.healpix_paint(x, nside, (2.0,) * 3, obs, 5.0, float("inf"), absolute=True).cpu().numpy()
    assert np.abs(out - at_direction(nside, theta, phi)).max() <= 1e-6
