"""Transforms of several maps in one launch against the same maps one at a time: the pieces a
batch is cut into, maps that are not finite beside ones that are, and the switch of the pairs per
thread between one map of nside 256 and two. FP64 sums in another order: 1e-12 of the norm."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from jfli_b200 import sht
from jfli_b200.power import angular_cl_spherical, angular_cls_spherical

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nside, lmax, count, together", [(1, 2, 3, 3), (8, 23, 5, 2), (16, 40, 3, 1), (64, 130, 4, 4),
                                                          (256, 300, 2, 2)])
def test_maps_together_match_maps_alone(monkeypatch, nside, lmax, count, together):
    monkeypatch.setattr(sht, "_BATCH_BYTES", together * 16 * (4 * nside - 1) * (lmax + 1))
    m = torch.as_tensor(np.random.default_rng(nside).standard_normal((count, 12 * nside * nside)), device="cuda")
    alms = sht.maps2alm(m, lmax)
    assert len(alms) == count
    for a, row in zip(alms, m):
        b = sht.map2alm(row, lmax)
        assert float((a - b).abs().norm() / b.abs().norm()) < 1e-12
    ell, cls = angular_cls_spherical(m, lmax=lmax)
    assert cls.shape == (count, lmax + 1) and ell.numel() == lmax + 1
    one = angular_cl_spherical(m[-1], lmax=lmax)[1]
    assert float((cls[-1] - one).norm() / one.norm()) < 1e-12


def test_a_map_that_is_not_finite_stays_alone():
    nside, lmax = 8, 20
    m = torch.as_tensor(np.random.default_rng(3).standard_normal((3, 12 * nside * nside)), device="cuda")
    ref = sht.maps2alm(m, lmax)
    m[1, 100] = float("nan")
    got = sht.maps2alm(m, lmax)
    assert torch.isnan(got[1].abs()).any()
    assert torch.equal(got[0], ref[0]) and torch.equal(got[2], ref[2])
