"""Device SHT kernels on both sides of their rules: ring transforms by direct sums or FFTs (short rings,
power-of-two belts and others, few and many coefficients), Legendre stages with two or eight ring
pairs per thread (few and many m).

Tolerance as the engine's existing tests against the same FP64 oracle: 1e-12 of the largest value."""

import numpy as np
import pytest
import torch

from tests import test_sht_edges as edges

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nside,lmax", [(2, 96), (16, 95), (16, 96), (63, 95), (63, 96), (64, 31), (64, 32), (100, 63),
                                        (100, 64), (512, 31), (513, 95), (513, 96)])
def test_ring_transforms(nside, lmax):
    edges.test_ring_transforms(nside, lmax)


@pytest.mark.parametrize("kind,nrings,lmax", [("mirror", 2048, 220), ("mirror", 2048, 221), ("any", 2100, 221),
                                              ("mirror", 4099, 221)])
def test_legendre_stages(kind, nrings, lmax):
    edges.test_legendre_stages(kind, nrings, lmax)
