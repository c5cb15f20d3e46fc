"""Edges of the device SHT kernels: ring lengths with and without a plain power-of-two
transform, rings shorter than a CTA, m far beyond the ring length, the direct sums of large
nside; Legendre stages over ring sets that are not mirror symmetric, odd, single or larger
than one CTA, and m whose lambda_mm underflows.

Tolerances as the engine's existing tests against the same FP64 oracle: 1e-12 of the largest
value (ring transforms and Legendre sums are O(1e-14) sums of that size)."""

import numpy as np
import pytest
import torch

from jfli_b200 import sht
from jfli_b200._lib import call, stream_ptr
from oracle import sht as osht

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda")


@pytest.mark.parametrize("nside,lmax", [(1, 0), (1, 50), (2, 7), (3, 400), (6, 20), (48, 150), (100, 301), (65, 10),
                                        (1025, 3)])
def test_ring_transforms(nside, lmax):
    rng = np.random.default_rng(nside)
    m = rng.standard_normal(12 * nside * nside)
    nr = 4 * nside - 1
    F = torch.empty(nr, lmax + 1, dtype=torch.complex128, device="cuda")
    md = dev(m)
    call("jfli_sht_ring_analysis", stream_ptr(), md.data_ptr(), nside, lmax, F.data_ptr())
    ref = osht._ring_ffts(m, nside, lmax)
    assert np.abs(F.cpu().numpy() - ref).max() < 1e-12 * np.abs(ref).max()
    G = rng.standard_normal((nr, lmax + 1)) + 1j * rng.standard_normal((nr, lmax + 1))
    Gd = dev(G)
    out = torch.empty(12 * nside * nside, dtype=torch.float64, device="cuda")
    call("jfli_sht_ring_synthesis", stream_ptr(), Gd.data_ptr(), nside, lmax, out.data_ptr())
    back = osht._ring_synth(G, nside, lmax)
    assert np.abs(out.cpu().numpy() - back).max() < 1e-12 * np.abs(back).max()


def rings(kind, n, rng):
    if kind == "mirror":
        z = np.sort(rng.uniform(0.0, 0.9999, n // 2))[::-1]
        return np.concatenate([z, [0.0] if n % 2 else [], -z[::-1]])
    return rng.uniform(-0.9999, 0.9999, n)


@pytest.mark.parametrize("kind,nrings,lmax", [("any", 1, 5), ("any", 2, 0), ("any", 37, 64), ("mirror", 36, 33),
                                              ("mirror", 65, 700), ("any", 300, 40), ("any", 5000, 6),
                                              ("mirror", 4099, 9), ("mirror", 2048, 2)])
def test_legendre_stages(kind, nrings, lmax):
    rng = np.random.default_rng(nrings + lmax)
    z = rings(kind, nrings, rng)
    F = rng.standard_normal((nrings, lmax + 1)) + 1j * rng.standard_normal((nrings, lmax + 1))
    off = sht.packed_offsets(lmax)
    alm = rng.standard_normal(off[-1]) + 1j * rng.standard_normal(off[-1])
    a_ref, g_ref = np.empty(off[-1], complex), np.empty((nrings, lmax + 1), complex)
    for m in range(lmax + 1):
        lam = osht._lambda_m(m, lmax, z, np.sqrt((1.0 - z) * (1.0 + z)))  # (l, ring)
        a_ref[off[m]:off[m + 1]] = 0.25 * lam @ F[:, m]
        g_ref[:, m] = lam.T @ alm[off[m]:off[m + 1]]
    zd, Fd, ad = dev(z), dev(F), dev(alm)
    out = torch.empty(off[-1], dtype=torch.complex128, device="cuda")
    call("jfli_sht_map2alm", stream_ptr(), Fd.data_ptr(), zd.data_ptr(), nrings, lmax, 0.25, out.data_ptr())
    assert np.abs(out.cpu().numpy() - a_ref).max() < 1e-12 * np.abs(a_ref).max()
    G = torch.empty(nrings, lmax + 1, dtype=torch.complex128, device="cuda")
    call("jfli_sht_alm2map", stream_ptr(), ad.data_ptr(), zd.data_ptr(), nrings, lmax, G.data_ptr())
    assert np.abs(G.cpu().numpy() - g_ref).max() < 1e-12 * np.abs(g_ref).max()


def test_nan_stays_in_its_ring_and_reaches_every_multipole():
    nside, lmax = 64, 191
    m = np.random.default_rng(3).standard_normal(12 * nside * nside)
    m[7] = np.nan  # second ring
    md = dev(m)
    F = torch.empty(4 * nside - 1, lmax + 1, dtype=torch.complex128, device="cuda")
    call("jfli_sht_ring_analysis", stream_ptr(), md.data_ptr(), nside, lmax, F.data_ptr())
    bad = torch.isnan(torch.view_as_real(F)).any(-1).any(-1)
    assert bad.nonzero().flatten().tolist() == [1]
    assert torch.isnan(sht.anafast(md, lmax)).all()
