"""Performance cases of the framework: what a user has it do, from single forces to whole
forward models, over the sizes of its configurations, tests and benchmark.

Each case names a `kind`:

* forces    the PM force of a particle set (`ops.pm_forces`)
* forward   white noise -> initial conditions -> LPT -> N-body -> density and P(k)
* gradient  the gradient of a log-P(k) loss with respect to the white noise, through the
            reversible N-body loop
* initial   initial conditions and second-order LPT from given P(k) and growth factors
* power     the binned power spectrum of a density
* poles     multipoles of an auto or cross spectrum
* shells    HEALPix shells of one particle set (`ParticleField.paint_spherical`)
* tiled     one HEALPix shell beyond the box, from 27 replicas drifted to the light cone
* cl        angular power spectra of HEALPix maps

Spectra are returned in FP32, the type the reference returns them in and the precision of
the fields they are taken from.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import jfli_b200 as jf
from jfli_b200 import ops
from jfli_b200.painting import paint_shell_tiled
from jfli_b200.pm.interp import get_all_47_symmetries, tile_shifts

T0, T1 = 0.1, 1.0
LPT2_FACTORS = (0.13, -0.0071, 0.056, 0.11)  # displacement and momentum factors of both orders near a = 0.1


# ------------------------------------------------------------------------------- the cases
def listed():
    return [
        # one force call on the smallest configuration: launches and latency
        dict(name="forces 64", kind="forces", nx=64, ny=64, nz=64, absolute=False, rms=2.0),
        # an ordinary force call on a mesh that is no power of two, positions in absolute units
        dict(name="forces 216x144x324", kind="forces", nx=216, ny=144, nz=324, absolute=True, rms=4.0),
        # the plain 64^3 configuration: 1LPT to a = 0.1, 10 steps
        dict(name="forward 64", kind="forward", n=64, box=256.0, order=1, steps=10),
        # the headline 256^3 configuration: 2LPT to a = 0.1, 40 steps
        dict(name="forward 256", kind="forward", n=256, box=1000.0, order=2, steps=40),
        # the differentiation configuration: 128^3, 20 reversible steps
        dict(name="gradient 128", kind="gradient", n=128, box=500.0, steps=20),
        # initial conditions and 2LPT of a large run
        dict(name="initial 384", kind="initial", nx=384, ny=384, nz=384),
        # P(k) of a large density
        dict(name="power 512", kind="power", nx=512, ny=512, nz=512, cross=False),
        # redshift-space style multipoles of a cross spectrum
        dict(name="poles 256", kind="poles", nx=256, ny=256, nz=256, cross=True, lmax=4),
        # the 16 shells of one 256^3 particle set, bilinear
        dict(name="shells 256", kind="shells", n=256, nside=256, shells=16, scheme="bilinear"),
        # one far shell of a light cone, 27 replicas with the drift
        dict(name="tiled 192", kind="tiled", n=192, nside=512, inner=0.75, width=0.1),
        # C_ell of the four shells of the 256^3 configuration
        dict(name="cl 256", kind="cl", nside=256, lmax=767, maps=4),
        # C_ell of a high-resolution convergence map
        dict(name="cl 1024", kind="cl", nside=1024, lmax=3000, maps=1),
    ]


def _smooth(lo, hi):
    """Even sizes 2^a 3^b in [lo, hi]: the FFT meshes the framework takes."""
    return sorted(2**a * 3**b for a in range(1, 13) for b in range(8) if lo <= 2**a * 3**b <= hi)


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _size(rng, lo, hi):
    """A mesh size spread over the logarithm of the range."""
    x = _log(rng, lo, hi)
    return min(_smooth(lo, hi), key=lambda n: abs(math.log(n / x)))


def _mesh(rng, lo, hi, cells):
    while True:
        nx, ny, nz = (_size(rng, lo, hi) for _ in range(3))
        if nx * ny * nz <= cells:
            return dict(nx=nx, ny=ny, nz=nz)


def draw(rng):
    kind = rng.choice(["forces", "forward", "gradient", "initial", "power", "poles", "shells", "tiled", "cl"])
    if kind == "forces":
        return dict(kind=kind, **_mesh(rng, 32, 384, 256**3), absolute=rng.random() < 0.3,
                    rms=round(_log(rng, 0.3, 8.0), 2))
    if kind == "forward":
        n = _size(rng, 32, 216)
        return dict(kind=kind, n=n, box=round(n * rng.uniform(2.0, 6.0), 1), order=rng.choice([1, 2]),
                    steps=rng.randint(5, 40))
    if kind == "gradient":
        n = _size(rng, 32, 144)
        return dict(kind=kind, n=n, box=round(n * rng.uniform(3.0, 5.0), 1), steps=rng.randint(5, 20))
    if kind == "initial":
        return dict(kind=kind, **_mesh(rng, 32, 512, 384**3))
    if kind == "power":
        return dict(kind=kind, **_mesh(rng, 32, 768, 400**3), cross=rng.random() < 0.3)
    if kind == "poles":
        return dict(kind=kind, **_mesh(rng, 32, 384, 256**3), cross=rng.random() < 0.5, lmax=rng.choice([2, 4]))
    if kind == "shells":
        return dict(kind=kind, n=rng.randint(40, 256), nside=rng.choice([64, 128, 256, 512]),
                    shells=rng.randint(1, 20), scheme=rng.choice(["bilinear", "bilinear", "ngp"]))
    if kind == "tiled":
        return dict(kind=kind, n=rng.randint(40, 192), nside=rng.choice([128, 256, 512]),
                    inner=round(rng.uniform(0.3, 0.9), 3), width=round(rng.uniform(0.03, 0.1), 3))
    nside = rng.choice([32, 48, 64, 128, 256, 512])
    return dict(kind="cl", nside=nside, lmax=rng.randint(nside, 3 * nside - 1), maps=rng.randint(1, 4))


# ------------------------------------------------------------------------------ the inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _noise(shape, gen):
    return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32)


def _k(shape, dtype=torch.float32):
    """Angular wavenumbers per cell of a half spectrum, one broadcastable array per axis."""
    nx, ny, nz = shape
    f = [torch.fft.fftfreq(nx, device="cuda", dtype=dtype), torch.fft.fftfreq(ny, device="cuda", dtype=dtype),
         torch.fft.rfftfreq(nz, device="cuda", dtype=dtype)]
    return [2.0 * math.pi * f[0][:, None, None], 2.0 * math.pi * f[1][None, :, None],
            2.0 * math.pi * f[2][None, None, :]]


def _linear_field(shape, gen):
    """(half spectrum, k, k^2) of a Gaussian field with a spectrum of the cold dark matter
    shape, rising below and falling above about 0.1 per cell."""
    k = _k(shape)
    k2 = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
    spec = torch.fft.rfftn(_noise(shape, gen)) * (k2**0.25 / (1.0 + k2 / 0.01))
    return spec, k, torch.where(k2 > 0, k2, torch.ones_like(k2))


def _displacements(shape, rms, gen):
    """Zel'dovich displacements (cells) of that field, `rms` cells per component."""
    spec, k, k2 = _linear_field(shape, gen)
    out = torch.empty(*shape, 3, device="cuda", dtype=torch.float32)
    for a in range(3):
        out[..., a] = torch.fft.irfftn(1j * k[a] / k2 * spec, s=shape)
    return (out * (rms / out.std())).contiguous()


def _density(shape, gen):
    """A positive density of mean about 1, lognormal."""
    spec, _, _ = _linear_field(shape, gen)
    d = torch.fft.irfftn(spec, s=shape)
    return torch.exp(d * (0.8 / d.std()) - 0.32)


def _pk_shape(k):
    return 2.0e4 * (k / 0.02) / (1.0 + (k / 0.02) ** 2) ** 1.3


def _shape(case):
    return (case["nx"], case["ny"], case["nz"])


def _kedges(shape, box):
    """Up to 32 bins from half the fundamental to the Nyquist frequency, each with modes."""
    fundamental = 2.0 * math.pi / max(box)
    nyquist = math.pi * min(n / length for n, length in zip(shape, box))
    return np.linspace(0.5 * fundamental, nyquist, min(32, max(shape) // 2) + 1)


def _particles(array, n, box, nside):
    return jf.ParticleField(array=array, mesh_size=(n,) * 3, box_size=(box,) * 3, nside=nside,
                            status=jf.FieldStatus.LPT1, unit=jf.PositionUnit.GRID_RELATIVE)


def _shell_radii(case, box):
    """Centres and widths of equal shells from 0.05 to 0.5 of the box."""
    edges = np.linspace(0.05, 0.5, case["shells"] + 1) * box
    return 0.5 * (edges[1:] + edges[:-1]), np.diff(edges)


def prepare(case, seed):
    gen = _generator(seed)
    kind = case["kind"]
    s = dict(case=case)
    if kind == "forces":
        shape = _shape(case)
        pos = _displacements(shape, case["rms"], gen)
        if case["absolute"]:
            for a, n in enumerate(shape):
                pos[..., a] += torch.arange(n, device="cuda").reshape([-1 if b == a else 1 for b in range(3)])
        s["pos"] = pos
    elif kind in ("forward", "gradient"):
        n = case["n"]
        s["noise"] = _noise((n,) * 3, gen)
        s["cosmo"] = jf.Planck18()
        s["kedges"] = _kedges((n,) * 3, (case["box"],) * 3)
        cls = jf.EfficientDriftDoubleKick if kind == "forward" else jf.ReversibleDoubleKickDrift
        s["solver"] = cls(interp_kernel=jf.NoInterp(painting=jf.PaintingOptions(target="density")))
        if kind == "gradient":
            k = 0.5 * (s["kedges"][1:] + s["kedges"][:-1])
            s["target"] = torch.as_tensor(0.5 * _pk_shape(k), device="cuda")
    elif kind == "initial":
        s["noise"] = _noise(_shape(case), gen)
        k = np.logspace(-4, 1, 128)
        s["ktab"] = torch.as_tensor(k, dtype=torch.float32, device="cuda")
        s["ptab"] = torch.as_tensor(_pk_shape(k), dtype=torch.float32, device="cuda")
    elif kind in ("power", "poles"):
        shape = _shape(case)
        s["box"] = tuple(4.0 * n for n in shape)
        s["kedges"] = _kedges(shape, s["box"])
        s["mesh"] = _density(shape, gen)
        s["mesh2"] = 0.7 * s["mesh"] + 0.3 * _density(shape, gen) if case["cross"] else None
    elif kind == "shells":
        n, box = case["n"], 4.0 * case["n"]
        s["field"] = _particles(_displacements((n,) * 3, 2.0, gen), n, box, case["nside"])
        s["centers"], s["widths"] = _shell_radii(case, box)
    elif kind == "tiled":
        n, box = case["n"], 4.0 * case["n"]
        disp = _displacements((n,) * 3, 2.0, gen)
        s["field"] = _particles(disp, n, box, case["nside"])
        s["vel"] = (0.5 * disp).contiguous()
        s["rotations"] = get_all_47_symmetries()[np.random.default_rng(42).integers(0, 47, size=27)]
        s["shifts"] = tile_shifts((0.5, 0.5, 0.5), (box,) * 3)
        s["r"], s["w"] = (case["inner"] + 0.5 * case["width"]) * box, case["width"] * box
        s["cosmo"] = jf.Planck18()
        s["t"] = float(jf.cosmology.a_of_chi(s["cosmo"], s["r"]))
    else:
        maps = torch.exp(0.5 * _noise((case["maps"], 12 * case["nside"] ** 2), gen))
        maps = maps / maps.mean(dim=1, keepdim=True) - 1.0  # contrast: no monopole above the other multipoles
        s["field"] = jf.SphericalDensity(array=maps, mesh_size=(64,) * 3, box_size=(500.0,) * 3, nside=case["nside"],
                                         status=jf.FieldStatus.LIGHTCONE, unit=jf.DensityUnit.DENSITY)
    return s


# ------------------------------------------------------------------------------- the calls
def _initial_particles(s, noise, order):
    n, box = s["case"]["n"], s["case"]["box"]
    ic = jf.interpolate_initial_conditions(noise, (n,) * 3, (box,) * 3, cosmo=s["cosmo"])
    return jf.lpt(s["cosmo"], ic, ts=T0, order=order)


def _spectrum(mesh, s, mesh2=None, **kw):
    k, pk = jf.power(mesh, mesh2, box_shape=s["box"], kedges=s["kedges"], **kw)
    return k.float(), pk.float()


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "forces":
        return ops.pm_forces(s["pos"], absolute=case["absolute"], scale=0.46)
    if kind == "forward":
        dx, p = _initial_particles(s, s["noise"], case["order"])
        density = jf.nbody(s["cosmo"], dx, p, t0=T0, t1=T1, dt0=(T1 - T0) / case["steps"], solver=s["solver"])
        pk = density.power(kedges=s["kedges"])
        return {"density": density.array, "k": pk.wavenumber.float(), "pk": pk.spectra.float()}
    if kind == "gradient":
        noise = s["noise"].detach().requires_grad_()
        dx, p = _initial_particles(s, noise, 2)
        density = jf.nbody(s["cosmo"], dx, p, t0=T0, t1=T1, dt0=(T1 - T0) / case["steps"], solver=s["solver"],
                           adjoint="reverse")
        pk = density.power(kedges=s["kedges"]).spectra
        loss = torch.sum((torch.log(pk) - torch.log(s["target"])) ** 2)
        (grad,) = torch.autograd.grad(loss, noise)
        return {"loss": loss.detach().float(), "grad": grad}
    if kind == "initial":
        ic = ops.ic_filter(s["noise"], s["ktab"], s["ptab"], tuple(4.0 * n for n in _shape(case)))
        dx, p = ops.lpt(ic, 2, *LPT2_FACTORS)
        return {"ic": ic, "dx": dx, "p": p}
    if kind == "power":
        return _spectrum(s["mesh"], s, s["mesh2"])
    if kind == "poles":
        return _spectrum(s["mesh"], s, s["mesh2"], multipoles=tuple(range(0, case["lmax"] + 1, 2)))
    if kind == "shells":
        return s["field"].paint_spherical(center=s["centers"], density_plane_width=s["widths"],
                                          scheme=case["scheme"]).array
    if kind == "tiled":
        return paint_shell_tiled(s["field"], s["vel"], s["r"], s["w"], s["rotations"], s["shifts"], telephoto=False,
                                 t=s["t"], cosmo=s["cosmo"])
    return s["field"].angular_cl(lmax=case["lmax"]).spectra


# -------------------------------------------------------------------------------- the work
def _fft_flops(cells):
    return 2.5 * cells * math.log2(cells)


def work(case):
    """Bytes and operations of one pass. An N-body step counts 120 bytes per particle (its
    state and the meshes of the force, each read or written once per pass), as the particle
    state of the larger runs does not stay on the chip."""
    kind = case["kind"]
    if kind in ("forward", "gradient", "shells", "tiled"):
        cells = case["n"] ** 3
    elif kind != "cl":
        cells = case["nx"] * case["ny"] * case["nz"]
    if kind == "forces":
        return {"bytes": 24 * cells, "flops": 2 * _fft_flops(cells) + 250 * cells}
    if kind == "forward":
        lpt = 2 * case["order"]
        return {"bytes": (120 * case["steps"] + 100) * cells,
                "flops": (2 * case["steps"] + lpt + 5) * _fft_flops(cells) + 250 * case["steps"] * cells}
    if kind == "gradient":
        return {"bytes": (300 * case["steps"] + 300) * cells,
                "flops": (4 * case["steps"] + 16) * _fft_flops(cells) + 800 * case["steps"] * cells}
    if kind == "initial":
        return {"bytes": 32 * cells, "flops": 6 * _fft_flops(cells) + 120 * cells}
    if kind in ("power", "poles"):
        fields = 2 if case["cross"] else 1
        return {"bytes": 4 * fields * cells, "flops": fields * _fft_flops(cells) + 20 * cells}
    npix = 12 * case["nside"] ** 2
    if kind == "shells":
        return {"bytes": 12 * cells + 4 * npix * case["shells"], "flops": 100 * cells}
    if kind == "tiled":
        return {"bytes": 24 * cells + 4 * npix, "flops": 300 * cells}
    pairs = (case["lmax"] + 1) * (case["lmax"] + 2) / 2
    legendre = pairs * 2 * case["nside"] * 8  # one hemisphere's rings, two parities
    return {"bytes": case["maps"] * (4 * npix + 8 * (case["lmax"] + 1)),
            "flops": case["maps"] * 7 * (legendre + 2.5 * npix * math.log2(4 * case["nside"]))}


# ------------------------------------------------------------------- the same in 64 bits
def _corners(pos, shape, absolute):
    """For the particles' 8 CIC corners: (flat cell index, weight)."""
    lower, frac = [], []
    for a, n in enumerate(shape):
        x = pos[..., a].double()
        f = torch.floor(x)
        i = f.long()
        if not absolute:
            i = i + torch.arange(n, device="cuda").reshape([-1 if b == a else 1 for b in range(3)])
        lower.append(torch.remainder(i, n))
        frac.append(x - f)
    for c in range(8):
        index, weight = 0, 1.0
        for a, n in enumerate(shape):
            up = (c >> a) & 1
            index = index * n + torch.remainder(lower[a] + up, n)
            weight = weight * (frac[a] if up else 1.0 - frac[a])
        yield index.reshape(-1), weight.reshape(-1)


def _paint(pos, shape, absolute=False):
    mesh = torch.zeros(shape[0] * shape[1] * shape[2], device="cuda", dtype=torch.float64)
    for index, weight in _corners(pos, shape, absolute):
        mesh.index_add_(0, index, weight)
    return mesh.reshape(shape)


def _gradient_kernel(k):
    return 1j * (8.0 * torch.sin(k) - torch.sin(2.0 * k)) / 6.0


def _potential(rho):
    """Half spectrum of the inverse Laplacian of a mesh."""
    k = _k(rho.shape, torch.float64)
    k2 = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
    spec = torch.fft.rfftn(rho) * torch.where(k2 > 0, -1.0 / torch.where(k2 > 0, k2, torch.ones_like(k2)),
                                              torch.zeros_like(k2))
    return spec, [_gradient_kernel(v) for v in k]


def _exact_forces(case, s):
    shape = _shape(case)
    spec, g = _potential(_paint(s["pos"], shape, case["absolute"]))
    out = torch.zeros(shape[0] * shape[1] * shape[2], 3, device="cuda", dtype=torch.float64)
    for a in range(3):
        mesh = torch.fft.irfftn(-g[a] * spec, s=shape).reshape(-1)
        for index, weight in _corners(s["pos"], shape, case["absolute"]):
            out[:, a] += mesh[index] * weight
    return 0.46 * out.reshape(*shape, 3)


def _exact_initial(case, s):
    shape = _shape(case)
    k = [v / 4.0 for v in _k(shape, torch.float64)]  # cells of 4 Mpc/h
    kk = torch.sqrt(k[0] ** 2 + k[1] ** 2 + k[2] ** 2)
    xp, fp = s["ktab"].double(), s["ptab"].double()
    i = (torch.searchsorted(xp, kk.contiguous()) - 1).clamp(0, xp.numel() - 2)
    pk = fp[i] + (kk - xp[i]) * (fp[i + 1] - fp[i]) / (xp[i + 1] - xp[i])
    ic = torch.fft.irfftn(torch.fft.rfftn(s["noise"].double()) * torch.sqrt(pk / 64.0), s=shape)
    c1x, c2x, c1p, c2p = LPT2_FACTORS
    spec, g = _potential(ic)
    h = {(a, b): torch.fft.irfftn(g[a] * g[b] * spec, s=shape) for a in range(3) for b in range(a, 3)}
    source = h[0, 0] * h[1, 1] + h[0, 0] * h[2, 2] + h[1, 1] * h[2, 2]
    source = source - h[0, 1] ** 2 - h[0, 2] ** 2 - h[1, 2] ** 2
    del h
    spec2, _ = _potential(source)
    dx = torch.empty(*shape, 3, device="cuda", dtype=torch.float64)
    p = torch.empty_like(dx)
    for a in range(3):
        f1, f2 = (torch.fft.irfftn(-g[a] * v, s=shape) for v in (spec, spec2))
        dx[..., a] = c1x * f1 + c2x * f2
        p[..., a] = c1p * c1x * f1 + c2p * c2x * f2
    return {"ic": ic, "dx": dx, "p": p}


def _exact_spectrum(case, s, ells):
    """Binned sums over the full grid; the bin of a mode is decided by |k| in FP32, the
    reference's grid."""
    shape, box = _shape(case), s["box"]
    f1 = torch.fft.fftn(s["mesh"].double())
    cross = s["mesh2"] is not None
    f = f1 * (torch.fft.fftn(s["mesh2"].double()) if cross else f1).conj() / f1.numel()
    del f1
    kv = []
    for a, (n, length) in enumerate(zip(shape, box)):
        i = torch.fft.fftfreq(n, 1.0 / n, device="cuda", dtype=torch.float32)
        kv.append((i * np.float32(2.0 * math.pi / length)).reshape([-1 if b == a else 1 for b in range(3)]))
    kmag = torch.sqrt(kv[0] * kv[0] + kv[1] * kv[1] + kv[2] * kv[2])
    edges = torch.as_tensor(s["kedges"], dtype=torch.float32, device="cuda")
    bins = torch.bucketize(kmag, edges, right=True).reshape(-1)
    nbins = edges.numel() + 1

    def total(v):
        return torch.zeros(nbins, device="cuda", dtype=torch.float64).index_add_(0, bins, v.reshape(-1))[1:-1]

    count = total(torch.ones_like(kmag, dtype=torch.float64)).clamp(min=1.0)
    k = total(kmag.double()) / count
    mu = kv[2].double() / torch.where(kmag > 0, kmag, torch.ones_like(kmag)).double()
    legendre = {0: lambda m: torch.ones_like(m), 2: lambda m: 1.5 * m**2 - 0.5,
                4: lambda m: (35.0 * m**4 - 30.0 * m**2 + 3.0) / 8.0}
    vol = float(np.prod([length / n for n, length in zip(shape, box)]))
    rows = []
    for ell in ells:
        w = (2 * ell + 1) * legendre[ell](mu)
        re = total(w * f.real)
        rows.append((torch.sqrt(re**2 + total(w * f.imag) ** 2) if cross else re) / count * vol)
    return k, rows[0] if len(rows) == 1 else torch.stack(rows)


def _ring(i, nside):
    """(first pixel, pixels, shifted by half a pixel) of rings 1 .. 4 nside - 1."""
    north = torch.where(i > 2 * nside, 4 * nside - i, i)
    cap = north < nside
    n = torch.where(cap, 4 * north, torch.full_like(north, 4 * nside))
    first = torch.where(cap, 2 * north * (north - 1), 2 * nside * (nside - 1) + (north - nside) * 4 * nside)
    first = torch.where(north != i, 12 * nside * nside - first - n, first)
    return first, n, torch.where(cap, torch.ones_like(north), ((north - nside) % 2 == 0).long())


def _ring_theta(i, nside):
    north = torch.where(i > 2 * nside, 4 * nside - i, i).double()
    t = north**2 / (3.0 * nside * nside)
    cap = torch.atan2(torch.sqrt(t * (2.0 - t)), 1.0 - t)
    belt = torch.acos(((2 * nside - north) * (2.0 / (3.0 * nside))).clamp(-1.0, 1.0))
    theta = torch.where(north < nside, cap, belt)
    return torch.where(i > 2 * nside, math.pi - theta, theta)


def _bilinear(v, r, nside):
    """Pixels and weights (4, n) of the bilinear interpolation at the directions v / r."""
    z = (v[:, 2] / r).clamp(-1.0, 1.0)
    theta = torch.acos(z)
    phi = torch.remainder(torch.atan2(v[:, 1], v[:, 0]), 2.0 * math.pi)
    belt = (nside * (2.0 - 1.5 * z)).long()
    cap = (nside * torch.sqrt(3.0 * (1.0 - z.abs()))).long()
    above = torch.where(z.abs() <= 2.0 / 3.0, belt, torch.where(z > 0, cap, 4 * nside - cap - 1))
    pix, w, th = [], [], []
    for ring in (above, above + 1):
        inside = (ring >= 1) & (ring <= 4 * nside - 1)
        i = ring.clamp(1, 4 * nside - 1)
        first, n, shift = _ring(i, nside)
        x = phi * n / (2.0 * math.pi) - 0.5 * shift
        low = torch.floor(x)
        j = low.long()
        pix += [first + torch.remainder(j, n), first + torch.remainder(j + 1, n)]
        w += [1.0 - (x - low), x - low]
        th.append(torch.where(inside, _ring_theta(i, nside), torch.where(ring < 1, torch.zeros_like(theta),
                                                                         torch.full_like(theta, math.pi))))
    lower = (theta - th[0]) / (th[1] - th[0])
    w = [w[0] * (1.0 - lower), w[1] * (1.0 - lower), w[2] * lower, w[3] * lower]
    # beyond the first or last ring the pole's share goes to its four pixels in equal parts
    npix = 12 * nside * nside
    for pole, near, far, base in ((above == 0, (2, 3), (0, 1), 0),
                                  (above == 4 * nside - 1, (0, 1), (2, 3), npix - 4)):
        share = 0.25 * (1.0 - lower if base == 0 else lower)
        for a, b in zip(near, far):
            w[a] = torch.where(pole, w[a] + share, w[a])
            w[b] = torch.where(pole, share, w[b])
            pix[b] = torch.where(pole, base + torch.remainder(pix[a] + 2, 4), pix[b])
    return torch.stack(pix), torch.stack(w)


def _nearest(v, r, nside):
    """RING pixel of the directions v / r."""
    z = v[:, 2] / r
    tt = torch.remainder(torch.atan2(v[:, 1], v[:, 0]), 2.0 * math.pi) / (0.5 * math.pi)
    jp, jm = (nside * (0.5 + tt) - nside * z * 0.75).long(), (nside * (0.5 + tt) + nside * z * 0.75).long()
    ring = nside + 1 + jp - jm
    ip = torch.remainder((jp + jm - nside + 1 - (ring & 1) + 1) // 2, 4 * nside)
    belt = 2 * nside * (nside - 1) + (ring - 1) * 4 * nside + ip
    x = nside * torch.sqrt(3.0 * (1.0 - z.abs()))
    tp = tt - torch.floor(tt)
    ring = (tp * x).long() + ((1.0 - tp) * x).long() + 1
    ip = torch.remainder((tt * ring).long(), 4 * ring)
    cap = torch.where(z > 0, 2 * ring * (ring - 1) + ip, 12 * nside * nside - 2 * ring * (ring + 1) + ip)
    return torch.where(z.abs() <= 2.0 / 3.0, belt, cap)


def _exact_shells(case, s):
    n, nside = case["n"], case["nside"]
    npix = 12 * nside * nside
    grid = torch.stack(torch.meshgrid(*[torch.arange(n, device="cuda", dtype=torch.float64)] * 3, indexing="ij"), -1)
    v = ((s["field"].array.double() + grid) * 4.0 - 2.0 * n).reshape(-1, 3)
    r = torch.sqrt((v**2).sum(-1))
    lo, hi = s["centers"] - s["widths"] / 2.0, s["centers"] + s["widths"] / 2.0
    out = torch.zeros(case["shells"], npix, device="cuda", dtype=torch.float64)
    for i in range(case["shells"]):
        take = (r > lo[i]) & (r <= hi[i])
        vi, ri = v[take], r[take]
        scale = 3.0 / (4.0 * math.pi / npix * (hi[i] ** 3 - lo[i] ** 3))
        if case["scheme"] == "ngp":
            out[i].index_add_(0, _nearest(vi, ri, nside), torch.full_like(ri, scale))
        else:
            pix, w = _bilinear(vi, ri, nside)
            out[i].index_add_(0, pix.reshape(-1), w.reshape(-1) * scale)
    return out


def _exact_cl(case, s):
    """healpy's anafast (three Jacobi iterations) with torch's FFT on the rings and the
    three-term recursion of the orthonormal Legendre functions in l, all m and rings at once."""
    nside, lmax = case["nside"], case["lmax"]
    maps = s["field"].array.double()
    npix, rings = 12 * nside * nside, 4 * nside - 1
    i = torch.arange(1, rings + 1, device="cuda")
    first, count, shift = (t.cpu().numpy() for t in _ring(i, nside))
    theta = _ring_theta(i, nside)
    z = torch.cos(theta)[None]
    m = torch.arange(lmax + 1, device="cuda", dtype=torch.float64)
    count_t = torch.as_tensor(count, device="cuda")
    # longitude of each ring's first pixel as the framework's transform takes it: in the belt
    # half a pixel where the painter's rings have none, and none where they have half a pixel
    phi0 = torch.as_tensor(np.where(count == 4 * nside, 1 - shift, shift) * math.pi / count, device="cuda")
    phase = torch.polar(torch.ones(rings, lmax + 1, device="cuda", dtype=torch.float64), -phi0[:, None] * m)
    wrap = torch.arange(lmax + 1, device="cuda")[None] % count_t[:, None]
    # runs of rings of one length, in ring order
    runs, r0 = [], 0
    while r0 < rings:
        r1 = r0
        while r1 < rings and count[r1] == count[r0]:
            r1 += 1
        runs.append((r0, r1, int(first[r0]), int(count[r0])))
        r0 = r1
    logmm = 0.5 * torch.cumsum(torch.cat([torch.zeros_like(m[:1]), torch.log((2 * m[1:] + 1) / (2 * m[1:]))]), 0)
    start = ((1.0 - 2.0 * (m % 2)) / math.sqrt(4.0 * math.pi))[:, None] * torch.exp(
        logmm[:, None] + m[:, None] * torch.log(torch.sin(theta))[None])

    def legendre():
        """(l, lambda_lm for m <= l over the rings), l ascending."""
        prev, cur = torch.zeros_like(start), torch.zeros_like(start)
        for ell in range(lmax + 1):
            mm = m[:ell]
            a = torch.sqrt((4.0 * ell * ell - 1.0) / (ell * ell - mm * mm)) if ell else mm
            b = torch.sqrt(((ell - 1.0) ** 2 - mm * mm) / (4.0 * (ell - 1.0) ** 2 - 1.0)) if ell > 1 else 0.0 * mm
            nxt = a[:, None] * (z * cur[:ell] - b[:, None] * prev[:ell])
            prev[:ell] = cur[:ell]
            cur[:ell] = nxt
            cur[ell] = start[ell]
            yield ell, cur[:ell + 1]

    def analysis(f):
        g = torch.empty(f.shape[0], rings, lmax + 1, device="cuda", dtype=torch.complex128)
        for r0, r1, p0, n in runs:
            spec = torch.fft.fft(f[:, p0:p0 + (r1 - r0) * n].reshape(-1, r1 - r0, n))
            g[:, r0:r1] = spec[..., wrap[r0]] * phase[r0:r1]
        g = torch.view_as_real(g.permute(2, 1, 0).contiguous()).flatten(2)  # (m, ring, maps x 2)
        alm = torch.zeros(lmax + 1, lmax + 1, 2 * f.shape[0], device="cuda", dtype=torch.float64)
        for ell, lam in legendre():
            alm[ell, :ell + 1] = torch.bmm(lam[:, None, :], g[:ell + 1])[:, 0]
        return alm * (4.0 * math.pi / npix)

    def synthesis(alm):
        g = torch.zeros(lmax + 1, rings, alm.shape[-1], device="cuda", dtype=torch.float64)
        for ell, lam in legendre():
            g[:ell + 1] += lam[:, :, None] * alm[ell, :ell + 1, None, :]
        g = torch.view_as_complex(g.reshape(lmax + 1, rings, -1, 2)).permute(2, 1, 0) * phase.conj()
        g[..., 1:] *= 2.0
        out = torch.empty(g.shape[0], npix, device="cuda", dtype=torch.float64)
        for r0, r1, p0, n in runs:
            spec = torch.zeros(g.shape[0], r1 - r0, n, device="cuda", dtype=torch.complex128)
            spec.index_add_(2, wrap[r0], g[:, r0:r1])
            out[:, p0:p0 + (r1 - r0) * n] = (torch.fft.ifft(spec).real * n).reshape(g.shape[0], -1)
        return out

    alm = analysis(maps)
    for _ in range(3):
        alm = alm + analysis(maps - synthesis(alm))
    power = (alm**2).reshape(lmax + 1, lmax + 1, -1, 2).sum(-1)
    cl = (2.0 * power.sum(1) - power[:, 0]) / (2.0 * m + 1.0)[:, None]
    return cl.T.contiguous()


def exact(case, seed):
    """What run() returns, in 64 bits. The whole runs and the drifted shells have none: they
    follow from the framework's own growth and distance tables; nor have the largest maps,
    whose plain transform takes minutes and needs scaled recursions."""
    kind = case["kind"]
    if kind in ("forward", "gradient", "tiled") or (kind == "cl" and case["nside"] > 256):
        return None
    s = prepare(case, seed)
    if kind == "forces":
        return _exact_forces(case, s)
    if kind == "initial":
        return _exact_initial(case, s)
    if kind == "power":
        return _exact_spectrum(case, s, (0,))
    if kind == "poles":
        return _exact_spectrum(case, s, tuple(range(0, case["lmax"] + 1, 2)))
    if kind == "shells":
        return _exact_shells(case, s)
    return _exact_cl(case, s)
