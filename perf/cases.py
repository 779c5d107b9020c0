"""The work that users of rubix_gb300 have it do, as measured cases.

A galaxy's star particles become an IFU datacube (one render), a mock survey renders many
galaxies of different sizes in one batch, and a fit differentiates the rendered cube with
respect to the stars and to the instrument widths.  Beside these whole calls stand the
layers a program calls by itself: the accumulation on an instrument and template grid of
odd sizes and with dust, the spaxel sort, the PSF and the LSF.

Sizes are those of the package's workloads (``rubix_gb300.synth.WORKLOADS``, the ragged
batch of ``rubix_gb300.ragged``) and numbers in between.
"""

import functools
import math

import numpy as np
import torch

from rubix_gb300 import ops, synth
from rubix_gb300 import telescope as tel
from rubix_gb300.api import IFURenderer
from rubix_gb300.autograd import render_cube
from rubix_gb300.ragged import RaggedBatch, galaxy_edges

C_KMS = 299792.458
DEV = "cuda"


def listed():
    return [
        # a quick-look render of a small simulated galaxy: launches and latency count
        dict(name="render_small", kind="render", n=10_000, sbin=25, n_age=20, n_met=6,
             n_ssp=1000, n_t=3721, psf=11, sigma=1.0, bulge=0.0, s2n=0.0),
        # the ordinary mock observation at IFU scale, full template grid
        dict(name="render_ifu", kind="render", n=1_000_000, sbin=150, n_age=221, n_met=6,
             n_ssp=1221, n_t=3721, psf=15, sigma=1.5, bulge=0.0, s2n=0.0),
        # the largest galaxy that is rendered in one piece: disk and bulge, noise at S/N 20
        dict(name="render_large", kind="render", n=10_000_000, sbin=300, n_age=221, n_met=6,
             n_ssp=1221, n_t=3721, psf=15, sigma=1.5, bulge=0.3, s2n=20.0),
        # a survey mock: galaxies of 1e3 to 1e6 stars on 16^2 to 64^2 spaxels, one batch
        dict(name="ragged_render", kind="ragged", n_gal=48, n_min=1000, n_max=1_000_000,
             s_min=16, s_max=64, layout=4, n_age=221, n_met=6, n_ssp=1221, n_t=3721,
             train=False),
        # one step of a fit: cube, inverse-variance loss, gradients of stars and widths
        dict(name="train_fit", kind="train", n=200_000, sbin=50, n_age=221, n_met=6,
             n_ssp=1221, n_t=3721, psf=15, sigma=1.5),
        # the same for a small galaxy and a coarse template grid (many such steps a second)
        dict(name="train_small", kind="train", n=10_000, sbin=25, n_age=20, n_met=6,
             n_ssp=1000, n_t=3721, psf=11, sigma=1.0),
        # one step of a joint fit of several galaxies
        dict(name="ragged_train", kind="ragged", n_gal=8, n_min=1000, n_max=500_000, s_min=16,
             s_max=48, layout=7, n_age=221, n_met=6, n_ssp=1221, n_t=3721, train=True),
        # the accumulation layer alone, on odd sizes: part of the wavelength range, odd grid
        dict(name="accumulate_odd", kind="accumulate", n=333_337, sbin=67, n_age=53, n_met=5,
             n_ssp=1447, n_t=2049, dust=False),
        # the accumulation layer with a dust column in front of every star
        dict(name="accumulate_dusty", kind="accumulate", n=500_000, sbin=101, n_age=221,
             n_met=6, n_ssp=1221, n_t=3721, dust=True),
        # spaxel assignment, aperture mask and stable sort of a large galaxy's stars
        dict(name="sort_large", kind="sort", n=10_000_000, sbin=300),
        # the instrument layers alone, on a cube that a program already has
        dict(name="psf_ifu", kind="psf", sbin=150, n_t=3721, psf=15, sigma=1.5),
        dict(name="lsf_ifu", kind="lsf", sbin=150, n_t=3721, sigma=1.2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render", "render", "ragged", "train", "accumulate", "accumulate",
                       "ragged_train", "sort", "psf", "lsf"])
    n_age, n_met, n_ssp = rng.choice([(20, 6, 1000), (221, 6, 1221), (221, 6, 1221),
                                      (rng.randint(8, 200), rng.randint(2, 6),
                                       rng.randint(800, 1500))])
    grid = dict(n_age=n_age, n_met=n_met, n_ssp=n_ssp, n_t=rng.choice([3721, 3721,
                                                                     rng.randint(700, 3721)]))
    if kind == "render":
        return dict(kind=kind, n=_log(rng, 1e4, 8e6), sbin=_log(rng, 16, 280), **grid,
                    psf=rng.choice([5, 11, 15, 21]), sigma=rng.uniform(0.6, 2.0),
                    bulge=rng.choice([0.0, 0.0, 0.3]), s2n=rng.choice([0.0, 20.0]))
    if kind in ("ragged", "ragged_train"):
        train = kind == "ragged_train"
        return dict(kind="ragged", n_gal=rng.randint(2, 8 if train else 40), n_min=1000,
                    n_max=500_000 if train else 1_000_000, s_min=16, s_max=48 if train else 64,
                    layout=rng.randint(0, 10**6), train=train, **grid)
    if kind == "train":
        return dict(kind=kind, n=_log(rng, 1e4, 1e6), sbin=_log(rng, 16, 80), **grid,
                    psf=rng.choice([5, 11, 15, 21]), sigma=rng.uniform(0.6, 2.0))
    if kind == "accumulate":
        return dict(kind=kind, n=_log(rng, 1e4, 2e6), sbin=_log(rng, 16, 200), **grid,
                    dust=rng.random() < 0.4)
    if kind == "sort":
        return dict(kind=kind, n=_log(rng, 1e4, 1e7), sbin=_log(rng, 16, 300))
    case = dict(kind=kind, sbin=_log(rng, 16, 250), n_t=rng.choice([3721, rng.randint(700, 3721)]),
                sigma=rng.uniform(0.8, 2.0))
    return case if kind == "lsf" else dict(case, psf=rng.choice([5, 11, 15, 21]))


# ------------------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=4)
def _ssp(n_age, n_met, n_ssp):
    return synth.make_ssp(n_age, n_met, n_ssp, seed=2)


def _wave_t(n_t):
    return tel.calculate_wave_seq(synth.WAVE_RANGE, synth.WAVE_RES)[:n_t]


def _field(sbin):
    """Field of view in arcsec and a scale length that fills it, as in the workloads."""
    return sbin * synth.SPATIAL_RES


def _stars(n, seed, bulge=0.0):
    """Exponential disk (R_d 3 kpc, h_z 0.3 kpc, 200 km/s rotation, 50 km/s dispersion,
    inclined by 60 degrees), optionally with a Plummer bulge; log-uniform ages and
    metallicities, log-normal masses.  All on the device."""
    g = torch.Generator(DEV).manual_seed(1_000_003 * seed + n)

    def uni(*shape):
        return torch.rand(*shape, generator=g, device=DEV, dtype=torch.float64)

    def nrm(*shape):
        return torch.randn(*shape, generator=g, device=DEV, dtype=torch.float64)

    R = -3.0 * torch.log((1 - uni(n)) * (1 - uni(n)))
    phi = 2 * math.pi * uni(n)
    u = uni(n) - 0.5
    z = -0.3 * torch.sign(u) * torch.log1p(-2 * u.abs())
    x, y = R * torch.cos(phi), R * torch.sin(phi)
    vx, vy, vz = -200.0 * torch.sin(phi), 200.0 * torch.cos(phi), torch.zeros_like(phi)
    if bulge > 0:
        b = uni(n) < bulge
        r = 1.0 / torch.sqrt(uni(n).clamp_min(1e-6) ** (-2.0 / 3.0) - 1.0)
        d = nrm(n, 3)
        d = d / d.norm(dim=1, keepdim=True) * r.clamp_max(50.0)[:, None]
        vb = 120.0 * nrm(n, 3)
        x, y, z = (torch.where(b, d[:, i], c) for i, c in enumerate((x, y, z)))
        vx, vy, vz = (torch.where(b, vb[:, i], c) for i, c in enumerate((vx, vy, vz)))
    ci, si = math.cos(math.pi / 3), math.sin(math.pi / 3)
    coords = torch.stack([x, ci * y - si * z, si * y + ci * z], dim=1)
    vel = torch.stack([vx, ci * vy - si * vz, si * vy + ci * vz + 50.0 * nrm(n)], dim=1)
    age = torch.exp(math.log(0.1) + uni(n) * math.log(135.0))
    met = torch.exp(math.log(1e-4) + uni(n) * math.log(500.0))
    mass = 1e5 * torch.exp(0.5 * nrm(n))
    return {k: v.to(torch.float32).contiguous() for k, v in
            dict(coords=coords, velocity=vel, mass=mass, metallicity=met, age=age).items()}


def _renderer(case, sbin, psf=None, sigma=None, s2n=None, lsf=True):
    ssp = _ssp(case["n_age"], case["n_met"], case["n_ssp"])
    edges, _ = tel.spatial_bin_edges(_field(sbin), sbin, synth.DIST_Z)
    return IFURenderer(
        ssp.age, ssp.metallicity, ssp.wavelength, ssp.flux, _wave_t(case["n_t"]), edges, sbin,
        synth.DIST_Z, psf_taps=None if psf is None else tel.gaussian_taps_1d(psf, sigma),
        lsf_taps=tel.lsf_taps(synth.LSF_SIGMA, synth.WAVE_RES) if lsf else None,
        device=DEV, noise_s2n=s2n or None)


def _layout(case):
    rng = np.random.Generator(np.random.PCG64(case["layout"]))
    g = case["n_gal"]
    counts = np.exp(rng.uniform(np.log(case["n_min"]), np.log(case["n_max"]), g)).astype(int)
    sbins = rng.integers(case["s_min"], case["s_max"] + 1, g)
    sig = rng.uniform(0.8, 2.0, g)
    sizes = 2 * np.ceil(3 * sig).astype(int) + 1
    return counts, sbins, sig, sizes


def _cube(sbin, n_t, seed):
    g = torch.Generator(DEV).manual_seed(seed + 17)
    return torch.rand(sbin, sbin, n_t, generator=g, device=DEV, dtype=torch.float32)


def _dust(case, seed):
    """A_V of every star (mean 0.5 mag) and -0.4 log2(10) A(lambda)/A(V) for a power law."""
    g = torch.Generator(DEV).manual_seed(seed + 29)
    av = torch.empty(case["n"], device=DEV, dtype=torch.float32).exponential_(2.0, generator=g)
    wt = torch.as_tensor(_wave_t(case["n_t"]), device=DEV)
    return av, (-0.4 * math.log2(10.0) * (wt.double() / 5500.0) ** -0.7).float()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "render":
        r = _renderer(case, case["sbin"], case["psf"], case["sigma"], case["s2n"])
        return dict(kind=kind, r=r, p=_stars(case["n"], seed, case["bulge"]))
    if kind == "sort":
        edges, _ = tel.spatial_bin_edges(_field(case["sbin"]), case["sbin"], synth.DIST_Z)
        return dict(kind=kind, coords=_stars(case["n"], seed)["coords"], sbin=case["sbin"],
                    edges=torch.as_tensor(edges, device=DEV))
    if kind == "psf":
        return dict(kind=kind, cube=_cube(case["sbin"], case["n_t"], seed),
                    taps=tel.gaussian_taps_1d(case["psf"], case["sigma"]))
    if kind == "lsf":
        return dict(kind=kind, cube=_cube(case["sbin"], case["n_t"], seed),
                    taps=tel.lsf_taps(case["sigma"], synth.WAVE_RES))
    if kind == "accumulate":
        r = _renderer(case, case["sbin"], lsf=False)
        p = _stars(case["n"], seed)
        perm, offs = r.sort(*r.assign(p["coords"]))
        av, e = _dust(case, seed) if case["dust"] else (None, None)
        return dict(kind=kind, r=r, p=p, perm=perm, offs=offs, av=av, e=e)
    if kind == "train":
        r = _renderer(case, case["sbin"], lsf=False)
        p = _stars(case["n"], seed)
        for k in ("mass", "metallicity", "age", "velocity"):
            p[k].requires_grad_()
        sbin = case["sbin"]
        edges, _ = tel.spatial_bin_edges(_field(sbin), sbin, synth.DIST_Z)
        obs = {k: v.view(sbin, sbin, -1)
               for k, v in _observed(case, [(p, edges, sbin)], seed).items()}
        return dict(kind=kind, r=r, p=p, psf=case["psf"], **obs,
                    sp=torch.tensor(case["sigma"], dtype=torch.float64, device=DEV,
                                    requires_grad=True),
                    sl=torch.tensor(synth.LSF_SIGMA, dtype=torch.float64, device=DEV,
                                    requires_grad=True))
    counts, sbins, sig, sizes = _layout(case)
    r = _renderer(case, int(sbins[0]), lsf=False)
    b = RaggedBatch(r, counts, sbins, [galaxy_edges(int(s), synth.DIST_Z) for s in sbins], sig,
                    sizes, synth.LSF_SIGMA, synth.WAVE_RES)
    parts = [_stars(int(n), seed * 1009 + i) for i, n in enumerate(counts)]
    p = {k: torch.cat([q[k] for q in parts]) for k in parts[0]}
    state = dict(kind=kind, b=b, p=p)
    if case["train"]:
        state.update(_observed(case, [(q, galaxy_edges(int(s), synth.DIST_Z), int(s))
                                      for q, s in zip(parts, sbins)], seed))
    return state


def _args(p):
    return dict(coords=p["coords"], velocity=p["velocity"], mass=p["mass"],
                metallicity=p["metallicity"], age=p["age"])


def _observed(case, fields, seed):
    """An observed cube and its inverse variance.  The cube is the mass of the stars in
    each spaxel times the mean template, smeared over 3 x 3 spaxels, with 2 % noise: it
    has the model's shape and scale, not its values.  ``fields``: (stars, edges, sbin)."""
    ssp = _ssp(case["n_age"], case["n_met"], case["n_ssp"])
    wz = (1.0 + synth.DIST_Z) * ssp.wavelength.astype(np.float64)
    mean = np.interp(_wave_t(case["n_t"]), wz, ssp.flux.astype(np.float64).mean(axis=(0, 1)))
    maps = []
    for p, edges, sbin in fields:
        seg, keep = _spaxels(p["coords"], edges, sbin)
        m = np.bincount(seg[keep].cpu().numpy(), minlength=sbin * sbin,
                        weights=p["mass"].detach()[keep].cpu().double().numpy())
        m = np.pad(m.reshape(sbin, sbin), 1)
        m = sum(m[i:i + sbin, j:j + sbin] for i in range(3) for j in range(3)) / 9.0
        maps.append(m.reshape(-1))
    m = torch.as_tensor(np.concatenate(maps), device=DEV)[:, None]
    cube = (m * torch.as_tensor(mean, device=DEV)[None, :]).float()
    scale = float(m.mean()) * float(mean.mean())
    g = torch.Generator(DEV).manual_seed(seed + 41)
    weight = 1.0 / (scale * (cube + 0.1 * scale))
    noise = torch.randn(cube.shape, generator=g, device=DEV, dtype=torch.float32)
    return dict(target=cube + 0.02 * scale * noise, weight=weight)


def run(state):
    kind = state["kind"]
    if kind == "render":
        return state["r"].render(**_args(state["p"])).final
    if kind == "sort":
        idx = ops.spaxel_assign(state["coords"], state["edges"])
        keep = ops.aperture_mask(state["coords"], state["edges"])
        return (idx, keep) + tuple(ops.spaxel_sort(idx, state["sbin"] ** 2, keep))
    if kind == "psf":
        return ops.psf_forward(state["cube"], state["taps"])
    if kind == "lsf":
        return ops.lsf_forward(state["cube"], state["taps"], (len(state["taps"]) - 1) // 2)
    if kind == "accumulate":
        r, p = state["r"], state["p"]
        return ops.cube_forward(
            r.ssp_flux, r.ssp_metallicity, r.ssp_age, r.ssp_wave_z, r.wave_t, p["mass"],
            p["metallicity"], p["age"], p["velocity"], r.velocity_axis, state["perm"],
            state["offs"], r.sbin * r.sbin, dust_av=state["av"], dust_exponent=state["e"])
    if kind == "train":
        p = state["p"]
        leaves = [p["mass"], p["metallicity"], p["age"], p["velocity"], state["sp"], state["sl"]]
        cube = render_cube(state["r"], p["coords"], p["velocity"], p["mass"], p["metallicity"],
                           p["age"], state["sp"], state["sl"], state["psf"], synth.WAVE_RES)
        loss = (state["weight"] * (cube - state["target"]) ** 2).sum()
        grads = torch.autograd.grad(loss, leaves)
        return dict(cube=cube.detach(), loss=loss.detach(), mass=grads[0], metallicity=grads[1],
                    age=grads[2], velocity=grads[3], sigma_psf=grads[4], sigma_lsf=grads[5])
    if "target" not in state:
        return state["b"].render(**_args(state["p"]))
    loss, grads, d_psf, d_lsf, cube = state["b"].forward_backward(
        **_args(state["p"]), target=state["target"], weight=state["weight"])
    return dict(cube=cube, loss=loss, mass=grads[0], metallicity=grads[1], age=grads[2],
                velocity=grads[3], sigma_psf=d_psf, sigma_lsf=d_lsf)


# ------------------------------------------------------------------ necessary work
def _accumulate_work(n, nseg, case):
    """24 bytes a star (mass, age, metallicity, velocity, sorted index), the template grid
    and the cube once; per star the four-corner mix and resampling of its templates over
    the part of the SSP grid that the instrument sees."""
    span = (synth.WAVE_RES * case["n_t"]) / ((1 + synth.DIST_Z) * 7000.0) * case["n_ssp"]
    nodes = min(span, case["n_ssp"])
    grid = 4.0 * case["n_age"] * case["n_met"] * case["n_ssp"]
    return 24.0 * n + grid + 4.0 * nseg * case["n_t"], n * nodes * 16.0


def work(case):
    kind = case["kind"]
    if kind == "sort":
        return {"bytes": 25.0 * case["n"], "flops": 0.0}
    if kind in ("psf", "lsf"):
        c = float(case["sbin"] ** 2 * case["n_t"])
        return {"bytes": 8.0 * c, "flops": c * 2 * (2 * case["psf"] if kind == "psf" else 25)}
    if kind == "ragged":
        counts, sbins, _, sizes = _layout(case)
        n, nseg, k = float(counts.sum()), float((sbins ** 2).sum()), float(sizes.mean())
        train = case["train"]
    else:
        n, nseg, k = float(case["n"]), float(case["sbin"] ** 2), float(case.get("psf", 0))
        train = kind == "train"
    b, f = _accumulate_work(n, nseg, case)
    if kind == "accumulate":
        return {"bytes": b + (4.0 * n if case["dust"] else 0.0), "flops": f}
    cube = nseg * case["n_t"]
    b, f = b + 12.0 * n, f + cube * 2 * (2 * k + 25)
    if train:  # target, weight and gradients; the adjoint of every stage
        b, f = b + 8.0 * cube + 16.0 * n, 3.0 * f
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ 64-bit results
def _grids(case):
    ssp = _ssp(case["n_age"], case["n_met"], case["n_ssp"])
    d = dict(age=ssp.age, met=ssp.metallicity, flux=ssp.flux,
             wz=(np.float32(1.0 + synth.DIST_Z) * ssp.wavelength).astype(np.float32),
             wt=_wave_t(case["n_t"]))
    return {k: torch.as_tensor(np.ascontiguousarray(v), device=DEV) for k, v in d.items()}


def _spaxels(coords, edges, sbin):
    """The spaxel of every star (last bin clipped) and whether it is inside the aperture."""
    e = torch.as_tensor(edges, device=DEV)
    x, y = coords[:, 0].contiguous(), coords[:, 1].contiguous()
    nb = e.numel() - 1
    ix = (torch.searchsorted(e, x, right=True) - 1).clamp(0, nb - 1)
    iy = (torch.searchsorted(e, y, right=True) - 1).clamp(0, nb - 1)
    keep = (x >= e[0]) & (x <= e[-1]) & (y >= e[0]) & (y <= e[-1])
    seg = ix + nb * iy
    return seg, keep & (seg < sbin * sbin)


def _rows(g, mass, met, age, vel):
    """[m, L] resampled spectra in 64 bits.  The Doppler-shifted wavelengths are the float32
    values that define the path (mask and brackets are taken on them)."""
    z, a = g["met"].double(), g["age"].double()
    iz = torch.searchsorted(g["met"], met.detach().float(), right=True).clamp(1, z.numel() - 1)
    ia = torch.searchsorted(g["age"], age.detach().float(), right=True).clamp(1, a.numel() - 1)
    tz = ((met - z[iz - 1]) / (z[iz] - z[iz - 1]))[:, None]
    ta = ((age - a[ia - 1]) / (a[ia] - a[ia - 1]))[:, None]
    inside = ((met >= z[0]) & (met <= z[-1]) & (age >= a[0]) & (age <= a[-1]))[:, None]
    F = g["flux"]
    G = ((1 - tz) * (1 - ta) * F[iz - 1, ia - 1] + tz * (1 - ta) * F[iz, ia - 1]
         + (1 - tz) * ta * F[iz - 1, ia] + tz * ta * F[iz, ia]) * inside
    v0 = vel.detach()
    lam32 = g["wz"][None, :] * torch.exp(v0 / C_KMS).float()[:, None]
    lam = lam32.double() * torch.exp((vel - v0) / C_KMS)[:, None]
    x32, x = g["wt"], g["wt"].double()
    mask = (lam32 >= x32[0]) & (lam32 <= x32[-1])
    T = (G[:, 1:] * (lam[:, 1:] - lam[:, :-1]) * mask[:, 1:]).sum(1)
    nw = lam32.shape[1]
    k = torch.searchsorted(lam32, x32[None, :].expand(lam32.shape[0], -1).contiguous(), right=True)
    lo = k.clamp(1, nw - 1) - 1
    l0, l1 = lam.gather(1, lo), lam.gather(1, lo + 1)
    G0, G1 = G.gather(1, lo), G.gather(1, lo + 1)
    t = ((x[None, :] - l0) / (l1 - l0)).clamp(0, 1)
    rows = G0 + t * (G1 - G0)
    dx = torch.diff(x, prepend=x[:1])
    return rows * (mass * torch.nan_to_num(T / (rows @ dx)))[:, None]


def _accumulate(g, p, seg, keep, nseg, chunk=16384, av=None, e=None):
    cube = torch.zeros(nseg, g["wt"].numel(), dtype=torch.float64, device=DEV)
    sel = torch.nonzero(keep).flatten()
    for s in sel.split(chunk):
        rows = _rows(g, *(p[k][s].double() for k in ("mass", "metallicity", "age")),
                     p["velocity"][s, 2].double())
        if av is not None:
            rows = rows * torch.exp2(e.double()[None, :] * av[s].double()[:, None])
        cube.index_add_(0, seg[s], rows)
    return cube


def _conv(x, taps, crop):
    """Full convolution along the last axis, cropped to [crop, crop + length)."""
    shape = x.shape
    k = taps.numel()
    y = torch.nn.functional.pad(x.reshape(-1, 1, shape[-1]), (k - 1 - crop, crop))
    out = torch.zeros_like(x.reshape(-1, 1, shape[-1]))
    for j in range(k):
        out = out + taps[k - 1 - j] * y[..., j:j + shape[-1]]
    return out.reshape(shape)


def _psf(x, taps):
    c = (taps.numel() - 1) // 2
    y = _conv(x.permute(2, 1, 0), taps, c)          # along y
    return _conv(y.permute(0, 2, 1), taps, c).permute(1, 2, 0)


def _gauss(pos, sigma):
    e = torch.exp(-pos ** 2 / (2 * sigma ** 2))
    return e / e.sum()


def _psf_taps(m, sigma):
    return _gauss(torch.arange(m, dtype=torch.float64, device=DEV) - (m - 1) / 2, sigma)


def _lsf_taps(sigma):
    d = synth.WAVE_RES
    x = np.arange(-12 * d, 12 * d + d, d, dtype=np.float32).astype(np.float64)
    return _gauss(torch.as_tensor(x, device=DEV), sigma)


def _lsf(x, taps):
    return _conv(x, taps, (taps.numel() - 1) // 2)


def _fit_exact(g, p, seg, keep, sbin, psf, sigma, target, weight):
    """Cube, loss and gradients of one galaxy's fit step."""
    acc = _accumulate(g, p, seg, keep, sbin * sbin).requires_grad_()
    sp = torch.tensor(float(sigma), dtype=torch.float64, device=DEV, requires_grad=True)
    sl = torch.tensor(synth.LSF_SIGMA, dtype=torch.float64, device=DEV, requires_grad=True)
    q = _lsf(acc, _lsf_taps(sl)).reshape(sbin, sbin, -1)
    cube = _psf(q, _psf_taps(psf, sp))
    weight, target = (t.double().reshape(cube.shape) for t in (weight, target))
    loss = (weight * (cube - target) ** 2).sum()
    h, gp, gl = torch.autograd.grad(loss, [acc, sp, sl])
    out = {k: torch.zeros(keep.numel(), dtype=torch.float64, device=DEV)
           for k in ("mass", "metallicity", "age", "vlos")}
    for s in torch.nonzero(keep).flatten().split(8192):
        leaves = [p[k][s].detach().double().requires_grad_()
                  for k in ("mass", "metallicity", "age")]
        leaves.append(p["velocity"][s, 2].detach().double().requires_grad_())
        rows = _rows(g, *leaves)
        gs = torch.autograd.grad((rows * h[seg[s]]).sum(), leaves)
        for k, v in zip(out, gs):
            out[k][s] = v
    return cube.detach(), loss.detach(), out, gp, gl


def exact(case, seed):
    kind = case["kind"]
    if kind == "sort":
        return None
    if kind in ("psf", "lsf"):
        x = _cube(case["sbin"], case["n_t"], seed).double()
        return (_psf(x, _psf_taps(case["psf"], case["sigma"])) if kind == "psf"
                else _lsf(x, _lsf_taps(case["sigma"])))
    g = _grids(case)
    if kind in ("render", "accumulate"):
        sbin = case["sbin"]
        p = _stars(case["n"], seed, case.get("bulge", 0.0))
        edges, _ = tel.spatial_bin_edges(_field(sbin), sbin, synth.DIST_Z)
        seg, keep = _spaxels(p["coords"], edges, sbin)
        av, e = _dust(case, seed) if case.get("dust") else (None, None)
        acc = _accumulate(g, p, seg, keep, sbin * sbin, av=av, e=e)
        if kind == "accumulate":
            return acc
        cube = _psf(_lsf(acc, _lsf_taps(synth.LSF_SIGMA)).reshape(sbin, sbin, -1),
                    _psf_taps(case["psf"], case["sigma"]))
        # the noise is zero when a spaxel is empty; else it is drawn from the path's generator
        return cube if not case["s2n"] or bool((cube.sum(-1) <= 0).any()) else None
    if kind == "train":
        s = prepare(case, seed)
        sbin = case["sbin"]
        edges, _ = tel.spatial_bin_edges(_field(sbin), sbin, synth.DIST_Z)
        p = {k: v.detach() for k, v in s["p"].items()}
        seg, keep = _spaxels(p["coords"], edges, sbin)
        cube, loss, d, gp, gl = _fit_exact(g, p, seg, keep, sbin, case["psf"], case["sigma"],
                                           s["target"], s["weight"])
        gv = torch.zeros(case["n"], 3, dtype=torch.float64, device=DEV)
        gv[:, 2] = d["vlos"]
        return dict(cube=cube, loss=loss, mass=d["mass"], metallicity=d["metallicity"],
                    age=d["age"], velocity=gv, sigma_psf=gp, sigma_lsf=gl)
    s = prepare(case, seed)
    counts, sbins, sig, sizes = _layout(case)
    po = np.concatenate([[0], np.cumsum(counts)])
    so = np.concatenate([[0], np.cumsum(sbins ** 2)])
    cubes, losses, gps, gls, ds = [], [], [], [], []
    for i, sbin in enumerate(int(x) for x in sbins):
        p = {k: v[po[i]:po[i + 1]] for k, v in s["p"].items()}
        seg, keep = _spaxels(p["coords"], galaxy_edges(sbin, synth.DIST_Z), sbin)
        if not case["train"]:
            acc = _accumulate(g, p, seg, keep, sbin * sbin)
            cube = _psf(_lsf(acc, _lsf_taps(synth.LSF_SIGMA)).reshape(sbin, sbin, -1),
                        _psf_taps(int(sizes[i]), float(sig[i])))
            cubes.append(cube.reshape(sbin * sbin, -1))
            continue
        cube, loss, d, gp, gl = _fit_exact(
            g, p, seg, keep, sbin, int(sizes[i]), float(sig[i]), s["target"][so[i]:so[i + 1]],
            s["weight"][so[i]:so[i + 1]])
        cubes.append(cube.reshape(sbin * sbin, -1))
        losses.append(loss)
        gps.append(gp)
        gls.append(gl)
        ds.append(d)
    if not case["train"]:
        return torch.cat(cubes)
    return dict(cube=torch.cat(cubes), loss=torch.stack(losses).sum(),
                mass=torch.cat([d["mass"] for d in ds]),
                metallicity=torch.cat([d["metallicity"] for d in ds]),
                age=torch.cat([d["age"] for d in ds]),
                velocity=torch.cat([d["vlos"] for d in ds]),
                sigma_psf=torch.stack(gps), sigma_lsf=torch.stack(gls).sum())
