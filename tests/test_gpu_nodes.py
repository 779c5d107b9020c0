"""The node-by-node forward (csrc/cube_nodes.cu) against the general accumulate path.

rubix_cube_fwd and rubix_cube_fwd_general on the same inputs.  Tolerance, per spaxel and relative to the spaxel's largest value: in either path
beta = m T / T' carries up to ~3e-7 (T and T' four float32 products each, T' also the
2e-8 of its alpha table), an interpolated value ~2e-7, and a float32 sum of n <= 2600
values of one sign about sqrt(n) * 6e-8 = 3e-6 at most; together below 4e-6.
"""

import ctypes

import numpy as np
import pytest

from helpers import to_dev
from rubix_gb300 import synth
from rubix_gb300 import telescope as tel

pytestmark = pytest.mark.gpu

TOL = 4e-6


def _problem(counts, ssp=(12, 4, 400), wave=(4700.15, 9351.4), res=5.0, seed=0, edit=None,
             dist_z=0.1, v_sigma=120.0):
    """Stars given spaxel by spaxel: counts[s] of them in spaxel s."""
    rng = np.random.default_rng(seed)
    s = synth.make_ssp(*ssp, seed=1)
    n = int(np.sum(counts))
    p = dict(mass=1e5 * np.exp(rng.normal(0, 0.5, n)),
             metallicity=np.exp(rng.uniform(np.log(1e-4), np.log(0.05), n)),
             age=np.exp(rng.uniform(np.log(0.1), np.log(13.5), n)),
             vel=rng.normal(0.0, v_sigma, n))
    if edit is not None:
        edit(p, rng)
    p = {k: np.asarray(v, np.float32) for k, v in p.items()}
    offs = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    wt = tel.calculate_wave_seq(wave, res)
    return s, tel.cosmological_doppler_shift(dist_z, s.wavelength), wt, p, offs


def _run(lib, prob, general, lsf=None, av=None):
    import torch

    from rubix_gb300 import _lib

    s, wz, wt, p, offs = prob
    nz, na, nw = s.flux.shape
    n, nseg, L = p["mass"].size, offs.size - 1, wt.size
    d = [to_dev(x) for x in (s.flux, s.metallicity, s.age, wz, wt, p["mass"], p["metallicity"],
                             p["age"], p["vel"])]
    perm, off = to_dev(np.arange(n, dtype=np.int32)), to_dev(offs)
    size = _lib.query("rubix_cube_general_workspace_size" if general
                      else "rubix_cube_workspace_size", n, nseg, L, nz, na, nw)
    ws = torch.zeros(size, dtype=torch.uint8, device="cuda")
    out = torch.full((nseg, L), float("nan"), device="cuda")
    taps = None if lsf is None else np.asarray(lsf, np.float32)
    dust = []
    if av is not None or general:
        e = None if av is None else to_dev((-1.33 * (wt / 5500.0) ** -0.7).astype(np.float32))
        v = None if av is None else to_dev(np.asarray(av, np.float32))
        dust = [None if t is None else t.data_ptr() for t in (v, e)]
    name = "rubix_cube_fwd_general" if general else (
        "rubix_cube_fwd" if av is None else "rubix_cube_fwd_dust")
    _lib.call(name, *[t.data_ptr() for t in d[:4]], nz, na, nw, d[4].data_ptr(), L,
              *[t.data_ptr() for t in d[5:9]], 1, 0, *dust, perm.data_ptr(), off.data_ptr(),
              nseg, n, None if taps is None else taps.ctypes.data,
              0 if taps is None else taps.size, 0 if taps is None else taps.size // 2,
              out.data_ptr(), L, ws.data_ptr(), size, torch.cuda.current_stream().cuda_stream)
    err = ctypes.c_int(0)
    _lib.call("rubix_cube_status", ws.data_ptr(), ctypes.byref(err),
              torch.cuda.current_stream().cuda_stream)
    return out.cpu().numpy()


def _compare(lib, prob, lsf=None, av=None):
    a, b = _run(lib, prob, False, lsf, av), _run(lib, prob, True, lsf, av)
    assert np.array_equal(np.isfinite(a), np.isfinite(b))
    assert np.array_equal(np.isnan(a), np.isnan(b))
    c = b
    if (prob[3]["mass"] < 0).any():  # the bound is on sums of one sign
        c = _run(lib, prob[:3] + (dict(prob[3], mass=np.abs(prob[3]["mass"])), prob[4]), True, lsf, av)
    scale = np.nanmax(np.where(np.isfinite(c), np.abs(c), 0.0), axis=1, keepdims=True)
    with np.errstate(invalid="ignore"):
        err = np.abs(a - b) / np.maximum(scale, 1e-30)
    assert np.nanmax(np.where(np.isfinite(b), err, 0.0)) <= TOL
    assert not a[scale[:, 0] == 0].any() or not np.isfinite(a[scale[:, 0] == 0]).all()
    return a


EDGES = [0, 1, 2, 3, 4, 31, 32, 33, 39, 40, 41, 63, 64, 65, 255, 256, 257, 0, 1023, 1024, 1025,
         2600, 1]


@pytest.mark.parametrize("lsf", [None, 25, 9])
def test_item_edges(rubix_lib, lsf):
    """Spaxels around every edge of a warp's batch, a sorted run and a work item."""
    taps = None if lsf is None else tel.gaussian_taps_1d(lsf, 1.3)
    out = _compare(rubix_lib, _problem(EDGES), taps)
    assert not out[0].any() and not out[17].any()


@pytest.mark.parametrize("n_wave, res, wave", [
    (400, 1.25, (4700.15, 9351.4)),    # 15 samples an interval: slices of 14 nodes
    (160, 1.25, (4700.15, 9351.4)),    # 39 samples an interval: slices of 2 nodes
    (1221, 6.2, (4700.15, 9351.4)),    # barely more than one sample an interval
    (1221, 1.25, (5000.0, 5002.0)),    # two telescope wavelengths
    (1000, 1.25, (6000.0, 6080.0)),    # less than one slice
    (1447, 1.25, (3400.0, 8519.0)),    # 4096 samples, near both ends of the SSP grid
])
def test_grids(rubix_lib, n_wave, res, wave):
    _compare(rubix_lib, _problem([3, 50, 0, 300, 700], ssp=(5, 3, n_wave), wave=wave, res=res))


def test_uneven_grids(rubix_lib):
    """Logarithmic SSP wavelengths on a telescope grid whose step changes."""
    s, wz, wt, p, offs = _problem([3, 50, 0, 300, 700], ssp=(5, 3, 500))
    wz = np.geomspace(3300.0, 11000.0, 500).astype(np.float32)
    step = np.concatenate([np.full(900, 1.2), np.full(500, 2.1), np.full(900, 0.9)])
    wt = (4700.0 + np.cumsum(step)).astype(np.float32)
    _compare(rubix_lib, (s, wz, wt, p, offs))


def _hypervelocity(p, rng):
    p["vel"][5], p["vel"][60], p["vel"][90] = 2600.0, -9000.0, 30000.0


def _spread(p, rng):
    p["vel"] = rng.uniform(-2300.0, 2300.0, p["vel"].size)


def _not_finite(p, rng):
    p["mass"][3] = np.nan
    p["mass"][20] = np.inf
    p["vel"][70] = np.nan
    p["age"][120] = np.nan
    p["mass"][200] = 0.0


def _outside(p, rng):
    p["age"][::7] = 40.0
    p["metallicity"][::11] = 1.0
    p["mass"][:40] = 0.0


def _extreme(p, rng):
    p["mass"][3] = 1e36
    p["mass"][60:64] = 1e-38
    p["mass"][70:110] *= -1.0


@pytest.mark.parametrize("edit", [_hypervelocity, _spread, _not_finite, _outside, _extreme])
def test_particles_of_the_general_path(rubix_lib, edit):
    """Spaxels with particles that the tables do not cover, beside others that they do."""
    with np.errstate(over="ignore"):
        _compare(rubix_lib, _problem([40, 30, 70, 0, 300, 5], edit=edit))


@pytest.mark.parametrize("case", ["short", "fine", "flat", "inf", "zero"])
def test_grids_of_the_general_path(rubix_lib, case):
    """Template grids that do not qualify: not spanning the telescope range, finer than the
    telescope's bins, with repeated wavelengths, with a value that is not finite, empty."""
    s, wz, wt, p, offs = _problem([40, 3, 0, 300])
    if case == "short":
        wz = (wz - 4000.0).astype(np.float32)
        wz = np.linspace(5000.0, 9000.0, wz.size).astype(np.float32)
    elif case == "fine":
        wz = np.linspace(4000.0, 10500.0, wz.size).astype(np.float32)
        wt = tel.calculate_wave_seq((4700.0, 9300.0), 40.0)
    elif case == "flat":
        wz[200:203] = wz[200]
    elif case == "inf":
        s.flux[1, 4, 250] = np.inf
    else:
        s.flux[:] = 0.0
    a, b = _run(rubix_lib, (s, wz, wt, p, offs), False), _run(rubix_lib, (s, wz, wt, p, offs), True)
    fin = np.isfinite(b)
    assert np.array_equal(fin, np.isfinite(a)) and np.array_equal(np.isnan(a), np.isnan(b))
    scale = np.max(np.abs(b[fin])) if fin.any() else 1.0
    assert np.max(np.abs(a[fin] - b[fin]), initial=0.0) <= TOL * max(scale, 1e-30)


def test_random_template_noise(rubix_lib):
    """Templates with 50 % noise from node to node: the roughest the T' table meets."""
    prob = _problem(EDGES)
    rng = np.random.default_rng(5)
    prob[0].flux[:] *= rng.uniform(0.5, 1.5, prob[0].flux.shape).astype(np.float32)
    _compare(rubix_lib, prob)


@pytest.mark.parametrize("n_wave, res", [(400, 1.25), (1447, 1.25), (1221, 1.25), (1000, 1.25),
                                         (400, 5.0), (800, 1.6)])
@pytest.mark.parametrize("lsf", [None, 25])
def test_dust(rubix_lib, n_wave, res, lsf):
    """2 to 15 samples between two nodes (at most 4, 6, 8, or the general kernel's) behind
    columns of 0 to 200 mag; the transmission 2^x adds an approximation of 2^-22 = 2.4e-7,
    the same in both paths."""
    prob = _problem(EDGES, ssp=(5, 3, n_wave), res=res)
    n = prob[3]["mass"].size
    av = np.random.default_rng(3).exponential(0.5, n)
    av[::17] = 0.0
    av[5::311] = 200.0
    _compare(rubix_lib, prob, None if lsf is None else tel.gaussian_taps_1d(lsf, 1.3), av)


def test_dust_outliers(rubix_lib):
    """Columns that are not finite, or negative so that the transmission overflows."""
    prob = _problem([40, 30, 70, 0, 300, 5])
    av = np.random.default_rng(3).exponential(0.5, prob[3]["mass"].size)
    av[3], av[45], av[100], av[200:220] = np.nan, -300.0, np.inf, -2.0
    _compare(rubix_lib, prob, None, av)
