"""The node path on templates with emission lines, where T'(alpha) has kinks that an
interpolation over the Doppler factor cuts: T' has to be summed on the shifted grid.

Tolerances are those of test_gpu_nodes.py and test_gpu_nodes_bwd.py, whose derivations do not
depend on the templates."""

import numpy as np
import pytest

import oracle
from rubix_gb300 import synth
from test_gpu_nodes import EDGES, TOL, _compare, _problem, _run
from test_gpu_nodes_bwd import _check

pytestmark = pytest.mark.gpu

LINES = (3727.0, 4102.0, 4340.0, 4861.0, 5007.0, 6563.0)


def _lines(s, kind):
    F, x = s.flux.astype(np.float64), s.wavelength.astype(np.float64)
    if kind.startswith("node"):  # one node at 10 or 100 times the continuum, in each line
        for line in LINES:
            F[..., np.argmin(np.abs(x - line))] *= float(kind[4:])
    elif kind == "pure":  # lines on next to no continuum
        F *= 1e-6
        for i, line in enumerate(LINES):
            F[..., np.argmin(np.abs(x - line))] += s.flux.mean() * (1 + i)
    elif kind == "young":  # only templates younger than 1 Gyr have lines
        for line in LINES:
            F[:, s.age < 1.0, np.argmin(np.abs(x - line))] *= 50.0
    else:  # Gaussian lines of 3 A sigma and 100 or 1000 A equivalent width
        for line in LINES:
            c = F[..., np.argmin(np.abs(x - line))][..., None]
            F += c * float(kind[4:]) * np.exp(-0.5 * ((x - line) / 3.0) ** 2) / (3.0 * 2.5066)
    s.flux[:] = F


CASES = [(kind, ssp, res) for kind in ("node10", "node100", "pure", "young", "line100", "line1000")
         for ssp, res in (((5, 3, 1221), 1.25), ((5, 3, 400), 5.0))]


@pytest.mark.parametrize("kind, ssp, res", CASES)
def test_forward(rubix_lib, kind, ssp, res):
    prob = _problem(EDGES, ssp=ssp, res=res)
    _lines(prob[0], kind)
    a = _compare(rubix_lib, prob)
    b = _run(rubix_lib, prob, True)
    assert not np.array_equal(a, b)  # two ways of summing: the node path has run
    # against float64, on the spaxels of up to 65 stars
    s, wz, wt, p, offs = prob
    small = np.flatnonzero((np.diff(offs) > 0) & (np.diff(offs) < 70))
    for seg in small:
        i = slice(offs[seg], offs[seg + 1])
        want = oracle.particle_spectra(p["mass"][i], p["metallicity"][i], p["age"][i], p["vel"][i],
                                       s.metallicity, s.age, s.flux, wz, wt).sum(0)
        scale = np.abs(want).max()
        assert np.abs(a[seg] - want).max() <= np.abs(b[seg] - want).max() + TOL * scale


def test_forward_dust(rubix_lib):
    prob = _problem(EDGES, ssp=(5, 3, 1221), res=1.25)
    _lines(prob[0], "node100")
    _compare(rubix_lib, prob, None, np.random.default_rng(3).exponential(0.5, prob[3]["mass"].size))


@pytest.mark.parametrize("kind, ssp, res", CASES)
def test_adjoint(rubix_lib, kind, ssp, res):
    prob = _problem(EDGES, ssp=ssp, res=res)
    _lines(prob[0], kind)
    _check(prob)


def test_uneven_samples(rubix_lib):
    """Samples whose step changes: the first sample of an interval is searched."""
    s, wz, wt, p, offs = _problem([3, 50, 0, 300, 700], ssp=(5, 3, 500))
    wz = np.geomspace(3300.0, 11000.0, 500).astype(np.float32)
    step = np.concatenate([np.full(900, 1.2), np.full(500, 2.1), np.full(900, 0.9)])
    wt = (4700.0 + np.cumsum(step)).astype(np.float32)
    _lines(s, "node100")
    _compare(rubix_lib, (s, wz, wt, p, offs))
