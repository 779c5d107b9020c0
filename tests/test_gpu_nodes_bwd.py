"""The node-by-node adjoint (csrc/cube_nodes_bwd.cu) against the general one, which the
dusty entry point runs; with columns of 0 mag its transmission is exactly 1.

Tolerance: a float32 sum of N products of either sign, formed in parts of n and then of
N / n terms, is off by about 6e-8 (sqrt(n) + sqrt(N / n)) of its rms size; with N = 3721 and
parts of about 60 that is 1e-6 per path, and the ratio T / T' and its derivatives add 3e-7.
4e-6 in the 2-norm covers both paths; single elements may be ten times as far off."""

import numpy as np
import pytest

from helpers import to_dev
from test_gpu_nodes import (EDGES, _extreme, _hypervelocity, _not_finite, _outside, _problem,
                            _spread)

pytestmark = pytest.mark.gpu


def _grads(prob, adj, general):
    import torch

    from rubix_gb300 import ops

    s, wz, wt, p, offs = prob
    n = p["mass"].size
    dust = {}
    if general:
        dust = dict(dust_av=torch.zeros(n, device="cuda"),
                    dust_exponent=torch.zeros(wt.size, device="cuda"))
    out = ops.cube_backward(
        *[to_dev(x) for x in (s.flux, s.metallicity, s.age, wz, wt, p["mass"], p["metallicity"],
                              p["age"], p["vel"])], 0,
        to_dev(np.arange(n, dtype=np.int32)), to_dev(offs), offs.size - 1, to_dev(adj), **dust)
    return [g.cpu().numpy() for g in out]


def _check(prob, seed=1, smooth=False, edit_adj=None):
    rng = np.random.default_rng(seed)
    nseg, L = prob[4].size - 1, prob[2].size
    adj = rng.normal(size=(nseg, L)).astype(np.float32)
    if smooth:
        adj = (1.0 + 0.3 * np.cos(np.arange(L) / 37.0))[None, :].repeat(nseg, 0).astype(np.float32)
    if edit_adj is not None:
        edit_adj(adj)
    got, want = _grads(prob, adj, False), _grads(prob, adj, True)
    for name, a, b in zip(("mass", "metallicity", "age", "velocity"), got, want):
        assert np.array_equal(np.isnan(a), np.isnan(b)), name
        ok = np.isfinite(b)
        assert np.array_equal(ok, np.isfinite(a)), name
        a, b = a[ok].astype(np.float64), b[ok].astype(np.float64)
        rms = np.sqrt(np.mean(b ** 2)) if b.size else 0.0
        assert np.sqrt(np.mean((a - b) ** 2)) <= 4e-6 * rms, name
        assert (np.abs(a - b) <= 4e-5 * np.maximum(np.abs(b), rms)).all(), name


@pytest.mark.parametrize("smooth", [False, True])
def test_item_edges(rubix_lib, smooth):
    _check(_problem(EDGES), smooth=smooth)


@pytest.mark.parametrize("n_wave, res, wave", [
    (400, 1.25, (4700.15, 9351.4)), (160, 1.25, (4700.15, 9351.4)),
    (1221, 6.2, (4700.15, 9351.4)), (1221, 1.25, (4700.15, 9351.4)),
    (1000, 1.25, (6000.0, 6080.0)), (1447, 1.25, (3400.0, 8519.0))])
def test_grids(rubix_lib, n_wave, res, wave):
    _check(_problem([3, 50, 0, 300, 700], ssp=(5, 3, n_wave), wave=wave, res=res))


@pytest.mark.parametrize("edit", [_hypervelocity, _spread, _not_finite, _outside])
def test_particles_of_the_general_path(rubix_lib, edit):
    _check(_problem([40, 30, 70, 0, 300, 5], edit=edit))


def test_adjoint_values_of_the_general_path(rubix_lib):
    """Spaxels whose adjoint is not finite, or so large that products may overflow."""

    def edit(adj):
        adj[1, 400] = np.nan
        adj[2, 10] = np.inf
        adj[4, 700] = 3e38
        adj[5] = 0.0

    _check(_problem([40, 30, 70, 0, 300, 5, 20]), edit_adj=edit)
