"""Which path a call takes by its sizes, and the node path on few stars and in workspaces that
hold half its rows (two waves)."""

import numpy as np
import pytest

import test_gpu_nodes as T
import test_gpu_nodes_bwd as B
from helpers import to_dev
from node_path import force_nodes, least_workspace
from rubix_gb300 import telescope as tel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("edit", [T._hypervelocity, T._spread, T._not_finite, T._outside,
                                  T._extreme])
def test_particles_of_the_general_path(rubix_lib, monkeypatch, edit):
    force_nodes(monkeypatch)
    T.test_particles_of_the_general_path(rubix_lib, edit)


@pytest.mark.parametrize("case", ["short", "fine", "flat", "inf", "zero"])
def test_grids_of_the_general_path(rubix_lib, monkeypatch, case):
    force_nodes(monkeypatch)
    T.test_grids_of_the_general_path(rubix_lib, case)


def test_dust_outliers(rubix_lib, monkeypatch):
    force_nodes(monkeypatch)
    T.test_dust_outliers(rubix_lib)


@pytest.mark.parametrize("counts", [[1], [0, 3, 1], [1] * 40])
def test_few_stars(rubix_lib, monkeypatch, counts):
    """By sizes the general path, bit for bit; forced, the node path to rounding."""
    prob = T._problem(counts)
    b = T._run(rubix_lib, prob, True)
    assert np.array_equal(T._run(rubix_lib, prob, False), b)
    force_nodes(monkeypatch)
    a = T._compare(rubix_lib, prob)
    assert not np.array_equal(a, b)


def test_parts_of_a_batch(rubix_lib):
    """A part rendered by itself takes the path of the batch whose size it is given."""
    from rubix_gb300 import ops

    counts = [700, 3, 0, 900, 1]
    s, wz, wt, p, offs = T._problem(counts)
    grid = [to_dev(a) for a in (s.flux, s.metallicity, s.age, wz, wt)]

    def run(i0, i1, segs, **kw):
        star = [to_dev(p[k][i0:i1]) for k in ("mass", "metallicity", "age", "vel")]
        perm = to_dev(np.arange(i1 - i0, dtype=np.int32))
        off = to_dev((offs[segs[0]:segs[1] + 1] - i0).astype(np.int32))
        return ops.cube_forward(*grid, *star, 0, perm, off, segs[1] - segs[0], **kw).cpu().numpy()

    whole = run(0, int(offs[-1]), (0, 5))
    sizes = (int(offs[-1]), 5)
    for seg in (0, 1, 3, 4):
        part = run(int(offs[seg]), int(offs[seg + 1]), (seg, seg + 1), sizes=sizes)
        assert np.array_equal(part[0], whole[seg])
    one = run(int(offs[1]), int(offs[2]), (1, 2))
    assert np.array_equal(one, run(int(offs[1]), int(offs[2]), (1, 2), general=True))
    assert not np.array_equal(one[0], whole[1])


MANY = T.EDGES + [5, 0, 17] * 200  # more spaxels than the fewest that a wave takes


def _fast(counts):
    offs = np.concatenate([[0], np.cumsum(counts)])

    def edit(p, rng):
        for s in range(0, len(counts), 11):
            if counts[s]:
                p["vel"][offs[s]] = 5000.0

    return edit


@pytest.mark.parametrize("lsf", [None, 25])
@pytest.mark.parametrize("fast", [False, True])
@pytest.mark.parametrize("dust", [False, True])
def test_two_waves_forward(rubix_lib, monkeypatch, lsf, fast, dust):
    """The rows of half the spaxels at a time: the same bits."""
    from rubix_gb300 import _lib

    prob = T._problem(MANY, edit=_fast(MANY) if fast else None)
    taps = None if lsf is None else tel.gaussian_taps_1d(lsf, 1.3)
    av = np.random.default_rng(3).exponential(0.5, prob[3]["mass"].size) if dust else None
    used = []

    def size(name, sizes):
        used.append((sizes, least_workspace(name, sizes)))
        return used[-1][1]

    with monkeypatch.context() as m:
        force_nodes(m)
        whole = T._run(rubix_lib, prob, False, taps, av)
    with monkeypatch.context() as m:
        force_nodes(m, size)
        parts = T._run(rubix_lib, prob, False, taps, av)
    sizes, least = used[-1]
    full = _lib.query("rubix_cube_nodes_workspace_size", *sizes)
    n = [_lib.query("rubix_cube_fwd_launches", *sizes, 2, b) for b in (full, least)]
    assert least < full and n[1] == n[0] + 2
    assert np.array_equal(whole, parts)
    general = T._run(rubix_lib, prob, True, taps, av)
    scale = np.maximum(np.abs(general).max(1, keepdims=True), 1e-30)
    assert (np.abs(whole - general) / scale).max() <= T.TOL


@pytest.mark.parametrize("fast", [False, True])
@pytest.mark.parametrize("bad_adj", [False, True])
def test_two_waves_adjoint(rubix_lib, monkeypatch, fast, bad_adj):
    """Half the stars at a time: the same bits; spaxels that straddle the waves, and flags that
    a later wave sets after an earlier one has written gradients."""
    from rubix_gb300 import _lib

    prob = T._problem(MANY, edit=_fast(MANY) if fast else None)
    n = prob[3]["mass"].size
    assert n > 8192
    adj = np.random.default_rng(1).normal(size=(len(MANY), prob[2].size)).astype(np.float32)
    if bad_adj:
        adj[21, 900] = 3e38  # a spaxel of 2600 stars: in its last slice only
        adj[400, 3] = np.nan
    used = []

    def size(name, sizes):
        used.append((sizes, least_workspace(name, sizes)))
        return used[-1][1]

    whole = B._grads(prob, adj, False)
    with monkeypatch.context() as m:
        force_nodes(m, size)
        parts = B._grads(prob, adj, False)
    sizes, least = used[-1]
    full = _lib.query("rubix_cube_bwd_workspace_size", *sizes)
    k = [_lib.query("rubix_cube_bwd_launches", *sizes, 0, b) for b in (full, least)]
    assert least < full and k[1] == k[0] + 2
    for a, b in zip(whole, parts):
        assert np.array_equal(a, b, equal_nan=True)
