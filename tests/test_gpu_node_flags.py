"""Spaxels that the node path leaves to the general kernel: found, listed and rendered as
rubix_cube_fwd_general renders them, whatever shares the call, with the caller's work items."""

import numpy as np
import pytest

from node_path import force_nodes
from test_gpu_nodes import TOL, _problem, _run
from test_gpu_nodes_bwd import _check

pytestmark = pytest.mark.gpu

# counts around the ends of the general kernel's chunks, of the node path's items, and many
COUNTS = ([0, 1, 63, 64, 65, 255, 256, 257, 1023, 1024, 1025, 2600] + [7] * 400 + [1300, 1, 40])


def _flag(counts, which, speed=9000.0):
    """One fast star in each spaxel of `which`."""
    offs = np.concatenate([[0], np.cumsum(counts)])

    def edit(p, rng):
        for s in which:
            if counts[s]:
                p["vel"][offs[s] + counts[s] // 2] = speed

    return edit


@pytest.mark.parametrize("which", ["few", "most", "last"])
@pytest.mark.parametrize("chunk", [32, 64, 256])
def test_flagged_spaxels_are_the_general_kernels(rubix_lib, which, chunk):
    """Bit for bit on the flagged spaxels, for every chunk; to rounding on the others."""
    from rubix_gb300 import autotune

    ids = dict(few=[2, 11, 200], last=[len(COUNTS) - 1],
               most=[s for s in range(len(COUNTS)) if s % 7])[which]
    prob = _problem(COUNTS, edit=_flag(COUNTS, ids))
    autotune.set_tuning(0, chunk=chunk)
    try:
        a, b = _run(rubix_lib, prob, False), _run(rubix_lib, prob, True)
    finally:
        autotune.set_tuning(0)
    assert np.array_equal(a[ids], b[ids])
    scale = np.maximum(np.abs(b).max(1, keepdims=True), 1e-30)
    assert (np.abs(a - b) / scale).max() <= TOL
    rest = [s for s in range(len(COUNTS)) if s not in ids and COUNTS[s] > 1]
    assert not np.array_equal(a[rest], b[rest])  # the node path has rendered the others


@pytest.mark.parametrize("which", [[2, 11, 200], [s for s in range(len(COUNTS)) if s % 7]])
def test_adjoint_of_flagged_spaxels(rubix_lib, which):
    _check(_problem(COUNTS, edit=_flag(COUNTS, which)))


@pytest.mark.parametrize("n_seg, per", [(40, 30), (9000, 5)])
@pytest.mark.parametrize("sigma", [400.0, 1500.0])
def test_wide_velocities(rubix_lib, monkeypatch, n_seg, per, sigma):
    """Some or nearly all spaxels ruled out by their velocities before there are work items; one
    block or several make those.  Slow stars' spaxels do not depend on the others."""
    rng = np.random.default_rng(4)
    counts = rng.poisson(per, n_seg)
    counts[0], counts[1] = 0, 1500
    offs = np.concatenate([[0], np.cumsum(counts)])
    slow = np.arange(n_seg) % 10 == 3

    def edit(p, rng):
        p["vel"] = np.where(np.repeat(slow, counts), rng.normal(0, 60.0, offs[-1]),
                            rng.normal(0, sigma, offs[-1]))

    force_nodes(monkeypatch)
    prob = _problem(counts, ssp=(5, 3, 400), edit=edit)
    a, b = _run(rubix_lib, prob, False), _run(rubix_lib, prob, True)
    scale = np.maximum(np.abs(b).max(1, keepdims=True), 1e-30)
    assert (np.abs(a - b) / scale).max() <= TOL
    keep = np.repeat(slow, counts)
    s, wz, wt, p, _ = prob
    alone = (s, wz, wt, {k: v[keep] for k, v in p.items()},
             np.concatenate([[0], np.cumsum(counts[slow])]).astype(np.int32))
    c = _run(rubix_lib, alone, False)
    assert np.array_equal(a[slow], c)
    assert not np.array_equal(a[slow], b[slow])


def test_wide_velocities_adjoint(rubix_lib):
    def edit(p, rng):
        p["vel"] = rng.normal(0, 1500.0, p["vel"].size)

    _check(_problem([40, 0, 1, 300, 700, 3], edit=edit))
