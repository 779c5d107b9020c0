"""Host-side choice between sums over SSP nodes and the general path (no GPU work)."""

import pytest

from rubix_gb300 import _lib

FULL = (6, 221, 1221)   # n_met, n_age, n_wave
COARSE = (6, 20, 1000)


@pytest.mark.parametrize("n, n_seg, n_t, grid, nodes", [
    # measured well apart: the node path 1.2 to 2.4 times as slow, or as fast
    (1, 1, 3721, FULL, 0), (100, 100, 3721, FULL, 0), (1000, 256, 3721, FULL, 0),
    (3000, 256, 3721, COARSE, 0), (10_000, 1024, 3721, FULL, 0), (10_000, 4096, 700, FULL, 0),
    (30_000, 4096, 3721, FULL, 0), (3000, 10_000, 700, FULL, 0),
    (1000, 1, 3721, FULL, 1), (30_000, 625, 3721, FULL, 1), (300_000, 4096, 3721, FULL, 1),
    (3000, 10_000, 700, (5, 50, 1450), 1), (3000, 10_000, 3721, COARSE, 1),
    (1000, 40_000, 3721, COARSE, 1),
    (100_000, 40_000, 700, FULL, 1), (1_000_000, 22_500, 3721, FULL, 1),
    (10_000_000, 90_000, 3721, FULL, 1), (333_337, 4489, 2049, (5, 53, 1447), 1),
])
def test_forward_path(rubix_lib, n, n_seg, n_t, grid, nodes):
    sizes = (n, n_seg, n_t, *grid)
    assert _lib.query("rubix_cube_fwd_path", *sizes) == nodes
    general = _lib.query("rubix_cube_general_workspace_size", *sizes)
    ws = _lib.query("rubix_cube_workspace_size", *sizes)
    if not nodes:
        assert ws == general
    launches = [_lib.query("rubix_cube_fwd_launches", *sizes, path, 1 << 40) for path in range(3)]
    assert launches[0] == launches[2 if nodes else 1] and launches[2] > launches[1]


@pytest.mark.parametrize("n, n_seg, n_t, grid, nodes", [
    (100, 100, 3721, FULL, 0), (1000, 256, 3721, FULL, 0), (1000, 4096, 2000, COARSE, 0),
    (3000, 4096, 3721, FULL, 0),
    (3000, 256, 700, COARSE, 1), (10_000, 4096, 3721, COARSE, 1), (10_000, 625, 3721, COARSE, 1),
    (200_000, 2500, 3721, FULL, 1), (30_000, 4096, 3721, FULL, 1), (1000, 22_500, 3721, FULL, 1),
])
def test_adjoint_path(rubix_lib, n, n_seg, n_t, grid, nodes):
    sizes = (n, n_seg, n_t, *grid)
    a, b = (_lib.query("rubix_cube_bwd_launches", *sizes, dust, 1 << 40) for dust in (0, 1))
    assert (a > b) == bool(nodes)


def test_monotonic(rubix_lib):
    """More stars never lead back to the general path; an empty call has no node path."""
    for n_seg in (1, 300, 2500, 11_000, 40_000):
        paths = [_lib.query("rubix_cube_fwd_path", n, n_seg, 3721, *FULL)
                 for n in (0, 10, 100, 1000, 10_000, 100_000, 1_000_000, 10_000_000)]
        assert paths == sorted(paths) and paths[0] == 0 and paths[-1] == 1
    assert _lib.query("rubix_cube_fwd_path", 1000, 0, 3721, *FULL) == 0
