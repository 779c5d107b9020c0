"""The layers where the choice between their kernels changes: LSF rows by length and taps, PSF
cubes by waves of strips, edges even or not, sorts by keys and segments."""

import numpy as np
import pytest

import test_gpu_lsf_rows as lsf
import test_gpu_psf_pair as psf
from helpers import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [12, 13, 25, 28])
@pytest.mark.parametrize("n", [599, 600, 980, 981, 1048, 1049, 1400, 1401])
def test_lsf_rows(rubix_lib, K, n):
    lsf.test_row_edges(rubix_lib, K, n)


@pytest.mark.parametrize("m", [1, 3, 7, 11, 15])
@pytest.mark.parametrize("ny, nx, nl, pad", [
    (17, 33, 8001, 0), (1, 1, 14001, 0), (40, 31, 14801, 0), (33, 161, 2305, 1),  # packed pairs
    (3, 129, 2561, 1), (32, 250, 2431, 0),  # 205 of 304 blocks; 304
    (31, 250, 2431, 0)])                    # two waves of few rows
def test_psf_strips(rubix_lib, m, ny, nx, nl, pad):
    psf.test_bits(rubix_lib, m, ny, nx, nl, pad)


def _bins(e, v):
    return np.clip(np.searchsorted(e, v, side="right") - 1, 0, e.size - 2)


@pytest.mark.parametrize("n_edges", [2, 23, 24, 25, 301, 9000])
@pytest.mark.parametrize("shift", [0.0, 0.45, 0.55, 3.0])
def test_assign_edges(rubix_lib, n_edges, shift):
    """Few and many edges (in and beyond shared memory), one of them off its even place by part
    of a step, up to past its neighbours' places."""
    import torch

    from rubix_gb300 import ops

    step = 0.37
    e = ((np.arange(n_edges) - n_edges / 2) * step).astype(np.float32)
    if n_edges > 2:
        e[n_edges // 2] += np.float32(shift * step)
        e = np.sort(e)
    rng = np.random.default_rng(n_edges)
    x = rng.uniform(e[0] - 1, e[-1] + 1, (20_000, 3)).astype(np.float32)
    k = min(e.size, 9000)
    x[:k, 0] = e[:k]
    x[:k, 1] = np.nextafter(e[:k], np.float32(np.inf))
    x[k:2 * k, 0] = np.nextafter(e[:k], np.float32(-np.inf))
    got = ops.spaxel_assign(to_dev(x), to_dev(e)).cpu().numpy()
    assert np.array_equal(got, _bins(e, x[:, 0]) + (e.size - 1) * _bins(e, x[:, 1]))
    idx, mask = ops.assign_and_mask(to_dev(x), to_dev(e))
    assert np.array_equal(idx.cpu().numpy(), got)
    assert torch.equal(mask, ops.aperture_mask(to_dev(x), to_dev(e)))


@pytest.mark.parametrize("n", [1 << 19, (1 << 19) + 1])
@pytest.mark.parametrize("n_seg", [1023, 1024, 262_143])
def test_sort_offsets(rubix_lib, n, n_seg):
    """Offsets by the pass over the keys and by search, with gaps."""
    from rubix_gb300 import ops

    rng = np.random.default_rng(n_seg)
    idx = (rng.integers(0, n_seg // 7 + 1, n) * 7).astype(np.int32)
    perm, offs = ops.spaxel_sort(to_dev(idx), n_seg)
    key = np.where(idx < n_seg, idx, n_seg)
    assert np.array_equal(perm.cpu().numpy(), np.argsort(key, kind="stable"))
    count = np.bincount(key, minlength=n_seg + 1)[:n_seg]
    assert np.array_equal(offs.cpu().numpy(), np.concatenate([[0], np.cumsum(count)]))
