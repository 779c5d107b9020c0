"""spaxel_sort and spaxel_assign where their dispatches change: digits of 1 to 9 bits and one
to four passes, more and fewer segments than keys, gaps between the occupied segments, and
bin edges that are uniform, uneven, repeated or not ascending.  Whole numbers: exact."""

import numpy as np
import pytest

from helpers import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_seg", [1, 2, 255, 256, 511, 512, 513, 1023, 131071, 262143, 262144,
                                   (1 << 27) - 1])
@pytest.mark.parametrize("n", [1, 4095, 4097, 200_003])
def test_sort(rubix_lib, n, n_seg):
    import torch

    from rubix_gb300 import ops

    rng = np.random.default_rng(n + n_seg)
    hi = min(n_seg + 2, n_seg // 3 + 5)  # some beyond the last segment, a gap at the end
    idx = rng.integers(-1, hi, n).astype(np.int32)
    keep = (rng.random(n) < 0.9).astype(np.uint8)
    perm, offs = ops.spaxel_sort(to_dev(idx), n_seg, to_dev(keep))
    key = np.where((idx >= 0) & (idx < n_seg) & (keep > 0), idx, n_seg).astype(np.int64)
    order = np.argsort(key, kind="stable")
    assert np.array_equal(perm.cpu().numpy(), order)
    want = torch.searchsorted(torch.as_tensor(key[order]), torch.arange(min(n_seg, 300_000) + 1))
    assert np.array_equal(offs[:want.numel()].cpu().numpy(), want.numpy())
    assert int(offs[n_seg]) == int((key < n_seg).sum())


@pytest.mark.parametrize("kind", ["uniform", "uneven", "repeated", "flat", "falling", "two"])
def test_assign(rubix_lib, kind):
    from rubix_gb300 import ops

    e = {"uniform": np.linspace(-7.3, 7.3, 301), "uneven": np.geomspace(0.01, 20.0, 77),
         "repeated": np.repeat(np.linspace(-2, 2, 9), 3), "flat": np.zeros(5),
         "falling": np.linspace(5, -5, 33), "two": np.array([-1.0, 1.0])}[kind].astype(np.float32)
    rng = np.random.default_rng(2)
    x = rng.uniform(-9, 25, (40_000, 3)).astype(np.float32)
    x[:e.size, 0] = e
    x[:e.size, 1] = np.nextafter(e, np.float32(-np.inf))
    x[-4:, 0] = [np.inf, -np.inf, np.nan, 3e38]
    got = ops.spaxel_assign(to_dev(x), to_dev(e)).cpu().numpy()

    def bins(v):  # the search of the general case, element by element
        lo, hi = np.zeros(v.size, np.int64), np.full(v.size, e.size)
        while (lo < hi).any():
            mid = np.minimum((lo + hi) >> 1, e.size - 1)
            le, on = e[mid] <= v, lo < hi
            lo, hi = np.where(on & le, mid + 1, lo), np.where(on & ~le, mid, hi)
        lo = np.where(np.isnan(v), e.size, lo)
        return np.clip(lo - 1, 0, e.size - 2)

    assert np.array_equal(got, bins(x[:, 0]) + (e.size - 1) * bins(x[:, 1]))
