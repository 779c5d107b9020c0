"""lsf_forward at the edges of its row kernel (12 outputs a thread, 3840 a round, several
rows a block), against a float64 convolution.  A sum of K products in float32, each
rounded once, is off by at most K 2^-24 sum |w x| (first order); 2 K covers the rest."""

import numpy as np
import pytest

from helpers import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [1, 4, 5, 25, 28, 29])
@pytest.mark.parametrize("n", [1, 11, 12, 13, 24, 3719, 3840, 3841, 4096])
def test_row_edges(rubix_lib, K, n):
    from rubix_gb300 import ops

    rng = np.random.default_rng(n * 31 + K)
    rows = 5 if n > 100 else 2000
    x = rng.normal(size=(rows, n)).astype(np.float32)
    w = rng.normal(size=K).astype(np.float32)
    for crop in {0, (K - 1) // 2, K - 1}:
        for taps in (w, to_dev(w)):
            got = ops.lsf_forward(to_dev(x), taps, crop).cpu().numpy()
            pick = rng.integers(0, rows, 4)
            for r in pick:
                ref = np.convolve(x[r].astype(np.float64), w.astype(np.float64))[crop:crop + n]
                mag = np.convolve(np.abs(x[r]).astype(np.float64),
                                  np.abs(w).astype(np.float64))[crop:crop + n]
                assert (np.abs(got[r] - ref) <= 2 * K * 2.0**-24 * mag + 1e-30).all()


def test_values_stay_in_their_row(rubix_lib):
    """A value that is not finite reaches the outputs of its own window only."""
    import torch

    from rubix_gb300 import ops

    x = torch.ones(700, 3721, device="cuda")
    x[3, 100] = float("inf")
    y = ops.lsf_forward(x, np.full(25, 0.04, np.float32), 12)
    bad = ~torch.isfinite(y)
    assert bad[3].any() and not bad[:3].any() and not bad[4:].any()
    assert not bad[3, :84].any() and not bad[3, 116:].any()
