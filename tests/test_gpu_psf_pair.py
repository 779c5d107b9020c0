"""The packed-pair PSF kernel (equal taps, enough strips to fill the chip) against the other
PSF kernels, which a second copy of the device taps selects: the same products in the same
order, so bit-identical.  Ragged strips and wavelength tiles, fewer rows than taps, spaxel
strides with and without 16-byte rows."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 3, 5, 7, 9, 11, 13, 15])
@pytest.mark.parametrize("ny, nx, nl, pad", [(3, 150, 3721, 0), (3, 150, 3721, 3), (17, 33, 6401, 0),
                                             (1, 1, 12000, 0), (40, 31, 12801, 3),
                                             (16, 129, 2560, 0), (9, 161, 2049, 1)])
def test_bits(rubix_lib, m, ny, nx, nl, pad):
    import torch

    from rubix_gb300 import ops

    g = torch.Generator("cuda").manual_seed(m + ny)
    cube = torch.randn(ny, nx, nl + pad, generator=g, device="cuda")[:, :, :nl]
    taps = np.random.default_rng(m).normal(size=m).astype(np.float32)
    t = torch.as_tensor(taps, device="cuda")
    want = ops.psf_forward(cube, t, t.clone())
    assert torch.equal(ops.psf_forward(cube, t), want)
    assert torch.equal(ops.psf_forward(cube, taps), want)
    assert ops.psf_status() == 0
