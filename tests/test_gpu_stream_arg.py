"""The wrappers take a device in every form that torch.cuda.current_stream does."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("device", ["cuda", "cuda:0", 0, None])
def test_psf_status_device(rubix_lib, device):
    import torch

    from rubix_gb300 import ops

    assert ops.psf_status(device) == 0
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        assert ops._stream(device) == side.cuda_stream
