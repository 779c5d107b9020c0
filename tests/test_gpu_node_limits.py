"""Stars at the edge of the node path's velocity range, in a workspace that an earlier call on
other templates has left its tables in.  Tolerance: that of test_gpu_nodes.py."""

import numpy as np
import pytest

from helpers import to_dev
from test_gpu_nodes import TOL, _problem

pytestmark = pytest.mark.gpu

ALPHA_LIMIT = 2040.0 / 2**18  # |alpha - 1| that the table over the Doppler factor covers


@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_velocity_limit_alone(rubix_lib, monkeypatch, sign):
    """One star at a time, its velocity in steps of one float around the limit."""
    import torch

    from rubix_gb300 import ops

    s, wz, wt, p, offs = _problem([1], ssp=(5, 3, 400))
    v = np.full(1, np.log1p(sign * ALPHA_LIMIT) * 299792.458, np.float32)
    around = [v]
    for way in (np.float32(1e9), np.float32(-1e9)):
        x = v
        for _ in range(40):
            x = np.nextafter(x, way)
            around.append(x)
    kept = {}

    def workspace(nbytes, device):
        if nbytes not in kept:
            kept[nbytes] = torch.zeros(max(int(nbytes), 256), dtype=torch.uint8, device=device)
        return kept[nbytes]

    monkeypatch.setattr(ops, "workspace", workspace)
    flux, met, age, wzd, wtd = (to_dev(a) for a in (s.flux, s.metallicity, s.age, wz, wt))

    def render(flux, vel, general):
        n = vel.size
        star = [to_dev(np.repeat(p[k], n)) for k in ("mass", "metallicity", "age")]
        return ops.cube_forward(flux, met, age, wzd, wtd, *star, to_dev(vel), 0,
                                to_dev(np.arange(n, dtype=np.int32)),
                                to_dev(np.array([0, n], np.int32)), 1, general=general,
                                sizes=None if general else (10**6, 1))

    for vel in around:
        render(2.0 * flux, np.array([sign * 2320.0], np.float32), False)  # leaves its tables
        a = render(flux, vel, False).cpu().numpy()
        b = render(flux, vel, True).cpu().numpy()
        assert np.abs(a - b).max() <= TOL * np.abs(b).max(), float(vel[0])
