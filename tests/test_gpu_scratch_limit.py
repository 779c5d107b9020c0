"""Calls on a device that has room for the general path's workspace but not for the node
path's: rendered and differentiated by the general path, as before there was another."""

import numpy as np
import pytest

import test_gpu_nodes_bwd as B
from helpers import to_dev
from test_gpu_nodes import TOL, _problem

pytestmark = pytest.mark.gpu


@pytest.fixture
def little_memory(monkeypatch):
    """ops.workspace that fails, as the allocator does, beyond a limit set by the test."""
    import torch

    from rubix_gb300 import ops

    real, state = ops.workspace, dict(limit=None, refused=0)

    def workspace(nbytes, device):
        if state["limit"] is not None and nbytes > state["limit"]:
            state["refused"] += 1
            raise torch.OutOfMemoryError("CUDA out of memory")
        return real(nbytes, device)

    monkeypatch.setattr(ops, "workspace", workspace)
    return state


def _forward(prob, **kw):
    from rubix_gb300 import ops

    s, wz, wt, p, offs = prob
    n = p["mass"].size
    return ops.cube_forward(*[to_dev(a) for a in (s.flux, s.metallicity, s.age, wz, wt, p["mass"],
                                                  p["metallicity"], p["age"], p["vel"])], 0,
                            to_dev(np.arange(n, dtype=np.int32)), to_dev(offs), offs.size - 1,
                            check=True, **kw)


@pytest.mark.parametrize("sizes", [None, (10**6, 10)])
def test_forward(rubix_lib, little_memory, sizes):
    import torch

    from rubix_gb300 import _lib

    prob = _problem([300, 900, 0, 40] * 20)
    n, L = prob[3]["mass"].size, prob[2].size
    whole, general = _forward(prob), _forward(prob, general=True)
    little_memory["limit"] = _lib.query("rubix_cube_general_workspace_size", n, 80, L,
                                        *prob[0].flux.shape)
    got = _forward(prob, sizes=sizes)
    assert little_memory["refused"] == 1
    assert torch.equal(got, general) and not torch.equal(got, whole)
    little_memory["limit"] -= 1
    with pytest.raises(torch.OutOfMemoryError):
        _forward(prob)


def test_adjoint(rubix_lib, little_memory):
    from rubix_gb300 import _lib

    prob = _problem([300, 900, 0, 40] * 20)
    n, L = prob[3]["mass"].size, prob[2].size
    adj = np.random.default_rng(1).normal(size=(80, L)).astype(np.float32)
    whole = B._grads(prob, adj, False)
    little_memory["limit"] = _lib.query("rubix_cube_general_workspace_size", n, 80, L,
                                        *prob[0].flux.shape)
    got = B._grads(prob, adj, False)
    assert little_memory["refused"] == 1
    for a, b in zip(whole, got):
        assert np.sqrt(np.mean((a - b) ** 2)) <= TOL * np.sqrt(np.mean(b ** 2))
