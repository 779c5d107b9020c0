"""The gradient arrays of the adjoint are independent allocations: rubix_cube_bwd clears each by
itself, and ops.cube_backward returns tensors that share nothing."""

import ctypes

import numpy as np
import pytest

from helpers import to_dev
from test_gpu_nodes import _problem

pytestmark = pytest.mark.gpu


class _MemsetParams(ctypes.Structure):  # CUDA_MEMSET_NODE_PARAMS
    _fields_ = [("dst", ctypes.c_uint64), ("pitch", ctypes.c_size_t), ("value", ctypes.c_uint),
                ("element", ctypes.c_uint), ("width", ctypes.c_size_t),
                ("height", ctypes.c_size_t)]


def _memsets(graph):
    """(first byte, bytes) of every memset node of a captured graph."""
    drv = ctypes.CDLL("libcuda.so.1")
    g, n = ctypes.c_void_p(graph), ctypes.c_size_t(0)
    assert drv.cuGraphGetNodes(g, None, ctypes.byref(n)) == 0
    nodes = (ctypes.c_void_p * n.value)()
    assert drv.cuGraphGetNodes(g, nodes, ctypes.byref(n)) == 0
    out = []
    for node in nodes:
        kind, p = ctypes.c_int(-1), _MemsetParams()
        assert drv.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
        if kind.value == 2:  # CU_GRAPH_NODE_TYPE_MEMSET
            assert drv.cuGraphMemsetNodeGetParams(ctypes.c_void_p(node), ctypes.byref(p)) == 0
            out.append((p.dst, p.element * p.width * max(p.height, 1)))
    return out


def _args(prob, adj):
    s, wz, wt, p, offs = prob
    n, nseg = p["mass"].size, offs.size - 1
    return [*(to_dev(a) for a in (s.flux, s.metallicity, s.age, wz, wt, p["mass"],
                                  p["metallicity"], p["age"], p["vel"])),
            0, to_dev(np.arange(n, dtype=np.int32)), to_dev(offs), nseg, adj]


def test_no_clear_spans_two_arrays(rubix_lib):
    """Four arrays that happen to follow one another in memory, as separate allocations may."""
    import torch

    from rubix_gb300 import _lib

    prob = _problem([40, 24])  # 64 stars: arrays of 256 bytes
    s, wz, wt, p, offs = prob
    nz, na, nw = s.flux.shape
    n, L = p["mass"].size, wt.size
    d = [to_dev(a) for a in (s.flux, s.metallicity, s.age, wz, wt, p["mass"], p["metallicity"],
                             p["age"], p["vel"])]
    perm, off, adj = to_dev(np.arange(n, dtype=np.int32)), to_dev(offs), torch.ones(2, L).cuda()
    size = _lib.query("rubix_cube_bwd_workspace_size", n, 2, L, nz, na, nw)
    ws = torch.zeros(size, dtype=torch.uint8, device="cuda")
    grads = torch.full((4, n), float("nan"), device="cuda")
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        _lib.call("rubix_cube_bwd", *[t.data_ptr() for t in d[:4]], nz, na, nw, d[4].data_ptr(), L,
                  *[t.data_ptr() for t in d[5:9]], 1, 0, perm.data_ptr(), off.data_ptr(), 2, n,
                  adj.data_ptr(), L, *[grads[i].data_ptr() for i in range(4)], ws.data_ptr(),
                  size, torch.cuda.current_stream().cuda_stream)
    for first, count in _memsets(graph.raw_cuda_graph()):
        for i in range(4):
            a = grads[i].data_ptr()
            if a <= first < a + 4 * n:
                assert first + count <= a + 4 * n
    graph.instantiate()
    graph.replay()
    assert torch.isfinite(grads).all() and grads[0].abs().min() > 0


def test_unsorted_stars_have_zero_gradients(rubix_lib):
    """Arrays of odd sizes; the last stars are in no spaxel."""
    import torch

    from rubix_gb300 import ops

    prob = _problem([3, 0, 34])
    args = _args(prob, torch.ones(3, prob[2].size).cuda())
    args[11] = to_dev(np.array([0, 3, 3, 30], np.int32))
    for g in ops.cube_backward(*args):
        assert g[:30].abs().min() > 0 and not g[30:].any()


def test_gradients_are_tensors_of_their_own(rubix_lib):
    import torch

    from rubix_gb300 import ops

    prob = _problem([3, 0, 34])
    grads = ops.cube_backward(*_args(prob, torch.ones(3, prob[2].size).cuda()))
    assert len({g.untyped_storage().data_ptr() for g in grads}) == 4
    versions = [g._version for g in grads]
    grads[0].mul_(2.0)
    assert [g._version for g in grads[1:]] == versions[1:]
    scale = torch.ones((), device="cuda", requires_grad=True)
    grads[1].mul_(scale)  # views of one unbind would refuse this
    assert grads[1].requires_grad
