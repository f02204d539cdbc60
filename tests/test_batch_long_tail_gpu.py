"""BFS from many sources on graphs with more levels than the bit-parallel pass
keeps: what the call reports and what it costs."""
import ctypes as C

import numpy as np
import pytest

import belewitte_gb300 as bw
from belewitte_gb300 import _abi, batch

pytestmark = pytest.mark.gpu

CSR = bw.REP_FWD_CSR | bw.REP_REV_CSR


def _tailed(scale, edge_factor, tail, seed=3):
    """A symmetrised R-MAT graph with a path of `tail` vertices at its hub."""
    h = bw.HostGraph.rmat(scale, edge_factor, seed=seed, symmetrise=True)
    n = h.vertex_count
    src = np.repeat(np.arange(n, dtype=np.uint32), np.diff(h.fwd_vertices.astype(np.int64)))
    a = np.concatenate([[h.max_out_degree_vertex()], np.arange(n, n + tail - 1)]).astype(np.uint32)
    b = np.arange(n, n + tail, dtype=np.uint32)
    return bw.HostGraph.from_edges(n + tail, np.concatenate([src, a, b]), np.concatenate([h.fwd_edges, b, a]))


def _call(ctx, g, roots, order, levels):
    """One bw_batch_run; its result and the time between events around it."""
    import torch
    res = _abi.BatchResult()
    st = torch.cuda.current_stream()
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a.record()
    _abi.check(bw.library().bw_batch_run(ctx.handle, C.byref(g.view), batch.SOURCES, None, 1, roots.data_ptr(),
                                         None if order is None else order.data_ptr(),
                                         len(roots) if order is None else len(order), g.vertex_count, 0,
                                         levels.data_ptr(), None, None, C.byref(res), C.c_void_p(st.cuda_stream)),
               "bw_batch_run")
    b.record()
    torch.cuda.synchronize()
    return res, a.elapsed_time(b)


def test_device_ms_covers_the_whole_call(ctx):
    """device_ms is the call's time on the stream, a pass that could not finish
    included."""
    import torch
    h = _tailed(17, 8, 60)
    g = bw.DeviceGraph(h, reps=CSR)
    roots = torch.tensor([h.max_out_degree_vertex()], dtype=torch.int32, device="cuda")
    levels = torch.empty((1, h.vertex_count), dtype=torch.int32, device="cuda")
    share = []
    for _ in range(8):
        res, around = _call(ctx, g, roots, None, levels)
        share.append(res.device_ms / around)
    assert max(share) <= 1.01
    assert max(share) >= 0.75, share
