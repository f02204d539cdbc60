"""A call refused for want of memory: the next one on the same context and
thread runs."""
import ctypes as C

import numpy as np
import pytest

import belewitte_gb300 as bw
import oracle

pytestmark = pytest.mark.gpu


def test_the_next_call_runs():
    import torch
    h = bw.HostGraph.rmat(10, 8, seed=3)
    want, _ = oracle.bfs(h.vertex_count, h.fwd_vertices, h.fwd_edges, 1)
    ctx = bw.Context(0)
    g = bw.DeviceGraph(h)
    levels = torch.empty(h.vertex_count, dtype=torch.int32, device="cuda")
    st = torch.cuda.current_stream()
    for first_use in (True, False):
        # the scratch for 2^40 vertices (4 TiB a queue) is refused before anything runs
        rc = bw.library().bw_bfs_init(ctx.handle, 1 << 40, 1, levels.data_ptr(), C.c_void_p(st.cuda_stream))
        assert rc == 5, rc                                  # BW_ERR_OUT_OF_MEMORY
        got = bw.bfs(ctx, g, "vertex-push", 1).levels.cpu().numpy()
        assert np.array_equal(got, want), first_use
    ctx.close()
