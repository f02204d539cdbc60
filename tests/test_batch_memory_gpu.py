"""Many sources on a graph whose words alone pass the bound of a pass's scratch:
the call runs, and what it took beyond the bound goes back to the device."""
import ctypes as C

import pytest

import belewitte_gb300 as bw
from belewitte_gb300 import _abi, batch

pytestmark = pytest.mark.gpu

BOUND = 24 << 30                     # bw_multisource.cu, MS_BYTES
N = 810_000_000                      # 32 bytes a vertex are more than that


def test_scratch_beyond_the_bound_is_given_back():
    import torch
    ctx = bw.Context(0)
    # 0 -> 1 -> 2 -> 3 -> N - 1
    fwd_e = torch.tensor([1, 2, 3, N - 1], dtype=torch.int32, device="cuda")
    rev_e = torch.tensor([0, 1, 2, 3], dtype=torch.int32, device="cuda")
    fwd_v = torch.full((N + 1,), 4, dtype=torch.int32, device="cuda")
    fwd_v[:4] = torch.arange(4, dtype=torch.int32, device="cuda")
    rev_v = torch.full((N + 1,), 3, dtype=torch.int32, device="cuda")
    rev_v[:4] = torch.tensor([0, 0, 1, 2], dtype=torch.int32, device="cuda")
    rev_v[N] = 4
    view = _abi.GraphView(N, 4, fwd_v.data_ptr(), fwd_e.data_ptr(), rev_v.data_ptr(), rev_e.data_ptr(), 0, 0, 0, 0)
    levels = torch.empty((1, N), dtype=torch.int32, device="cuda")
    root = torch.zeros(1, dtype=torch.int32, device="cuda")
    res = _abi.BatchResult()
    st = torch.cuda.current_stream()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    _abi.check(bw.library().bw_batch_run(ctx.handle, C.byref(view), batch.SOURCES, None, 1, root.data_ptr(), None, 1, N,
                                         0, levels.data_ptr(), None, None, C.byref(res), C.c_void_p(st.cuda_stream)),
               "bw_batch_run")
    torch.cuda.synchronize()
    kept = before - torch.cuda.mem_get_info()[0]
    path = [0, 1, 2, 3, N - 1]
    assert levels[0, path].tolist() == [0, 1, 2, 3, 4]
    assert int((levels == 2147483647).sum()) == N - 5
    assert res.traversed_edges == 4
    assert kept <= BOUND + (256 << 20), kept
    ctx.close()
    del fwd_v, rev_v, levels
    torch.cuda.empty_cache()
