"""bw_batch_run over many sources with an explicit unit order: the units that
`order` names run, into their own rows; the others' rows stay as they were."""
import ctypes as C

import numpy as np
import pytest

import belewitte_gb300 as bw
import oracle
from belewitte_gb300 import _abi, batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5000, 98305], ids=["a CTA per source", "together"])
@pytest.mark.parametrize("units,order", [(40, "reversed"), (7, [5, 0, 3]), (1100, "every other")])
def test_units_named_by_order(ctx, n, units, order):
    import torch
    h = bw.HostGraph.rmat_n(n, 8, seed=6)
    g = bw.DeviceGraph(h, reps=bw.REP_FWD_CSR | bw.REP_REV_CSR)
    rng = np.random.default_rng(units)
    few = rng.choice(n, 20, replace=False)
    roots = few[rng.integers(0, 20, units)].astype(np.int32)
    if order == "reversed":
        order = list(range(units))[::-1]
    elif order == "every other":
        order = list(range(1, units, 2)) + list(range(0, units - 50, 2))      # past one pass; 25 units left out
    levels = torch.full((units, n), -7, dtype=torch.int32, device="cuda")
    d_roots = torch.from_numpy(roots).cuda()
    d_order = torch.tensor(order, dtype=torch.int32, device="cuda")
    res = _abi.BatchResult()
    st = torch.cuda.current_stream()
    _abi.check(bw.library().bw_batch_run(ctx.handle, C.byref(g.view), batch.SOURCES, None, 1, d_roots.data_ptr(),
                                         d_order.data_ptr(), len(order), n, 0, levels.data_ptr(), None, None,
                                         C.byref(res), C.c_void_p(st.cuda_stream)), "bw_batch_run")
    got = levels.cpu().numpy()
    deg = h.out_degrees().astype(np.int64)
    want = {int(r): oracle.bfs(n, h.fwd_vertices, h.fwd_edges, int(r))[0] for r in few}
    named = set(order)
    total = 0
    for u in range(units):
        if u in named:
            d = want[int(roots[u])]
            assert np.array_equal(got[u], d), u
            total += int(deg[d != oracle.INF].sum())
        else:
            assert (got[u] == -7).all(), u
    assert res.units == len(order) and res.traversed_edges == total
