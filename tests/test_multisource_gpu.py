"""BFS from many sources with a bit per source and vertex (bw_batch_run),
where it can go wrong: source counts around the word and pass sizes, vertex
counts off the multiples of 32, rows around the chunk length, hubs, sources
that meet, directed graphs, and graphs with more levels than it keeps (given
back to the per-source kernel).  Against the oracle, depth for depth."""
import numpy as np
import pytest

import belewitte_gb300 as bw
import oracle
from belewitte_gb300 import batch
from graphs import chain, star, star_in

pytestmark = pytest.mark.gpu

CSR = bw.REP_FWD_CSR | bw.REP_REV_CSR


def _hub_rows(n):
    """In-rows of 127, 128, 129, 257 and 1025 edges from low vertices, and one
    hub; a ring connects everything."""
    src, dst = list(range(n)), [(i + 1) % n for i in range(n)]
    for k, d in enumerate([127, 128, 129, 257, 1025]):
        src += list(range(10, 10 + d))
        dst += [n - 1 - 40 * k] * d            # 40 vertices apart: other warps' batches
    src += [0] * (n // 3)
    dst += list(range(5, 5 + n // 3))
    return bw.HostGraph.from_edges(n, src, dst)


GRAPHS = {
    "rmat_sym": lambda: bw.HostGraph.rmat(17, 8, seed=8, symmetrise=True),
    "rmat_ragged": lambda: bw.HostGraph.rmat_n(98305, 12, seed=5),
    "rmat_small": lambda: bw.HostGraph.rmat_n(98303, 12, seed=5),      # below the dispatch's line
    "er_directed": lambda: bw.HostGraph.erdos_renyi(100003, 400000, seed=4),
    "hubs": lambda: _hub_rows(100007),
    "star_in": lambda: star_in(100000),
    "star": lambda: star(100001),
    "chain": lambda: chain(98400),
    "grid": lambda: bw.HostGraph.grid(331, 301),
}


@pytest.fixture(scope="module")
def built():
    made = {}

    def get(name):
        if name not in made:
            h = GRAPHS[name]()
            made[name] = (h, bw.DeviceGraph(h, reps=CSR))
        return made[name]
    return get


def _check(ctx, h, g, sources):
    levels, res = batch.run_sources(ctx, g, sources)
    got = levels.cpu().numpy()
    deg = h.out_degrees().astype(np.int64)
    seen = {}
    total = 0
    for k, s in enumerate(sources):
        if s not in seen:
            seen[s], _ = oracle.bfs(h.vertex_count, h.fwd_vertices, h.fwd_edges, int(s))
        want = seen[s]
        assert np.array_equal(got[k], want), (k, s)
        total += int(deg[want != oracle.INF].sum())
    assert res.units == len(sources) and res.traversed_edges == total


@pytest.mark.parametrize("count", [1, 2, 31, 32, 33, 64, 65, 129, 257, 513, 1024, 1025])
def test_source_counts(ctx, built, count):
    h, g = built("rmat_ragged" if count % 2 else "rmat_sym")
    rng = np.random.default_rng(count)
    few = rng.choice(h.vertex_count, 60, replace=False)          # sources repeat
    _check(ctx, h, g, [int(few[i]) for i in rng.integers(0, 60, count)])


@pytest.mark.parametrize("name", sorted(GRAPHS))
@pytest.mark.parametrize("count", [3, 40])
def test_graph_shapes(ctx, built, name, count):
    h, g = built(name)
    rng = np.random.default_rng(count)
    n = h.vertex_count
    _check(ctx, h, g, [0, n - 1, int(n // 2)] + [int(v) for v in rng.integers(0, n, count - 3)])


def test_without_the_reverse_csr(ctx, built):
    """A caller that holds only the forward CSR keeps the per-source kernel."""
    import ctypes as C

    import torch
    from belewitte_gb300 import _abi
    h, g = built("rmat_sym")
    v = g.view
    view = _abi.GraphView(v.vertex_count, v.edge_count, v.fwd_vertices, v.fwd_edges, 0, 0, 0, 0, 0, 0)
    roots = torch.tensor([5, 77, 5], dtype=torch.int32, device="cuda")
    levels = torch.empty((3, h.vertex_count), dtype=torch.int32, device="cuda")
    res = _abi.BatchResult()
    st = torch.cuda.current_stream()
    _abi.check(bw.library().bw_batch_run(ctx.handle, C.byref(view), batch.SOURCES, None, 1, roots.data_ptr(), None, 3,
                                         h.vertex_count, 0, levels.data_ptr(), None, None, C.byref(res),
                                         C.c_void_p(st.cuda_stream)), "bw_batch_run")
    for k, s in enumerate([5, 77, 5]):
        want, _ = oracle.bfs(h.vertex_count, h.fwd_vertices, h.fwd_edges, s)
        assert np.array_equal(levels[k].cpu().numpy(), want)
