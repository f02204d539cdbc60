"""The batched launch's PageRank over packed graphs as one set of rows, where
it can go wrong: graphs at the dispatch's size line, rows at the edges of the
long-row classes, a graph of one vertex, graphs without in-edges between
others, and vertices that belong to no graph."""
import ctypes as C

import numpy as np
import pytest

import belewitte_gb300 as bw
import oracle
from belewitte_gb300 import _abi, batch
from graphs import chain, star, star_in

pytestmark = pytest.mark.gpu


def _rows(lengths, n):
    """Vertex i has lengths[i] in-edges, from the lowest other vertices."""
    src, dst = [], []
    for v, d in enumerate(lengths):
        s = [u for u in range(d + 1) if u != v][:d]
        src += s
        dst += [v] * d
    return bw.HostGraph.from_edges(n, src, dst)


def _hosts(largest):
    return [bw.HostGraph.rmat_n(1500, 20, seed=3), bw.HostGraph.from_edges(1, [], []), star_in(3000), chain(40),
            bw.HostGraph.from_edges(3, [0], [1]), _rows([255, 256, 257, 511, 512, 513, 1023, 2047, 2048, 2049, 2600], 2700),
            bw.HostGraph.rmat_n(largest, 16, seed=9), star(70)]


@pytest.mark.parametrize("largest,iterations", [(4095, 6), (4096, 1), (4096, 4), (9001, 2), (9001, 20)])
def test_ranks_match_each_graph_alone(ctx, largest, iterations):
    hosts = _hosts(largest)
    packed = batch.pack([bw.DeviceGraph(h, reps=bw.REP_FWD_CSR | bw.REP_REV_CSR) for h in hosts])
    levels, ranks, res = batch.run_graphs(ctx, packed, pr_iterations=iterations)
    offs = packed.offsets.cpu().numpy().astype(np.int64)
    roots = packed.roots.cpu().numpy().astype(np.int64)
    for i, h in enumerate(hosts):
        lo, hi = offs[i], offs[i + 1]
        want, _ = oracle.bfs(h.vertex_count, h.fwd_vertices, h.fwd_edges, int(roots[i] - lo))
        assert np.array_equal(levels[lo:hi].cpu().numpy(), want), i
        pr, _ = oracle.pagerank(oracle.PR_DIV, h.vertex_count, h.rev_vertices, h.rev_edges, iterations)
        assert np.array_equal(ranks[lo:hi].cpu().numpy().view(np.uint32), pr.view(np.uint32)), i


def test_vertices_of_no_graph_keep_their_ranks(ctx):
    """A view whose first and last graphs are left out of the offsets."""
    import torch
    hosts = _hosts(5000)
    packed = batch.pack([bw.DeviceGraph(h, reps=bw.REP_FWD_CSR | bw.REP_REV_CSR) for h in hosts])
    n, cut = packed.vertex_count, len(hosts) - 2
    offsets, roots = packed.offsets[1:-1].contiguous(), packed.roots[1:-1].contiguous()
    levels = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    ranks = torch.full((n,), -7.0, dtype=torch.float32, device="cuda")
    res = _abi.BatchResult()
    st = torch.cuda.current_stream()
    bw._abi.check(bw.library().bw_batch_run(ctx.handle, C.byref(packed.view), batch.GRAPHS, offsets.data_ptr(), cut,
                                            roots.data_ptr(), None, cut, 5000, 5, levels.data_ptr(), ranks.data_ptr(),
                                            None, C.byref(res), C.c_void_p(st.cuda_stream)), "bw_batch_run")
    offs = packed.offsets.cpu().numpy().astype(np.int64)
    got = ranks.cpu().numpy()
    assert (got[:offs[1]] == -7.0).all() and (got[offs[-2]:] == -7.0).all()
    for i in range(1, len(hosts) - 1):
        h = hosts[i]
        pr, _ = oracle.pagerank(oracle.PR_DIV, h.vertex_count, h.rev_vertices, h.rev_edges, 5)
        assert np.array_equal(got[offs[i]:offs[i + 1]].view(np.uint32), pr.view(np.uint32)), i
