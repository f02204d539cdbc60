"""edge-list BFS by chunks with source ranges: edge counts around the change
and around a chunk, quiet levels (a chain behind a random graph), sources with
wide gaps, lists in any order, every reduction, both loops, and schedules that
change variants on the way, against the oracle."""
import numpy as np
import pytest

import belewitte_gb300 as bw
import oracle

pytestmark = pytest.mark.gpu

MIN_EDGES = 16 << 20
CHAIN = 20
REDUCTIONS = ["edge-list", "edge-list-bulk", "edge-list-warpreduce", "edge-list-blockreduce"]


def random_and_chain(m, gap=1):
    """m edges: a random graph on 300,000 vertices (`gap` apart in id), then a
    chain from its last one, a chain that ends in the last vertex."""
    rng = np.random.default_rng(m + gap)
    n0 = 300_000
    k = m - CHAIN
    src = np.sort(rng.integers(0, n0, k, dtype=np.int64))
    dst = rng.integers(0, n0, k, dtype=np.int64)
    chain = n0 - 1 + np.arange(CHAIN + 1)
    src, dst = np.concatenate([src, chain[:-1]]), np.concatenate([dst, chain[1:]])
    n = (n0 + CHAIN) * gap
    return bw.HostGraph.from_edges(n, (src * gap).astype(np.uint32), (dst * gap).astype(np.uint32),
                                   dedupe=False, drop_self_loops=False)


def check(run, want, counts):
    assert np.array_equal(run.levels.cpu().numpy(), want)
    assert (run.level_count, run.visited) == (len(counts), (want != oracle.INF).sum())


@pytest.mark.parametrize("m", [MIN_EDGES - 1, MIN_EDGES, MIN_EDGES + 1, MIN_EDGES + 1023, MIN_EDGES + 1026])
def test_edge_counts(ctx, m):
    h = random_and_chain(m)
    assert h.edge_count == m
    g = bw.DeviceGraph(h, reps=bw.REP_FWD_CSR | bw.REP_FWD_EL)
    want, counts = oracle.bfs(h.vertex_count, h.fwd_vertices, h.fwd_edges, 5)
    for variant in REDUCTIONS:
        for loop in ("host", "graph"):
            check(bw.bfs(ctx, g, variant, 5, loop=loop), want, counts)
    run = bw.bfs(ctx, g, REDUCTIONS[1], 5, loop="graph", stats=True)
    check(run, want, counts)
    assert [s["frontier_vertices"] for s in run.level_stats] == list(counts)
    last = h.vertex_count - 1                    # no edges: one level
    want, counts = oracle.bfs(h.vertex_count, h.fwd_vertices, h.fwd_edges, last)
    check(bw.bfs(ctx, g, REDUCTIONS[1], last), want, counts)


@pytest.mark.parametrize("gap", [7, 40])
def test_gaps(ctx, gap):
    h = random_and_chain(MIN_EDGES + 77, gap)
    g = bw.DeviceGraph(h, reps=bw.REP_FWD_CSR | bw.REP_FWD_EL)
    want, counts = oracle.bfs(h.vertex_count, h.fwd_vertices, h.fwd_edges, 0)
    for loop in ("host", "graph"):
        check(bw.bfs(ctx, g, "edge-list-bulk", 0, loop=loop), want, counts)


@pytest.mark.parametrize("shift", [0, 1])
def test_any_order_and_alignment(ctx, shift):
    import torch
    h = random_and_chain(MIN_EDGES + 5)
    m = h.edge_count
    g = bw.DeviceGraph(h, reps=bw.REP_FWD_CSR | bw.REP_FWD_EL)
    want, counts = oracle.bfs(h.vertex_count, h.fwd_vertices, h.fwd_edges, 5)
    order = torch.randperm(m, device="cuda")
    order[:m // 2] = order[:m // 2].sort().values          # half in order, half not
    src, dst = (torch.cat([torch.zeros(shift, dtype=torch.int32, device="cuda"), t[:m][order]])
                for t in (g.fwd_in_edges, g.fwd_edges))
    g.view.fwd_in_edges, g.view.fwd_edges = src[shift:].data_ptr(), dst[shift:].data_ptr()
    for loop in ("host", "graph"):
        check(bw.bfs(ctx, g, "edge-list-bulk", 5, loop=loop), want, counts)


def test_mixed_schedules(ctx):
    h = random_and_chain(MIN_EDGES + 13)
    g = bw.DeviceGraph(h)
    want, counts = oracle.bfs(h.vertex_count, h.fwd_vertices, h.fwd_edges, 5)
    for schedule in (["edge-list", "vertex-push", "edge-list"], ["vertex-push", "frontier-push", "edge-list-bulk"],
                     ["edge-list", "rev-edge-list", "struct-edge-list", "edge-list", "frontier-push", "edge-list"]):
        check(bw.bfs_schedule(ctx, g, schedule, 5), want, counts)
