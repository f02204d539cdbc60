"""vertex-pull with the frontier's filter: vertex counts around the filter's
sizes (every vertex a bit, and folded), rows from none to thousands of edges,
a long quiet start, edge counts around the change, every reduction, both
loops, level statistics and mixed schedules, against the oracle."""
import numpy as np
import pytest

import belewitte_gb300 as bw
import oracle

pytestmark = pytest.mark.gpu

MIN_EDGES = 4 << 20
REDUCTIONS = ["vertex-pull", "vertex-pull-bulk", "vertex-pull-warpreduce", "vertex-pull-blockreduce"]


def chain_then_random(n, m, seed, hubs=0):
    """0 -> 1 -> ... -> 12, then m - 12 random edges among the vertices from 12
    on, in shuffled ids; the last third of the vertices has no edges in, and
    `hubs` vertices share a tenth of the edges in."""
    rng = np.random.default_rng(seed)
    k = m - 12
    live = 12 + max(1, (n - 12) * 2 // 3)
    src, dst = rng.integers(12, n, k), rng.integers(12, live, k)
    if hubs:
        dst[: k // 10] = 12 + rng.integers(0, hubs, k // 10)
    src[:3] = 12                                      # the chain's end reaches on
    src, dst = np.concatenate([np.arange(12), src]), np.concatenate([np.arange(1, 13), dst])
    ids = rng.permutation(n)
    h = bw.HostGraph.from_edges(n, ids[src].astype(np.uint32), ids[dst].astype(np.uint32), dedupe=False,
                                drop_self_loops=False)
    return h, int(ids[0])


def check(run, want, counts):
    assert np.array_equal(run.levels.cpu().numpy(), want)
    assert (run.level_count, run.visited) == (len(counts), (want != oracle.INF).sum())


@pytest.mark.parametrize("n,m,hubs", [((1 << 20) - 1, MIN_EDGES, 0), (1 << 20, MIN_EDGES + 3, 0), ((1 << 20) + 1, MIN_EDGES, 0),
                                      (2_600_000, 6_000_000, 5), (4096, MIN_EDGES, 0), (4097, MIN_EDGES + 1, 2),
                                      (70_001, 5_000_001, 40), (300_000, MIN_EDGES - 1, 0), (100, MIN_EDGES, 0)])
def test_sizes(ctx, n, m, hubs):
    h, root = chain_then_random(n, m, n + m, hubs)
    assert h.edge_count == m
    g = bw.DeviceGraph(h, reps=bw.REP_FWD_CSR | bw.REP_REV_CSR)
    want, counts = oracle.bfs(n, h.fwd_vertices, h.fwd_edges, root)
    for variant in REDUCTIONS:
        for loop in ("host", "graph"):
            check(bw.bfs(ctx, g, variant, root, loop=loop), want, counts)
    for loop in ("host", "graph"):
        run = bw.bfs(ctx, g, "vertex-pull-bulk", root, loop=loop, stats=True)
        check(run, want, counts)
        assert [s["frontier_vertices"] for s in run.level_stats] == list(counts)


def test_mixed_schedules(ctx):
    n = 1_500_000
    h, root = chain_then_random(n, 17_000_000, 3)
    g = bw.DeviceGraph(h)
    want, counts = oracle.bfs(n, h.fwd_vertices, h.fwd_edges, root)
    for schedule in (["vertex-pull", "frontier-push", "vertex-pull-bulk", "vertex-push"],
                     ["edge-list", "vertex-pull", "edge-list", "vertex-pull", "edge-list", "frontier-pull"],
                     ["vertex-pull"] * 10 + ["frontier-push", "vertex-pull"]):
        check(bw.bfs_schedule(ctx, g, schedule, root), want, counts)
