"""The traversed-edge total over vertex counts with every remainder of four,
depth arrays that are not 16-byte aligned, and PageRank into a rank array that
is not, against the oracle."""
import numpy as np
import pytest

import belewitte_gb300 as bw
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 4, 5, 1023, 50_002, 50_003])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_traversed_and_alignment(ctx, n, shift):
    import torch
    rng = np.random.default_rng(n)
    m = 4 * n + 8
    h = bw.HostGraph.from_edges(n, rng.integers(0, n, m, dtype=np.uint32), rng.integers(0, n, m, dtype=np.uint32),
                                dedupe=False, drop_self_loops=False)
    g = bw.DeviceGraph(h)
    want, counts = oracle.bfs(n, h.fwd_vertices, h.fwd_edges, 0)
    edges = int(np.diff(h.fwd_vertices.astype(np.int64))[want != oracle.INF].sum())
    room = torch.empty(n + shift, dtype=torch.int32, device="cuda")
    for variant in ("vertex-push", "vertex-pull-bulk", "edge-list", "frontier-push"):
        for loop in ("host", "graph"):
            run = bw.bfs(ctx, g, variant, 0, loop=loop, levels=room[shift:])
            assert np.array_equal(run.levels.cpu().numpy(), want), (variant, loop)
            assert (run.level_count, run.traversed_edges) == (len(counts), edges), (variant, loop)
    ranks = torch.empty(n + shift, dtype=torch.float32, device="cuda")
    exact, _ = oracle.pagerank(oracle.PR_DIV, n, h.rev_vertices, h.rev_edges, 4)
    got = bw.pagerank(ctx, g, "vertex-pull", 4, ranks=ranks[shift:]).ranks.cpu().numpy()
    assert np.array_equal(got.view(np.uint32), exact.view(np.uint32))
    f64 = oracle.pagerank_f64(oracle.PR_DIV, n, h.rev_vertices, h.rev_edges, 4)
    for variant in ("rev-edge-list", "vertex-push"):
        got = bw.pagerank(ctx, g, variant, 4, ranks=ranks[shift:]).ranks.cpu().numpy().astype(np.float64)
        assert float((np.abs(got - f64) / f64).max()) <= 1e-4, variant
