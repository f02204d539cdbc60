"""The device loop's two parts (rounds the host launches, then a CUDA graph):
traversals that end just before, at and after the change, and level limits
there, for a fixed variant and for the learned switch."""
import numpy as np
import pytest

import belewitte_gb300 as bw
import oracle
from belewitte_gb300 import learn
from graphs import chain

pytestmark = pytest.mark.gpu

AROUND = [1, 2, 46, 47, 48, 49, 50, 51, 120]


@pytest.mark.parametrize("n", AROUND)
@pytest.mark.parametrize("variant", ["vertex-push", "edge-list-blockreduce", "frontier-pull", "frontier-push"])
def test_levels_around_the_change(ctx, n, variant):
    h = chain(n)
    g = bw.DeviceGraph(h)
    want, counts = oracle.bfs(n, h.fwd_vertices, h.fwd_edges, 0)
    for stats in (False, True):
        run = bw.bfs(ctx, g, variant, 0, loop="graph", stats=stats)
        assert np.array_equal(run.levels.cpu().numpy(), want)
        assert (run.level_count, run.visited, run.traversed_edges) == (len(counts), n, n - 1)
        if stats:
            assert [s["frontier_vertices"] for s in run.level_stats] == list(counts)


@pytest.mark.parametrize("n", AROUND)
@pytest.mark.parametrize("mlp_only", [False, True])
def test_learned_levels_around_the_change(ctx, n, mlp_only):
    h = chain(n)
    g = bw.DeviceGraph(h)
    want, counts = oracle.bfs(n, h.fwd_vertices, h.fwd_edges, 0)
    run = learn.run_learned(ctx, g, learn.load_predictor(), 0, mlp_only=mlp_only)
    assert np.array_equal(run.levels.cpu().numpy(), want)
    assert (run.level_count, run.visited, run.traversed_edges) == (len(counts), n, n - 1)
    assert [s["frontier_vertices"] for s in run.level_stats] == list(counts)


@pytest.mark.parametrize("limit", [1, 47, 48, 49, 60])
def test_level_limit_around_the_change(ctx, limit):
    g = bw.DeviceGraph(chain(200))
    for loop in ("host", "graph"):
        with pytest.raises(bw.BwError):
            bw.bfs(ctx, g, "vertex-pull-bulk", 0, loop=loop, max_levels=limit)
    run = bw.bfs(ctx, g, "vertex-pull-bulk", 0, loop="graph")
    assert run.level_count == 200
