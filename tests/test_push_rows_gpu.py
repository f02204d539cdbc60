"""The push kernels' row handling: rows around the 256-edge cut, warps whose
32 rows mix empty, short and cut ones, targets shared by many rows, and queue
lengths around one row a warp and 32 rows a warp, against the oracle."""
import numpy as np
import pytest

import belewitte_gb300 as bw
import oracle

pytestmark = pytest.mark.gpu

PUSH = ["vertex-push", "vertex-push-bulk", "vertex-push-warp", "frontier-push"]


def two_levels(degrees, shared):
    """Root 0 -> one vertex per entry of `degrees`; vertex i then points at
    degrees[i] leaves, its own ones or (`shared`) the same first ones."""
    degrees = np.asarray(degrees, np.int64)
    k = len(degrees)
    first = 1 + k
    starts = np.zeros(k, np.int64) if shared else np.concatenate([[0], np.cumsum(degrees)[:-1]])
    src = np.repeat(np.arange(1, k + 1), degrees)
    within = np.arange(degrees.sum()) - np.repeat(np.cumsum(degrees) - degrees, degrees)
    dst = first + np.repeat(starts, degrees) + within
    n = int(max(first + 1, dst.max(initial=0) + 1))
    src = np.concatenate([np.zeros(k, np.int64), src]).astype(np.uint32)
    dst = np.concatenate([np.arange(1, k + 1), dst]).astype(np.uint32)
    return bw.HostGraph.from_edges(n, src, dst)


ROWS = {
    "one-edge": [1] * 40,
    "empty-then-one": [0] * 31 + [1] + [0] * 32 + [3],
    "around-the-cut": [255, 256, 257, 0, 511, 512, 513, 1, 0],
    "cut-rows-only": [257] * 33,
    "around-a-step": [127, 1, 128, 0, 129, 31, 32, 33] * 5,
    "mixed": [0, 1, 300, 7, 0, 0, 64, 1025, 33, 2] * 13,
    "warp-of-full-rows": [256] * 32,
    "last-row-empty": [5] * 31 + [0],
}


@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("rows", list(ROWS))
def test_rows(ctx, rows, shared):
    h = two_levels(ROWS[rows], shared)
    g = bw.DeviceGraph(h)
    want, counts = oracle.bfs(h.vertex_count, h.fwd_vertices, h.fwd_edges, 0)
    for variant in PUSH:
        for loop in ("host", "graph"):
            for stats in (False, True):
                run = bw.bfs(ctx, g, variant, 0, loop=loop, stats=stats)
                assert np.array_equal(run.levels.cpu().numpy(), want), (variant, loop, stats)
                assert (run.level_count, run.visited) == (len(counts), (want != oracle.INF).sum()), (variant, loop, stats)


@pytest.mark.parametrize("queue", [1, 31, 32, 33, 9727, 9728, 9729, 40000])
def test_queue_lengths(ctx, queue):
    """152 SMs x 64 warps = 9728: at most one row a warp up to there."""
    rng = np.random.default_rng(queue)
    h = two_levels(rng.integers(0, 6, queue), shared=False)
    g = bw.DeviceGraph(h)
    want, counts = oracle.bfs(h.vertex_count, h.fwd_vertices, h.fwd_edges, 0)
    for variant in PUSH:
        for loop in ("host", "graph"):
            run = bw.bfs(ctx, g, variant, 0, loop=loop)
            assert np.array_equal(run.levels.cpu().numpy(), want), (variant, loop)
            assert run.visited == (want != oracle.INF).sum()
