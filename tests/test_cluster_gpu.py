"""frontier-push's small-frontier kernel: frontiers around the lengths where
lists stay with their block, fill a step, and leave the kernel's caps; rows at
the length where a lane stops taking its own; lists that grow and shrink;
with and without level statistics, and under the learned switch."""
import numpy as np
import pytest

import belewitte_gb300 as bw
import oracle
from belewitte_gb300 import learn

pytestmark = pytest.mark.gpu

BLOCKS, KEEP, THREADS, LIST = 8, 256, 512, 4096


def layers(widths, degree):
    """Vertex 0, then layers of the given widths; the i-th vertex of a layer
    points at `degree` vertices of the next one, all of which are reached."""
    starts = 1 + np.concatenate([[0], np.cumsum(widths)])
    src, dst = [np.zeros(widths[0], np.int64)], [np.arange(1, 1 + widths[0])]
    for a, b, s, t in zip(widths[:-1], widths[1:], starts[:-1], starts[1:]):
        d = max(degree, -(-b // a))
        i = np.repeat(np.arange(a), d)
        k = np.tile(np.arange(d), a)
        src.append(s + i)
        dst.append(t + (i * b // a + k) % b)
    n = 1 + sum(widths)
    return bw.HostGraph.from_edges(n, np.concatenate(src).astype(np.uint32), np.concatenate(dst).astype(np.uint32))


def check(ctx, h):
    g = bw.DeviceGraph(h)
    want, counts = oracle.bfs(h.vertex_count, h.fwd_vertices, h.fwd_edges, 0)
    for stats in (False, True):
        run = bw.bfs(ctx, g, "frontier-push", 0, loop="graph", stats=stats)
        assert np.array_equal(run.levels.cpu().numpy(), want), stats
        assert (run.level_count, run.visited) == (len(counts), (want != oracle.INF).sum())
        if stats:
            assert [s["frontier_vertices"] for s in run.level_stats] == list(counts)
            deg = np.diff(h.fwd_vertices.astype(np.int64))
            edges = [int(deg[want == k + 1].sum()) for k in range(len(counts))]
            assert [s["frontier_edges"] for s in run.level_stats] == edges
    run = learn.run_learned(ctx, g, learn.load_predictor(), 0)
    assert np.array_equal(run.levels.cpu().numpy(), want)


@pytest.mark.parametrize("width", [1, KEEP - 1, KEEP, KEEP + 1, THREADS + 1, BLOCKS * KEEP - 1, BLOCKS * KEEP,
                                   BLOCKS * KEEP + 1, BLOCKS * THREADS + 1, 4 * THREADS * BLOCKS + 5,
                                   BLOCKS * LIST - 1, BLOCKS * LIST + 1])
def test_widths(ctx, width):
    check(ctx, layers([width] * 5, 1))


@pytest.mark.parametrize("degree", [3, 4, 5, 8, 33])
@pytest.mark.parametrize("width", [40, 700, 2100])
def test_degrees(ctx, degree, width):
    check(ctx, layers([width] * 6, degree))


@pytest.mark.parametrize("widths", [[1, 255, 1, 300, 2, 2100, 3, 5000, 1, 1],          # kept and shared in turn
                                    [5, 4096, 5, 4097, 5, 12000, 6],                   # one block's list, and past it
                                    [100, 40000, 100, 100, 40000, 7],                  # leaves the kernel and returns
                                    [3, 1023, 3, 3072, 1, 1024, 1, 1025, 1]])          # rows at the heavy limit
def test_growth(ctx, widths):
    check(ctx, layers(widths, 1))
