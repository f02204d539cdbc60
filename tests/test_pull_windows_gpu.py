"""vertex-pull with the frontier's filter over uneven in-rows: 32 neighbouring
vertices with in-edge counts around a piece's, in one row or spread, rows cut by
a piece's end, rows already reached beside open ones; and what a skewed graph
costs against the plain kernel."""
import time

import numpy as np
import pytest

import belewitte_gb300 as bw
import oracle

pytestmark = pytest.mark.gpu

PIECE = 2048                         # bw_internal.cuh, FILTER_PIECE
MIN_EDGES = 4 << 20                  # bfs.cu, FILTERED_EDGES
VARIANTS = ["vertex-pull", "vertex-pull-bulk", "vertex-pull-warpreduce", "vertex-pull-blockreduce"]


def windows_graph(n, seed):
    """A quiet traversal through the windows that matter: a path 0, .. visits a
    row of each; a star on the way reaches all rows but one of a heavy window,
    whose last row comes later.  All other edges come from vertices that are
    never reached."""
    rng = np.random.default_rng(seed)
    last = (n - 1) // 32
    totals = [PIECE - 1, PIECE, PIECE + 1, 2 * PIECE, 2 * PIECE + 1, 5 * PIECE - 7, 40 * PIECE + 3, 3 * PIECE, 700_001, 3 * PIECE]
    ws = [0, 1, 2, 5, 40, 41, 42, 300, 301, last]
    lonely = lambda k: rng.integers(n // 2, 32 * last, k)              # sources that nothing reaches
    src, dst, path = [], [], [0]
    for i, (w, total) in enumerate(zip(ws, totals)):
        rows = 32 * w + np.arange(min(32, n - 32 * w))
        if i % 3 == 0:
            r = rng.choice(rows, total)                                # spread
        elif i % 3 == 1:
            r = np.concatenate([np.full(total - 20, rows[len(rows) // 2]), rng.choice(rows, 20)])      # one long row
        else:
            r = np.sort(rng.choice(rows[[0, 3, len(rows) - 1]], total))          # three, the last among them
        src.append(lonely(total))
        dst.append(r)
        path.append(int(rows[-1] if i % 2 else rows[len(rows) // 2]))
    star = 32 * 302 + np.arange(32)                                    # 31 rows reached together, the last one later
    src.append(lonely(64 * 3000))
    dst.append(np.concatenate([np.repeat(star[:31], 6000), np.full(6000, star[31])]))
    src.append(np.full(31, path[4])); dst.append(star[:31])
    path.append(int(star[31]))
    path += [n // 4 + 7 * k for k in range(8)]
    src.append(np.array(path[:-1])); dst.append(np.array(path[1:]))
    k = MIN_EDGES + 77 - sum(len(x) for x in src)
    src.append(lonely(k))
    dst.append(rng.integers(32 * 400, 32 * last, k))
    src, dst = np.concatenate(src), np.concatenate(dst)
    return bw.HostGraph.from_edges(n, src.astype(np.uint32), dst.astype(np.uint32), dedupe=False, drop_self_loops=False)


@pytest.mark.parametrize("n", [70_001, 70_016, 1_300_037])
def test_windows(ctx, n):
    h = windows_graph(n, n)
    assert h.edge_count >= MIN_EDGES
    g = bw.DeviceGraph(h, reps=bw.REP_FWD_CSR | bw.REP_REV_CSR)
    want, counts = oracle.bfs(n, h.fwd_vertices, h.fwd_edges, 0)
    assert len(counts) > 15 and max(counts) * 256 <= n
    for variant in VARIANTS:
        for loop, stats in (("host", False), ("graph", False), ("host", True), ("graph", True)):
            run = bw.bfs(ctx, g, variant, 0, loop=loop, stats=stats, tuned=False)
            assert np.array_equal(run.levels.cpu().numpy(), want), (variant, loop, stats)
            assert (run.level_count, run.visited) == (len(counts), (want != oracle.INF).sum())
            if stats:
                assert [s["frontier_vertices"] for s in run.level_stats] == list(counts)


@pytest.mark.parametrize("kind,args", [("rmat", dict(scale=20, edge_factor=16, symmetrise=True)),
                                       ("rmat_n", dict(n=300_007, edge_factor=30)), ("ba", dict(n=1_000_003, m=8))])
def test_skewed_graphs_are_not_slower(ctx, kind, args):
    """From the hub, whose out-neighbours end the plain kernel's scans early: the
    filter may take as long as the plain kernel (chosen by asking for a shape)
    and a third.  With 32 rows a warp at once it took 2 to 5 times as long."""
    import torch
    g = bw.DeviceGraph.generate(kind, seed=20, **args)
    root = int((g.fwd_vertices[1:] - g.fwd_vertices[:-1]).argmax().item())
    took = {}
    for name, shape in (("filter", {}), ("plain", dict(block=256, grid=8 * ctx.sm_count))):
        ts = []
        for _ in range(12):
            torch.cuda.synchronize()
            t = time.perf_counter()
            bw.bfs(ctx, g, "vertex-pull-bulk", root, tuned=False, **shape)
            ts.append(time.perf_counter() - t)
        took[name] = min(ts)
    print(took)
    assert took["filter"] <= 1.33 * took["plain"], took
