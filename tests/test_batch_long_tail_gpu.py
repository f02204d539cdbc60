"""BFS from many sources on graphs with more levels than the bit-parallel pass
keeps: their depths, what the call reports and what it costs."""
import ctypes as C

import numpy as np
import pytest

import belewitte_gb300 as bw
import oracle
from belewitte_gb300 import _abi, batch

pytestmark = pytest.mark.gpu

CSR = bw.REP_FWD_CSR | bw.REP_REV_CSR


def _tailed(scale, edge_factor, tail, seed=3):
    """A symmetrised R-MAT graph with a path of `tail` vertices at its hub."""
    h = bw.HostGraph.rmat(scale, edge_factor, seed=seed, symmetrise=True)
    n = h.vertex_count
    src = np.repeat(np.arange(n, dtype=np.uint32), np.diff(h.fwd_vertices.astype(np.int64)))
    a = np.concatenate([[h.max_out_degree_vertex()], np.arange(n, n + tail - 1)]).astype(np.uint32)
    b = np.arange(n, n + tail, dtype=np.uint32)
    return bw.HostGraph.from_edges(n + tail, np.concatenate([src, a, b]), np.concatenate([h.fwd_edges, b, a]))


def _call(ctx, g, roots, order, levels):
    """One bw_batch_run; its result and the time between events around it."""
    import torch
    res = _abi.BatchResult()
    st = torch.cuda.current_stream()
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a.record()
    _abi.check(bw.library().bw_batch_run(ctx.handle, C.byref(g.view), batch.SOURCES, None, 1, roots.data_ptr(),
                                         None if order is None else order.data_ptr(),
                                         len(roots) if order is None else len(order), g.vertex_count, 0,
                                         levels.data_ptr(), None, None, C.byref(res), C.c_void_p(st.cuda_stream)),
               "bw_batch_run")
    b.record()
    torch.cuda.synchronize()
    return res, a.elapsed_time(b)


def test_device_ms_covers_the_whole_call(ctx):
    """device_ms is the call's time on the stream, a pass that could not finish
    included."""
    import torch
    h = _tailed(17, 8, 60)
    g = bw.DeviceGraph(h, reps=CSR)
    roots = torch.tensor([h.max_out_degree_vertex()], dtype=torch.int32, device="cuda")
    levels = torch.empty((1, h.vertex_count), dtype=torch.int32, device="cuda")
    share = []
    for _ in range(8):
        res, around = _call(ctx, g, roots, None, levels)
        share.append(res.device_ms / around)
    assert max(share) <= 1.01
    assert max(share) >= 0.75, share


def _check(ctx, h, sources):
    """Depths, units and traversed edges of one call against the oracle."""
    import torch
    g = bw.DeviceGraph(h, reps=CSR)
    levels = torch.full((len(sources), h.vertex_count), -7, dtype=torch.int32, device="cuda")
    res, _ = _call(ctx, g, torch.tensor(sources, dtype=torch.int32, device="cuda"), None, levels)
    deg = h.out_degrees().astype(np.int64)
    want, total = {}, 0
    for k, s in enumerate(sources):
        if s not in want:
            want[s] = oracle.bfs(h.vertex_count, h.fwd_vertices, h.fwd_edges, s)[0]
        assert np.array_equal(levels[k].cpu().numpy(), want[s]), (k, s)
        total += int(deg[want[s] != oracle.INF].sum())
    assert res.units == len(sources) and res.traversed_edges == total


@pytest.mark.parametrize("tail", [29, 30, 31, 32, 33, 61, 200])
def test_levels_around_the_planes(ctx, tail):
    """From the hub the last level is `tail`, from the path's end a few more,
    from its middle the frontier is one vertex for long."""
    h = _tailed(17, 8, tail)
    n = h.vertex_count
    rng = np.random.default_rng(tail)
    _check(ctx, h, [h.max_out_degree_vertex(), n - 1, n - tail // 2] + [int(v) for v in rng.integers(0, n, 37)])


def test_more_vertices_than_the_visited_bitmap(ctx):
    """Going on without the shared-memory bitmap."""
    h = _tailed(21, 2, 50)
    _check(ctx, h, [h.max_out_degree_vertex(), h.vertex_count - 1, 5])


def test_passes_that_end_differently(ctx):
    """Three passes: sources whose component is done in a few levels, sources of
    one with a long path, and the first kind again."""
    a, b = bw.HostGraph.rmat(16, 8, seed=1, symmetrise=True), _tailed(16, 8, 70)
    n = a.vertex_count
    rows = [np.repeat(np.arange(h.vertex_count, dtype=np.uint32), np.diff(h.fwd_vertices.astype(np.int64))) for h in (a, b)]
    h = bw.HostGraph.from_edges(n + b.vertex_count, np.concatenate([rows[0], rows[1] + np.uint32(n)]),
                                np.concatenate([a.fwd_edges, b.fwd_edges + np.uint32(n)]))
    rng = np.random.default_rng(2)
    short, long_ = [int(v) for v in rng.integers(0, n, 30)], [int(n + v) for v in rng.integers(0, b.vertex_count, 30)]
    pick = lambda of, k: [of[i] for i in rng.integers(0, 30, k)]
    _check(ctx, h, pick(short, 1024) + pick(long_, 1024) + pick(short, 17))


@pytest.mark.parametrize("name,count", [("grid", 1030), ("chain", 3)])
def test_meshes(ctx, name, count):
    """Passes that end early, the next ones never begun."""
    h = bw.HostGraph.grid(331, 301) if name == "grid" else bw.HostGraph.from_edges(98400, np.arange(98399), np.arange(1, 98400))
    few = [0, h.vertex_count - 1] + [int(v) for v in np.random.default_rng(1).integers(0, h.vertex_count, 18)]
    _check(ctx, h, [few[i % 20] for i in range(count)])


def test_a_long_path_costs_its_levels(ctx):
    """512 sources on a graph with and without a path of 60 vertices: the pass up
    to the planes' end is kept, so the call takes at most four times as long (a
    pass thrown away and a CTA per source from the root take more than six)."""
    import torch
    took = []
    for h in (bw.HostGraph.rmat(18, 16, seed=3, symmetrise=True), _tailed(18, 16, 60)):
        g = bw.DeviceGraph(h, reps=CSR)
        roots = torch.from_numpy(np.random.default_rng(4).integers(0, h.vertex_count, 512).astype(np.int32)).cuda()
        levels = torch.empty((512, h.vertex_count), dtype=torch.int32, device="cuda")
        took.append(min(_call(ctx, g, roots, None, levels)[1] for _ in range(6)))
    print(took)
    assert took[1] <= 4 * took[0], took


def test_a_short_path_before_the_graph(ctx):
    """One source at the end of a path of 6 and one at the hub the path leads
    to: the path adds its few levels to the traversal, which stays
    bit-parallel (given back after four levels it took 3.6 times as long)."""
    import torch
    h = _tailed(19, 16, 6)
    g = bw.DeviceGraph(h, reps=CSR)
    levels = torch.empty((1, h.vertex_count), dtype=torch.int32, device="cuda")
    took = []
    for source in (h.max_out_degree_vertex(), h.vertex_count - 1):
        root = torch.tensor([source], dtype=torch.int32, device="cuda")
        took.append(min(_call(ctx, g, root, None, levels)[1] for _ in range(8)))
    print(took)
    assert took[1] <= 2.5 * took[0], took
