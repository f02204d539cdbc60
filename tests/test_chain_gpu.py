"""A run's kernels launched as a chain, each while the one before it runs and
waiting on the device, give what the same kernels give when every iteration or
level is timed, and so launched after the one before it has ended."""
import numpy as np
import pytest

import belewitte_gb300 as bw

pytestmark = pytest.mark.gpu

EXACT = ("vertex-pull", "vertex-pull-nodiv", "pull-segmented")
REL = 1e-5                           # float atomics: the order of the additions differs from run to run


@pytest.fixture(scope="module")
def chain_graphs():
    hosts = [bw.HostGraph.rmat(14, 16, seed=7), bw.HostGraph.grid(61, 67), bw.HostGraph.rmat_n(50021, 20, seed=3)]
    return [(h, bw.DeviceGraph(h)) for h in hosts]


@pytest.mark.parametrize("variant", bw.pagerank_variant_names())
def test_pagerank(ctx, chain_graphs, variant):
    for _, g in chain_graphs:
        want = bw.pagerank_schedule(ctx, g, [variant], 12, time_iterations=True).ranks.cpu().numpy()
        for loop in ("host", "graph"):
            got = bw.pagerank(ctx, g, variant, 12, loop=loop).ranks.cpu().numpy()
            if variant in EXACT:
                assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), loop
            else:
                rel = np.abs(got.astype(np.float64) - want) / want
                assert rel.max() <= REL, (loop, rel.max())


@pytest.mark.parametrize("variant", ["edge-list-bulk", "rev-struct-edge-list", "vertex-push", "vertex-pull-blockreduce",
                                     "vertex-push-warp", "vertex-pull-warp", "frontier-push", "frontier-pull"])
def test_bfs(ctx, chain_graphs, variant):
    for h, g in chain_graphs:
        root = h.max_out_degree_vertex()
        want = bw.bfs_schedule(ctx, g, [variant], root, time_levels=True)
        for loop in ("host", "graph"):
            got = bw.bfs(ctx, g, variant, root, loop=loop)
            assert got.level_count == want.level_count and got.visited == want.visited, loop
            assert np.array_equal(got.levels.cpu().numpy(), want.levels.cpu().numpy()), loop
