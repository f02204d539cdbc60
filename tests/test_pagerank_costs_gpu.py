"""What PageRank iterations cost next to one another on the same graph: the
shares that rounding, rows without in-edges and chained launches may take."""
import pytest

import belewitte_gb300 as bw

pytestmark = pytest.mark.gpu


def _timed(ctx, g, variant, **kw):
    """The least time of each of four iterations, launched one by one."""
    runs = [bw.pagerank_schedule(ctx, g, [variant], 4, time_iterations=True, **kw).iteration_ms for _ in range(5)]
    return [min(t) for t in zip(*runs)]


@pytest.fixture(scope="module")
def web():
    return bw.DeviceGraph.generate("rmat_n", n=8_000_009, edge_factor=8, seed=22)


def test_rows_without_in_edges(ctx, web):
    """The first two iterations also write the rows without in-edges, two thirds
    of this graph's: a sixth more than the others (a branch of single lanes in
    their rounding made it twice as much)."""
    t = _timed(ctx, web, "vertex-pull", relabel=False)
    print(t)
    assert max(t[0], t[1]) <= 1.5 * t[2], t


def test_rounding_beside_the_warp_sums(ctx, web):
    """vertex-pull-warp with the divided contributions takes what it takes
    without (1.29 times as long when lanes rounded by themselves)."""
    div, nodiv = min(_timed(ctx, web, "vertex-pull-warp")), min(_timed(ctx, web, "vertex-pull-warp-nodiv"))
    print(div, nodiv)
    assert div <= 1.15 * nodiv, (div, nodiv)


@pytest.mark.parametrize("variant", ["vertex-pull-warp", "vertex-pull-warp-nodiv", "vertex-push-warp"])
def test_chained_launches_on_a_skewed_graph(ctx, variant):
    """30 iterations launched as a chain take no longer than the same ones
    launched one by one (up to 1.25 times as long when the next kernel's blocks
    gathered on the SMs that were free first)."""
    g = bw.DeviceGraph.generate("ba", n=300_007, m=20, seed=8)
    chain = min(bw.pagerank(ctx, g, variant, 30).device_ms for _ in range(6)) / 30
    single = min(_timed(ctx, g, variant))
    print(chain, single)
    assert chain <= 1.08 * single, (chain, single)
