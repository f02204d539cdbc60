"""The reverse edge-list kernels' runs: edge counts around a lane's four edges,
a warp's 128 and its unrolled steps, runs that begin and end at every place of
a lane, streams that are not 16-byte aligned and streams in any order, against
the FP64 oracle."""
import numpy as np
import pytest

import belewitte_gb300 as bw
import oracle

pytestmark = pytest.mark.gpu

REL_F64 = 1e-4
VARIANTS = ["rev-edge-list", "rev-struct-edge-list"]


def close(run, want):
    got = run.ranks.cpu().numpy().astype(np.float64)
    return float((np.abs(got - want) / np.abs(want)).max()) <= REL_F64


def graph(m, n, seed):
    """m edges whose in-rows are 0 to 12 long, two of them of 300 edges."""
    rng = np.random.default_rng(seed)
    lengths = rng.integers(0, 13, n)
    lengths[rng.integers(0, n, 2)] = 300
    dst = np.repeat(np.arange(n), lengths)
    dst = np.concatenate([dst, rng.integers(0, n, m)])[:m]
    src = rng.integers(0, n, m)
    return bw.HostGraph.from_edges(n, src.astype(np.uint32), dst.astype(np.uint32), dedupe=False, drop_self_loops=False)


@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 31, 127, 128, 129, 255, 256, 257, 1023, 1025, 5000])
def test_edge_counts(ctx, m):
    n = max(3, m // 6)
    h = graph(m, n, m)
    assert h.edge_count == m
    g = bw.DeviceGraph(h)
    want = oracle.pagerank_f64(oracle.PR_DIV, n, h.rev_vertices, h.rev_edges, 5)
    for variant in VARIANTS:
        assert close(bw.pagerank(ctx, g, variant, 5), want), variant


@pytest.mark.parametrize("shift", [1, 2, 3])
@pytest.mark.parametrize("shuffled", [False, True])
def test_alignment_and_order(ctx, shift, shuffled):
    import torch
    n, m = 700, 4099
    h = graph(m, n, 17)
    g = bw.DeviceGraph(h)
    want = oracle.pagerank_f64(oracle.PR_DIV, n, h.rev_vertices, h.rev_edges, 5)
    order = torch.randperm(m, device="cuda") if shuffled else torch.arange(m, device="cuda")
    pairs = torch.stack([g.rev_in_edges[:m][order], g.rev_edges[:m][order]], 1).contiguous()

    def moved(t):
        """The same values `shift` words further on."""
        room = torch.zeros(t.numel() + shift, dtype=torch.int32, device="cuda")
        room[shift:] = t.reshape(-1)
        return room[shift:]
    dst, src = moved(pairs[:, 0]), moved(pairs[:, 1])
    g.view.rev_in_edges, g.view.rev_edges = dst.data_ptr(), src.data_ptr()
    assert close(bw.pagerank(ctx, g, "rev-edge-list", 5), want)
    if shift == 2:                               # pairs stay 8-byte aligned
        both = moved(pairs)
        g.view.rev_struct_edges = both.data_ptr()
        assert close(bw.pagerank(ctx, g, "rev-struct-edge-list", 5), want)


@pytest.mark.parametrize("m", [(24 << 20) - 1, (24 << 20) + 3])
def test_large(ctx, m):
    n = 1 << 20
    rng = np.random.default_rng(m)
    src, dst = rng.integers(0, n, m, dtype=np.uint32), np.sort(rng.integers(0, n, m, dtype=np.uint32))
    h = bw.HostGraph.from_edges(n, src, dst, dedupe=False, drop_self_loops=False)
    g = bw.DeviceGraph(h)
    want = oracle.pagerank_f64(oracle.PR_DIV, n, h.rev_vertices, h.rev_edges, 3)
    for variant in VARIANTS:
        assert close(bw.pagerank(ctx, g, variant, 3), want), variant


@pytest.mark.parametrize("n", [311295, 311296, 311297, 311299, 622593])
@pytest.mark.parametrize("variant", ["vertex-push", "vertex-push-warp", "edge-list", "rev-edge-list"])
def test_consolidation_sizes(ctx, n, variant):
    """Vertex counts around the consolidation's change to four vertices a
    thread (152 SMs x 8 blocks x 256 threads), every remainder of four."""
    rng = np.random.default_rng(n)
    m = 2 * n
    h = bw.HostGraph.from_edges(n, rng.integers(0, n, m, dtype=np.uint32), rng.integers(0, n, m, dtype=np.uint32))
    want = oracle.pagerank_f64(oracle.PR_DIV, n, h.rev_vertices, h.rev_edges, 4)
    assert close(bw.pagerank(ctx, bw.DeviceGraph(h), variant, 4), want)
