"""Long-row sums at the lengths where their path changes (batch rows, giant
rows, pieces of 512 edges) and at the edge counts where the giant-row length
does: bit-exact against the oracle."""
import numpy as np
import pytest

import belewitte_gb300 as bw
import oracle

pytestmark = pytest.mark.gpu

MEGA = 1 << 20
N = 1 << 17
LENGTHS = [0, 1, 31, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 1535, 1536, 1537, 2047, 2048, 2049,
           4095, 4096, 4097, 8191, 8192, 8193, 16 * 512, 32 * 512 + 1, 33 * 512, 65 * 512 + 511, 100000]


def in_rows(m):
    """N vertices whose in-rows have the lengths above, three times each, and
    filler rows up to exactly `m` edges (rows in shuffled order)."""
    rng = np.random.default_rng(m)
    lengths = LENGTHS * 3
    left = m - sum(lengths)
    lengths = lengths + [100000] * (left // 100000) + [left % 100000]
    rows = rng.permutation(N)[:len(lengths)].astype(np.uint32)
    starts = rng.integers(0, N, len(lengths))
    src = np.concatenate([(s + np.arange(k)) % N for s, k in zip(starts, lengths)]).astype(np.uint32)
    dst = np.repeat(rows, lengths)
    return bw.HostGraph.from_edges(N, src, dst, dedupe=False, drop_self_loops=False)


@pytest.mark.parametrize("m", [MEGA, 8 * MEGA - 1, 8 * MEGA, 24 * MEGA - 1, 24 * MEGA, 128 * MEGA])
def test_rows_around_the_lengths(ctx, m):
    h = in_rows(m)
    assert h.edge_count == m
    g = bw.DeviceGraph(h)
    its = 3
    want = {"vertex-pull": oracle.PR_DIV, "vertex-pull-nodiv": oracle.PR_NODIV}
    for variant, semantics in want.items():
        ranks, _ = oracle.pagerank(semantics, N, h.rev_vertices, h.rev_edges, its)
        run = bw.pagerank(ctx, g, variant, its)
        assert np.array_equal(run.ranks.cpu().numpy().view(np.uint32), ranks.view(np.uint32)), variant
