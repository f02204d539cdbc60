"""The measured workloads: BFS, PageRank and batched runs as a program that
uses this framework makes them, through the public entry points.

A case is a dict of plain values.  ``task`` says which call is made:

  bfs               one traversal with a fixed variant (bw.bfs)
  bfs-learned       one traversal with the learned per-level switch
  pagerank          a fixed number of iterations of one variant (bw.pagerank)
  pagerank-learned  the same with the learned choice of the variant
  batch-graphs      BFS and PageRank of many small graphs in one launch
  batch-sources     BFS from many sources on one graph in one launch

Graphs are the seeded generators' (R-MAT, Erdos-Renyi, 2-D grid,
Barabasi-Albert), generated on the device; the case's seed is the graph's, and
also picks the root or the sources (a grid has no seed of its own).
"""
import random

import numpy as np
import torch

import belewitte_gb300 as bw
from belewitte_gb300 import batch, learn

INF = 2147483647
DAMPING = float(np.float32(0.85))       # the framework's damping factor is single precision

PULL = ["vertex-pull", "vertex-pull-nodiv", "pull-segmented"]
ATOMIC = ["edge-list", "rev-edge-list", "struct-edge-list", "rev-struct-edge-list", "vertex-push",
          "vertex-push-warp", "vertex-pull-warp", "vertex-pull-warp-nodiv"]
BFS_FAMILIES = ["edge-list", "rev-edge-list", "struct-edge-list", "rev-struct-edge-list", "vertex-push",
                "vertex-pull", "vertex-push-warp", "vertex-pull-warp"]
BFS_SUFFIXES = ["", "-bulk", "-warpreduce", "-blockreduce"]


def listed():
    return [
        # The headline: PageRank in the reference's summation order on a
        # skewed web-like graph, the size the benchmark quotes.
        dict(name="pagerank-rmat22", task="pagerank", graph="rmat", scale=22, edge_factor=16, symmetric=False,
             variant="vertex-pull", iterations=30, loop="host"),
        # PageRank on a graph without skew (no hub helps a cache), the
        # benchmark's second graph, with the iterations in one CUDA graph.
        dict(name="pagerank-er4m", task="pagerank", graph="er", n=4194304, m=67108864, symmetric=False,
             variant="vertex-pull-nodiv", iterations=30, loop="graph"),
        # A small ragged graph: one request of a service that ranks small
        # graphs one at a time, where launches and set-up count.
        dict(name="pagerank-rmat50k", task="pagerank", graph="rmat_n", n=50021, edge_factor=20, symmetric=False,
             variant="vertex-pull", iterations=30, loop="host"),
        # A caller that holds a destination-sorted edge list, mid-sized and
        # ragged: the representation a loader without offsets gives.
        dict(name="pagerank-revel1m", task="pagerank", graph="rmat_n", n=1000003, edge_factor=16, symmetric=False,
             variant="rev-edge-list", iterations=30, loop="host"),
        # The learned choice on a mesh: low, even degrees, ids that follow
        # the geometry.
        dict(name="pagerank-learned-grid", task="pagerank-learned", graph="grid", h=1531, w=2049, symmetric=True,
             iterations=30, loop="graph"),
        # BFS of the largest benchmark graph with the shipped per-level
        # switch and the device-side loop.
        dict(name="bfs-learned-rmat24", task="bfs-learned", graph="rmat", scale=24, edge_factor=16, symmetric=True,
             loop="graph"),
        # High diameter: thousands of levels of a few thousand vertices.
        dict(name="bfs-push-grid2048", task="bfs", graph="grid", h=2048, w=2048, symmetric=True,
             variant="frontier-push", loop="graph"),
        # A fixed reference variant, host-driven, on the preferential
        # attachment graph: every level streams the whole edge list.
        dict(name="bfs-edgelist-ba8m", task="bfs", graph="ba", n=8388608, m=8, symmetric=True,
             variant="edge-list-bulk", loop="host"),
        # The smallest call: a traversal of a graph of a few thousand
        # vertices, all of it latency.
        dict(name="bfs-push-rmat12", task="bfs", graph="rmat", scale=12, edge_factor=16, symmetric=False,
             variant="vertex-push", loop="host"),
        # A fixed bottom-up variant on a mid-sized directed random graph.
        dict(name="bfs-pull-er1m", task="bfs", graph="er", n=1000003, m=16000033, symmetric=False,
             variant="vertex-pull-warpreduce", loop="host"),
        # Many uneven graphs in one launch, each a BFS and 20 PageRank
        # iterations: the batched benchmark's distribution of sizes.
        dict(name="batch-graphs", task="batch-graphs", graphs=512, min_vertices=1000, max_vertices=200000,
             iterations=20),
        # Many sources on one graph (all-pairs style analyses).
        dict(name="batch-sources", task="batch-sources", graph="rmat", scale=20, edge_factor=16, symmetric=True,
             sources=512),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _draw_graph(rng, kinds, max_n, max_m):
    """A graph of one of `kinds` with at most about max_m edges."""
    kind = rng.choice(kinds)
    if kind == "grid":
        h = _log_int(rng, 16, 2048)
        return dict(graph="grid", h=h, w=max(2, min(_log_int(rng, 16, 2048), max_m // (4 * h))), symmetric=True)
    n = _log_int(rng, 1000, max_n)
    ef = rng.randint(4, 32)
    sym = kind in ("ba", "rmat_sym", "er_sym")
    ef = max(2, min(ef, max_m // (n * (2 if sym else 1))))
    if kind == "ba":
        return dict(graph="ba", n=n, m=ef, symmetric=True)
    if kind.startswith("er"):
        return dict(graph="er", n=n, m=n * ef + rng.randint(0, n - 1) // 2, symmetric=sym)
    return dict(graph="rmat_n", n=n, edge_factor=ef, symmetric=sym)


def draw(rng):
    task = rng.choice(["pagerank-pull", "pagerank-pull", "pagerank-atomic", "pagerank-learned", "bfs", "bfs",
                       "bfs-learned", "batch-graphs", "batch-sources"])
    loop = rng.choice(["host", "graph"])
    if task.startswith("pagerank"):
        c = dict(iterations=rng.randint(5, 30), loop=loop)
        c.update(_draw_graph(rng, ["rmat", "rmat", "er", "ba", "grid"], 4194304, 1 << 26))
        if task == "pagerank-learned":
            c["task"] = task
        else:
            c.update(task="pagerank", variant=rng.choice(PULL if task == "pagerank-pull" else ATOMIC))
        return c
    if task == "bfs":
        variant = rng.choice(["frontier-push", "frontier-push", "frontier-pull",
                              rng.choice(BFS_FAMILIES) + rng.choice(BFS_SUFFIXES),
                              rng.choice(BFS_FAMILIES) + rng.choice(BFS_SUFFIXES)])
        # the other variants look at every vertex or edge at every level, so
        # nobody runs them on a mesh of thousands of levels
        kinds = ["rmat", "rmat_sym", "er", "er_sym", "ba"] + (["grid"] if variant == "frontier-push" else [])
        c = dict(task="bfs", variant=variant, loop=loop)
        c.update(_draw_graph(rng, kinds, 8388608, 1 << 27))
        if c["graph"] == "grid" and c["h"] + c["w"] > 512:
            c["loop"] = "graph"         # thousands of levels: the device-side loop
        return c
    if task == "bfs-learned":
        c = dict(task="bfs-learned", loop="graph")
        c.update(_draw_graph(rng, ["rmat_sym", "rmat_sym", "er_sym", "ba", "grid"], 8388608, 1 << 27))
        return c
    if task == "batch-graphs":
        lo = _log_int(rng, 200, 4000)
        return dict(task="batch-graphs", graphs=_log_int(rng, 16, 350), min_vertices=lo,
                    max_vertices=_log_int(rng, 4 * lo, 200000), iterations=rng.randint(5, 20))
    c = dict(task="batch-sources", sources=_log_int(rng, 4, 512))
    c.update(_draw_graph(rng, ["rmat_sym", "rmat", "er_sym", "ba"], 1 << 20, 1 << 25))
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _reps(case):
    """The representations the case's call reads (the CSRs are always there)."""
    csr = bw.REP_FWD_CSR | bw.REP_REV_CSR
    if case["task"].endswith("-learned"):
        return 63
    v = case.get("variant", "")
    if v.startswith("rev-struct"):
        return csr | bw.REP_REV_ST
    if v.startswith("struct"):
        return csr | bw.REP_FWD_ST
    if v.startswith("rev-edge"):
        return csr | bw.REP_REV_EL
    if v.startswith("edge"):
        return csr | bw.REP_FWD_EL
    return csr


def _graph(case, seed):
    k = case["graph"]
    reps = _reps(case)
    if k == "grid":
        return bw.DeviceGraph.generate("grid", h=case["h"], w=case["w"], reps=reps)
    if k == "ba":
        return bw.DeviceGraph.generate("ba", n=case["n"], m=case["m"], seed=seed + 1, reps=reps)
    if k == "er":
        return bw.DeviceGraph.generate("er", n=case["n"], m=case["m"], seed=seed + 1, symmetrise=case["symmetric"],
                                       reps=reps)
    if k == "rmat":
        return bw.DeviceGraph.generate("rmat", scale=case["scale"], edge_factor=case["edge_factor"], seed=seed + 1,
                                       symmetrise=case["symmetric"], reps=reps)
    return bw.DeviceGraph.generate("rmat_n", n=case["n"], edge_factor=case["edge_factor"], seed=seed + 1,
                                   symmetrise=case["symmetric"], reps=reps)


def _pick(g, seed, count):
    """`count` seeded vertices of at least the mean out-degree."""
    n = g.vertex_count
    deg = g.fwd_vertices[1:n + 1] - g.fwd_vertices[:n]
    mean = max(1, -(-g.edge_count // n) if n else 1)
    some = torch.nonzero(deg >= min(mean, int(deg.max().item()))).flatten()
    rng = random.Random(seed * 7919 + 13)
    where = torch.tensor([rng.randrange(some.numel()) for _ in range(count)], device=some.device)
    return [int(v) for v in some[where].cpu()]


def _packed(case, seed):
    # the sizes are the case's, the edges the seed's
    sizes = random.Random(case["graphs"] * 104729 + case["min_vertices"])
    seeds = random.Random(seed)
    gs = []
    for _ in range(case["graphs"]):
        n = _log_int(sizes, case["min_vertices"], case["max_vertices"])
        gs.append(bw.DeviceGraph.generate("rmat_n", n=n, edge_factor=sizes.randint(8, 32),
                                          seed=seeds.randrange(1, 2 ** 31)))
    return batch.pack(gs)


def prepare(case, seed):
    """The graph on the device, the context, and what else the program keeps."""
    state = dict(case=case, ctx=bw.Context(0))
    task = case["task"]
    if task == "batch-graphs":
        state["packed"] = _packed(case, seed)
        return state
    state["g"] = g = _graph(case, seed)
    if task == "batch-sources":
        state["sources"] = _pick(g, seed, case["sources"])
    elif task in ("bfs", "bfs-learned"):
        state["root"] = _pick(g, seed, 1)[0]
    if task == "bfs-learned":
        state["predictor"] = learn.load_predictor()
    elif task == "pagerank-learned":
        state["predictor"] = learn.load_pagerank_predictor()
    return state


def run(state):
    case, ctx = state["case"], state["ctx"]
    task = case["task"]
    if task == "batch-graphs":
        levels, ranks, res = batch.run_graphs(ctx, state["packed"], pr_iterations=case["iterations"])
        return dict(levels=levels, ranks=ranks, traversed_edges=res.traversed_edges)
    g = state["g"]
    if task == "batch-sources":
        levels, res = batch.run_sources(ctx, g, state["sources"])
        return dict(levels=levels, traversed_edges=res.traversed_edges)
    if task in ("bfs", "bfs-learned"):
        if task == "bfs":
            r = bw.bfs(ctx, g, case["variant"], state["root"], loop=case["loop"])
        else:
            r = learn.run_learned(ctx, g, state["predictor"], state["root"], loop=case["loop"], stats=False)
        return dict(levels=r.levels, level_count=r.level_count, visited=r.visited,
                    traversed_edges=r.traversed_edges)
    if task == "pagerank":
        r = bw.pagerank(ctx, g, case["variant"], case["iterations"], loop=case["loop"])
    else:
        r, _ = learn.run_pagerank_learned(ctx, g, state["predictor"], case["iterations"], loop=case["loop"])
    return dict(ranks=r.ranks, diffs=np.asarray(r.diffs, np.float32))


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _size(case):
    """(vertices, edges): the generators' sample counts, before duplicates
    are dropped (2-3% of R-MAT's)."""
    k = case["graph"]
    if k == "grid":
        return case["h"] * case["w"], 4 * case["h"] * case["w"]
    if k == "rmat":
        n = 1 << case["scale"]
        m = n * case["edge_factor"]
    elif k == "rmat_n":
        n, m = case["n"], case["n"] * case["edge_factor"]
    elif k == "er":
        n, m = case["n"], case["m"]
    else:
        n, m = case["n"], case["n"] * case["m"]
    return n, m * (2 if case["symmetric"] else 1)


def _pagerank_work(n, m, iterations):
    # Every iteration depends on the one before it: it reads a source id per
    # edge, the offsets, and each rank once, and writes each rank once.
    return iterations * (4 * m + 4 * (n + 1) + 8 * n), iterations * (m + 4 * n)


def _bfs_work(n, m):
    # The adjacency and the offsets read once, a depth written per vertex.
    return 4 * (n + 1) + 4 * m + 4 * n, 0


def work(case):
    task = case["task"]
    if task == "batch-graphs":
        # the mean of the log-uniform sizes, 20 edges per vertex
        lo, hi = case["min_vertices"], case["max_vertices"]
        n = int(case["graphs"] * (hi - lo) / np.log(hi / lo))
        b, f = _pagerank_work(n, 20 * n, case["iterations"])
        return {"bytes": b + _bfs_work(n, 20 * n)[0], "flops": f}
    n, m = _size(case)
    if task == "batch-sources":
        # the graph read once, a depth written per vertex and source
        return {"bytes": 4 * (n + 1) + 4 * m + 4 * n * case["sources"], "flops": 0}
    b, f = _bfs_work(n, m) if task.startswith("bfs") else _pagerank_work(n, m, case["iterations"])
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# the same in 64 bits, plain torch
# ---------------------------------------------------------------------------
def _csr(vertices, edges, n, m):
    return vertices[:n + 1].long(), edges[:m].long()


def _exact_bfs(off, edges, roots, n):
    levels = torch.full((n,), INF, dtype=torch.int32, device=off.device)
    frontier = torch.as_tensor(roots, dtype=torch.long, device=off.device)
    levels[frontier] = 0
    depth = 0
    while frontier.numel():
        deg = off[frontier + 1] - off[frontier]
        ends = torch.cumsum(deg, 0)
        total = int(ends[-1].item())
        at = torch.repeat_interleave(off[frontier] - (ends - deg), deg, output_size=total)
        at += torch.arange(total, device=off.device)
        v = edges[at]
        v = v[levels[v] == INF]
        depth += 1
        levels[v] = depth
        frontier = torch.unique(v)
    return levels, depth


def _exact_pagerank(fwd_off, rev_off, rev_edges, n, init, base, iterations, nodiv):
    """Ranks and per-iteration differences.  `init` and `base` are per vertex
    (1/N and (1 - d)/N of the vertex's graph)."""
    deg = (fwd_off[1:] - fwd_off[:-1]).double()
    rows = torch.repeat_interleave(torch.arange(n, device=rev_off.device), rev_off[1:] - rev_off[:-1])
    rank = init.clone()
    diffs = []
    for it in range(iterations):
        if nodiv:
            # ranks are kept divided by the out-degree, the initial ones not
            src = rank
        else:
            src = torch.where(deg > 0, rank / deg, torch.zeros_like(rank))
        acc = torch.zeros_like(rank)
        acc.index_add_(0, rows, src[rev_edges])
        new = base + DAMPING * acc
        diffs.append(float((new - rank).abs().sum().item()))
        if nodiv and it + 1 < iterations:
            new = torch.where(deg > 0, new / deg, new)
        rank = new
    return rank, np.asarray(diffs)


def exact(case, seed):
    task = case["task"]
    if task == "batch-graphs":
        p = _packed(case, seed)
        fwd_v, fwd_e, rev_v, rev_e = p.tensors
        n, m = p.vertex_count, p.edge_count
        fo, fe = _csr(fwd_v, fwd_e, n, m)
        levels, _ = _exact_bfs(fo, fe, p.roots.long(), n)
        trav = int((fo[1:] - fo[:-1])[levels != INF].sum().item())
        del fe
        ro, re = _csr(rev_v, rev_e, n, m)
        offs = p.offsets.long()
        size = torch.repeat_interleave(offs[1:] - offs[:-1], offs[1:] - offs[:-1]).double()
        ranks, _ = _exact_pagerank(fo, ro, re, n, 1.0 / size, (1.0 - DAMPING) / size, case["iterations"], False)
        return dict(levels=levels, ranks=ranks, traversed_edges=trav)
    g = _graph(case, seed)
    n, m = g.vertex_count, g.edge_count
    fo = g.fwd_vertices[:n + 1].long()
    deg = fo[1:] - fo[:-1]
    if task == "batch-sources":
        fe = g.fwd_edges[:m].long()
        levels = torch.empty((case["sources"], n), dtype=torch.int32, device=fo.device)
        trav = 0
        for i, s in enumerate(_pick(g, seed, case["sources"])):
            levels[i], _ = _exact_bfs(fo, fe, [s], n)
            trav += int(deg[levels[i] != INF].sum().item())
        return dict(levels=levels, traversed_edges=trav)
    if task in ("bfs", "bfs-learned"):
        levels, depth = _exact_bfs(fo, g.fwd_edges[:m].long(), _pick(g, seed, 1), n)
        seen = levels != INF
        return dict(levels=levels, level_count=depth, visited=int(seen.sum().item()),
                    traversed_edges=int(deg[seen].sum().item()))
    ro, re = _csr(g.rev_vertices, g.rev_edges, n, m)
    one = torch.ones(n, dtype=torch.float64, device=fo.device)
    nodiv = case.get("variant", "").endswith("-nodiv")
    ranks, diffs = _exact_pagerank(fo, ro, re, n, one / n, one * ((1.0 - DAMPING) / n), case["iterations"], nodiv)
    return dict(ranks=ranks, diffs=diffs)
