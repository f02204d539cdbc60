// BFS half of the C ABI: variant registry, level launch, host-loop and
// CUDA-graph (device-side conditional loop) traversals.
//
// Reference: BFS::runImplementation (bfs/bfs.cpp:51-118) and the variant
// registration of bfs/bfs.cpp:121-224.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <string>

#include "bw_internal.cuh"

namespace bw {
namespace {

constexpr int FAMILIES = 8;
constexpr int V_FRONTIER_PUSH = 32;
constexpr int V_FRONTIER_PULL = 33;
constexpr int VARIANT_COUNT = 34;

const char *const kFamily[FAMILIES] = {
    "edge-list", "rev-edge-list", "struct-edge-list", "rev-struct-edge-list",
    "vertex-push", "vertex-pull", "vertex-push-warp", "vertex-pull-warp"};
const char *const kSuffix[4] = {"", "-bulk", "-warpreduce", "-blockreduce"};

constexpr int REP_FWD_CSR = 1, REP_REV_CSR = 2, REP_FWD_EL = 4, REP_REV_EL = 8,
              REP_FWD_ST = 16, REP_REV_ST = 32;
const int kFamilyReps[FAMILIES] = {REP_FWD_EL, REP_REV_EL, REP_FWD_ST, REP_REV_ST,
                                   REP_FWD_CSR, REP_REV_CSR, REP_FWD_CSR, REP_REV_CSR};

struct NameTable {
    std::string names[VARIANT_COUNT];
    NameTable()
    {
        for (int f = 0; f < FAMILIES; f++)
            for (int r = 0; r < 4; r++) names[f * 4 + r] = std::string(kFamily[f]) + kSuffix[r];
        names[V_FRONTIER_PUSH] = "frontier-push";
        names[V_FRONTIER_PULL] = "frontier-pull";
    }
};
const NameTable &names()
{
    static NameTable t;
    return t;
}

int variant_reps(int v)
{
    if (v >= 0 && v < 32) return kFamilyReps[v / 4];
    if (v == V_FRONTIER_PUSH) return REP_FWD_CSR;
    if (v == V_FRONTIER_PULL) return REP_REV_CSR;
    return 0;
}

int check_reps(const bw_graph_view *g, int reps)
{
    if ((reps & REP_FWD_CSR) && (!g->fwd_vertices || !g->fwd_edges)) return BW_ERR_MISSING_REPRESENTATION;
    if ((reps & REP_REV_CSR) && (!g->rev_vertices || !g->rev_edges)) return BW_ERR_MISSING_REPRESENTATION;
    if ((reps & REP_FWD_EL) && (!g->fwd_in_edges || !g->fwd_edges)) return BW_ERR_MISSING_REPRESENTATION;
    if ((reps & REP_REV_EL) && (!g->rev_in_edges || !g->rev_edges)) return BW_ERR_MISSING_REPRESENTATION;
    if ((reps & REP_FWD_ST) && !g->fwd_struct_edges) return BW_ERR_MISSING_REPRESENTATION;
    if ((reps & REP_REV_ST) && !g->rev_struct_edges) return BW_ERR_MISSING_REPRESENTATION;
    return BW_OK;
}

}  // namespace

// Depth initialisation (bfs/bfs.cpp:69-76) plus the control block; with
// `outdeg` the root's degree statistics seed the frontier features.
__global__ void k_bfs_init_side(int32_t *levels, uint64_t n, uint32_t root, uint32_t *q0, BfsCtl *ctl,
                                uint32_t max_levels, const uint32_t *outdeg)
{
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t v = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; v < n; v += stride)
        levels[v] = v == root ? 0 : INF;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        q0[0] = root;
        for (int i = 0; i < 3; i++) ctl->slot[i] = LevelSlot{};
        ctl->slot[2].frontier = 1;
        ctl->slot[2].qlen = 1;     // input queue of level 0 = {root}
        ctl->depth = 0;
        ctl->levels_done = 0;
        ctl->variant = 0;
        ctl->status = 0;
        ctl->visited = 1;
        ctl->traversed = 0;
        ctl->max_levels = max_levels;
        ctl->skip = 0;
        ctl->edges = 0;
        if (outdeg) {
            const uint32_t d = outdeg[root];
            const float l = __log2f(1.0f + static_cast<float>(d));
            ctl->slot[2].fedges = d;
            ctl->slot[2].lsum = lsum_fx(l);
            ctl->slot[2].lsq = lsq_fx(l);
            ctl->slot[2].lmax_bits = __float_as_uint(l);
            ctl->traversed = d;
        }
    }
}

namespace {

// The host loop's read of a level's counts (getFrontier(), bfs/bfs.cu:13-18),
// and of the totals: written to the host, then the number it waits for.
__global__ void k_bfs_post(const BfsCtl *ctl, int slot, BfsMail *mail, uint32_t seq)
{
    chain_wait();
    mail->slot = ctl->slot[slot];
    mail->edges = ctl->edges;
    __threadfence_system();
    *reinterpret_cast<volatile uint32_t *>(&mail->seq) = seq;
}

// Device-loop step, after every level: logs the level, advances the depth;
// true when the level visited nothing or the level cap is reached (status =
// LEVEL_LIMIT).
__device__ __forceinline__ bool step_level(BfsCtl *ctl, LevelSlot *log, uint32_t log_cap)
{
    const int32_t L = ctl->depth;
    const LevelSlot s = ctl->slot[L % 3];
    if (log && static_cast<uint32_t>(L) < log_cap) log[L] = s;
    ctl->visited += s.frontier;
    ctl->traversed += s.fedges;
    ctl->levels_done = static_cast<uint32_t>(L) + 1;
    ctl->depth = L + 1;
    ctl->skip = 0;
    bool stop = s.frontier == 0;
    if (!stop && ctl->levels_done >= ctl->max_levels) {
        ctl->status = BW_ERR_LEVEL_LIMIT;
        stop = true;
    }
    return stop;
}

// In the graph's conditional body: ends the loop.
__global__ void k_bfs_step(BfsCtl *ctl, LevelSlot *log, uint32_t log_cap,
                           cudaGraphConditionalHandle loop)
{
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    if (step_level(ctl, log, log_cap)) cudaGraphSetConditional(loop, 0);
}

// Launched by the host, which waits for it.
__global__ void k_bfs_step_post(BfsCtl *ctl, LevelSlot *log, uint32_t log_cap, BfsMail *mail, uint32_t seq)
{
    chain_wait();
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    mail->stop = step_level(ctl, log, log_cap) ? 1u : 0u;
    mail->status = ctl->status;
    mail->levels_done = ctl->levels_done;
    mail->visited = ctl->visited;
    mail->slot = ctl->slot[(ctl->depth + 2) % 3];     // the next level's input
    __threadfence_system();
    *reinterpret_cast<volatile uint32_t *>(&mail->seq) = seq;
}

// Sum of out-degrees of reached vertices (TEPS numerator).  Four vertices a
// thread and load where the arrays allow it, two loads of each in flight; one
// atomic per block.  16.7M vertices on GB300: 100 us with one at a time, 26
// so.
__global__ void __launch_bounds__(256) k_traversed(const int32_t *levels, const uint32_t *off, uint64_t n,
                                                   unsigned long long *out)
{
    chain_wait();
    __shared__ unsigned long long part[8];
    const uint64_t tid = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x, stride = uint64_t(gridDim.x) * blockDim.x;
    const bool wide = ((reinterpret_cast<uintptr_t>(levels) | reinterpret_cast<uintptr_t>(off)) & 15) == 0;
    const uint64_t quads = wide ? n / 4 : 0;
    unsigned long long acc = 0;
#pragma unroll 2
    for (uint64_t q = tid; q < quads; q += stride) {
        const int4 d = reinterpret_cast<const int4 *>(levels)[q];
        const uint4 o = reinterpret_cast<const uint4 *>(off)[q];
        const uint32_t e = off[4 * q + 4];
        acc += d.x != INF ? o.y - o.x : 0u;
        acc += d.y != INF ? o.z - o.y : 0u;
        acc += d.z != INF ? o.w - o.z : 0u;
        acc += d.w != INF ? e - o.w : 0u;
    }
    for (uint64_t v = 4 * quads + tid; v < n; v += stride)
        if (levels[v] != INF) acc += off[v + 1] - off[v];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(FULL_MASK, acc, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (unsigned w = 1; w < blockDim.x / 32; w++) acc += part[w];
        if (acc) atomicAdd(out, acc);
    }
}

struct Launch {
    BfsKernelFn k;
    BfsKernelFn k2;    // the level's second kernel: hub chunks, or edge-list's edges
    unsigned block, grid;
    size_t smem;
    unsigned grid2;    // of k2
    // k2 may start while k ends: not the edges' kernel, one resident wave whose
    // blocks would gather on the SMs that are free first (BA(8.4M, 8) 1000 ->
    // 1050 us a traversal)
    bool k2_early = true;
};

// Blocks of the hub-chunk kernel per SM, the resident ones: most levels have no
// chunk, and starting and retiring blocks is all that it then does.  Eight (a
// wave that waits for the first) on GB300: frontier-push on R-MAT-20
// symmetrised 338 us a traversal, 320 so; vertex-push-warp on BA(4.2M, 12)
// 1471 and 1404.
constexpr unsigned HUB_BLOCKS = 4;

int plan_launch(const bw_context *ctx, const bw_graph_view *g, int variant, bool side, const bw_launch_config *cfg,
                Launch *out)
{
    Launch l{nullptr, nullptr, 256, static_cast<unsigned>(ctx->sm_count) * 8, 0, 0};
    const uint32_t W = (cfg && cfg->warp_size) ? cfg->warp_size : 32;
    const uint32_t C = (cfg && cfg->chunk_size) ? cfg->chunk_size : 32;
    if (variant >= 0 && variant < 16) {
        // edge-list families (0..3 rev/struct via variant / 4)
        const int fam = variant / 4;
        const int layout = fam == 0 ? 0 : fam == 1 ? 1 : fam == 2 ? 2 : 3;
        l.k = bfs_edge_kernel(layout, variant % 4, side);
        l.block = 512;
        l.grid = static_cast<unsigned>(ctx->sm_count) * 4;
    } else if (variant >= 16 && variant < 32) {
        l.k = bfs_vertex_kernel(variant / 4, variant % 4, side);
        const int fam = variant / 4;
        if (fam == 4 || fam == 6) l.k2 = bfs_hub_kernel(side);   // vertex-push(-warp): hub rows in chunks
        if (fam == 6 || fam == 7) {
            // ImplementationTemplate.hpp:463-471: power-of-two W <= 32, C % W == 0
            if (W == 0 || W > 32 || (W & (W - 1)) || C == 0 || C % W) return BW_ERR_INVALID_ARGUMENT;
        }
    } else if (variant == V_FRONTIER_PUSH) {
        l.k = bfs_frontier_push_kernel(side);
        l.k2 = bfs_hub_kernel(side);
    } else if (variant == V_FRONTIER_PULL) {
        l.k = bfs_frontier_pull_kernel(side);
    } else {
        return BW_ERR_UNKNOWN_VARIANT;
    }
    if (cfg && cfg->block_size) {
        if (cfg->block_size % 32 || cfg->block_size > 1024) return BW_ERR_INVALID_ARGUMENT;
        if ((variant == V_FRONTIER_PUSH || variant == V_FRONTIER_PULL) && cfg->block_size != 256)
            return BW_ERR_INVALID_ARGUMENT;
        if (cfg->block_size > 512) return BW_ERR_INVALID_ARGUMENT;   // __launch_bounds__(512)
        l.block = cfg->block_size;
    }
    if (cfg && cfg->grid_size) l.grid = cfg->grid_size;
    if (variant >= 24 && variant < 32) {
        if (l.block % W) return BW_ERR_INVALID_ARGUMENT;
        l.smem = (l.block / W) * (C * 4 + (C + 1) * 4);
        if (l.smem > ctx->max_smem_per_block) return BW_ERR_INVALID_ARGUMENT;
    }
    // A graph smaller than the grid gets the blocks that have work: starting
    // and retiring 1216 idle blocks is most of a small level.
    l.grid2 = hub_grid(l.grid, l.block);
    const uint64_t n = g->vertex_count, m = g->edge_count;
    auto blocks = [](uint64_t items, uint64_t per_block) { return std::max<uint64_t>(1, (items + per_block - 1) / per_block); };
    uint64_t need;
    if (variant < 16) need = blocks(m, 4 * uint64_t(l.block));                        // 4 edges a thread
    else if (variant < 20) need = blocks(n, 4 * uint64_t(l.block));                   // vertex-push: 4 depths a thread
    else if (variant >= 24 && variant < 32) need = blocks(n, uint64_t(C) * (l.block / W));
    else if (variant == V_FRONTIER_PUSH) need = blocks(n, 32);                        // 8 warps of 4 rows
    else need = blocks(n, l.block);
    l.grid = static_cast<unsigned>(std::min<uint64_t>(l.grid, need));
    // at most this many hub chunks in a level (ensure_bfs_scratch), one per warp
    l.grid2 = static_cast<unsigned>(std::min<uint64_t>(std::min(l.grid2, HUB_BLOCKS * static_cast<unsigned>(ctx->sm_count)),
                                                       blocks(2 * m / 256 + n / 256, 8)));
    *out = l;
    return BW_OK;
}

BfsArgs make_args(bw_context *ctx, const bw_graph_view *g, int32_t *levels, int32_t depth,
                  const bw_launch_config *cfg)
{
    BfsArgs a{};
    a.fwd_v = g->fwd_vertices; a.fwd_e = g->fwd_edges;
    a.rev_v = g->rev_vertices; a.rev_e = g->rev_edges;
    a.fwd_in = g->fwd_in_edges; a.rev_in = g->rev_in_edges;
    a.fwd_s = reinterpret_cast<const uint2 *>(g->fwd_struct_edges);
    a.rev_s = reinterpret_cast<const uint2 *>(g->rev_struct_edges);
    a.outdeg = ctx->outdeg;
    a.n = g->vertex_count; a.m = g->edge_count;
    a.levels = levels;
    a.ctl = ctx->bfs_ctl;
    a.q0 = ctx->queue[0]; a.q1 = ctx->queue[1];
    a.heavy = ctx->heavy;
    a.depth = depth;
    a.warp_size = (cfg && cfg->warp_size) ? cfg->warp_size : 32;
    a.chunk_size = (cfg && cfg->chunk_size) ? cfg->chunk_size : 32;
    return a;
}

// early: as a chain (chain_wait), when the host waits for nothing in between
int launch(const Launch &l, const BfsArgs &a, cudaStream_t s, bool early = false)
{
    BW_CUDA(launch_chained(l.k, l.grid, l.block, l.smem, s, early, a));
    // the hub-chunk kernel is built for 256-thread blocks
    if (l.k2) BW_CUDA(launch_chained(l.k2, l.grid2, 256, 0, s, early && l.k2_early, a));
    return BW_OK;
}

int validate_graph(const bw_graph_view *g)
{
    if (!g) return BW_ERR_INVALID_ARGUMENT;
    if (g->vertex_count == 0 || g->vertex_count >= 0x7fffffffULL || g->edge_count > 0xffffffffULL)
        return BW_ERR_INVALID_ARGUMENT;
    return BW_OK;
}

void fill_stats(const LevelSlot &s, int variant, bw_bfs_level_stats *out)
{
    out->frontier_vertices = s.frontier;
    out->variant = static_cast<uint32_t>(variant);
    out->frontier_edges = s.fedges;
    out->log_degree_sum = static_cast<float>(lsum_value(s.lsum));
    out->log_degree_sq_sum = static_cast<float>(lsq_value(s.lsq));
    uint32_t bits = s.lmax_bits;
    float f;
    std::memcpy(&f, &bits, sizeof f);
    out->log_degree_max = f;
    out->device_ms = 0.0f;
}

// Posts level slot `slot` (and the edge total) and waits for it.
int post_and_wait(bw_context *ctx, int slot, cudaStream_t s)
{
    const uint32_t seq = ++ctx->mail_seq;
    BW_CUDA(launch_chained(k_bfs_post, 1, 1, 0, s, true, static_cast<const BfsCtl *>(ctx->bfs_ctl), slot, ctx->mail, seq));
    return bfs_wait(ctx, seq, s);
}

// ctl->edges is zero since the run's initialisation.
int traversed_edges(bw_context *ctx, const bw_graph_view *g, int32_t *levels, cudaStream_t s,
                    uint64_t *out)
{
    *out = 0;
    if (!g->fwd_vertices) return BW_OK;
    const uint64_t n = g->vertex_count;
    const unsigned grid = static_cast<unsigned>(std::min<uint64_t>((n + 255) / 256, uint64_t(ctx->sm_count) * 8));
    BW_CUDA(launch_chained(k_traversed, grid, 256, 0, s, true, static_cast<const int32_t *>(levels), g->fwd_vertices, n,
                           &ctx->bfs_ctl->edges));
    BW_TRY(post_and_wait(ctx, 0, s));
    *out = ctx->mail->edges;
    return BW_OK;
}

// edge-list levels by chunk (k_bfs_edge_chunks), where a level would stream
// the list from HBM and no launch shape is asked for (bfs() fills one in on
// graphs near a class that the autotuner's cache holds, whose levels then run
// whole: R-MAT-22 edge-list-bulk 765 us so, 552 by chunk).
constexpr uint64_t CHUNKED_EDGES = uint64_t(16) << 20;
bool chunked(const bw_graph_view *g, int variant, const bw_launch_config *cfg)
{
    return variant >= 0 && variant < 4 && g->edge_count >= CHUNKED_EDGES && !(cfg && (cfg->block_size || cfg->grid_size)) &&
           ((reinterpret_cast<uintptr_t>(g->fwd_in_edges) | reinterpret_cast<uintptr_t>(g->fwd_edges)) & 15) == 0;
}
void plan_chunks(const bw_context *ctx, int variant, bool side, Launch *l)
{
    l->k = bfs_edge_active_kernel();
    l->block = 256;
    l->k2 = bfs_edge_chunk_kernel(variant, side);
    l->k2_early = false;
    l->grid = static_cast<unsigned>(ctx->sm_count) * 8;
    l->grid2 = static_cast<unsigned>(ctx->sm_count) * (side ? 4 : 5);      // one resident wave
}
void chunk_args(bw_context *ctx, BfsArgs *a)
{
    a->ranges = ctx->heavy;
    a->active = reinterpret_cast<uint32_t *>(ctx->heavy + (a->m + EDGE_CHUNK - 1) / EDGE_CHUNK);
}

// vertex-pull levels with the frontier's filter (k_bfs_pull_filter): `frontier`
// vertices of this level, `visited` so far.  A level of ER(1M, 8M) takes 25 to
// 29 us with it and 44 to 47 without while the frontier is under a 256th of the
// vertices; at a 70th 42 and 53, from a 25th on the hits cost more than the
// filter saves.  Once half the vertices are visited the plain kernel has few
// rows left.  Whole traversals on GB300, every level plain and with the filter:
// ER(1M, 16M) 524 -> 373 us, ER(4M, 67M) 1607 -> 960, ER(8M, 32M) 1871 -> 1593;
// from the hub R-MAT-20 symmetrised 379 -> 230, R-MAT-22 1302 -> 505 and
// BA(4.2M, 12) 1385 -> 549, from other roots (a thread per hub row then scans
// all of it) 9.0 ms -> 0.32, 16.3 -> 0.68 and 8.5 -> 0.81.  No launch shape may
// be asked for: bfs() fills one in on graphs near a class that the autotuner's
// cache holds, whose levels then run plain.
constexpr uint64_t FILTERED_EDGES = uint64_t(4) << 20;
constexpr uint64_t FILTERED_SHARE = 256;
// In the hub-chunk queue: the filter, then the heavy windows' pieces (a window
// of more than FILTER_PIECE edges has at most twice edges / FILTER_PIECE).
constexpr uint64_t FILTER_WORDS2 = FILTER_BITS / 64;
bool filtered(const bw_context *ctx, const bw_graph_view *g, int variant, const bw_launch_config *cfg, uint64_t frontier,
              uint64_t visited)
{
    return variant >= 20 && variant < 24 && g->edge_count >= FILTERED_EDGES && !(cfg && (cfg->block_size || cfg->grid_size)) &&
           frontier * FILTERED_SHARE <= g->vertex_count && 2 * visited <= g->vertex_count &&
           ctx->heavy_cap >= FILTER_WORDS2 + 2 * (g->edge_count / FILTER_PIECE);
}
int launch_filtered(bw_context *ctx, int variant, bool side, BfsArgs a, cudaStream_t s, bool early)
{
    uint32_t bits = 4096;
    while (bits < a.n && bits < FILTER_BITS) bits *= 2;
    a.filter = reinterpret_cast<uint32_t *>(ctx->heavy);
    a.filter_mask = bits - 1;
    a.pieces = ctx->heavy + FILTER_WORDS2;
    const BfsKernelFn k = bfs_pull_filter_kernel(variant % 4, side);
    const unsigned sms = static_cast<unsigned>(ctx->sm_count);
    BW_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(FILTER_BITS / 8)));
    BW_CUDA(launch_chained(bfs_filter_kernel(), std::min(sms * 8, bits / 32 / 8), 256, 0, s, early, a));
    BW_CUDA(launch_chained(k, sms, 1024, bits / 8, s, early, a));
    return BW_OK;
}

// Host-loop traversal with a per-level variant schedule.
int run_host(bw_context *ctx, const bw_graph_view *g, const int32_t *schedule, uint32_t sched_len,
             uint32_t root, int32_t *levels, const bw_launch_config *cfg, uint32_t max_levels,
             int time_levels, bool side, bw_bfs_result *result, bw_bfs_level_stats *stats,
             uint32_t stats_cap, cudaStream_t s)
{
    const uint64_t n = g->vertex_count;
    if (max_levels == 0) max_levels = static_cast<uint32_t>(std::min<uint64_t>(n + 1, 0xffffffffULL));
    Launch plans[VARIANT_COUNT];
    bool planned[VARIANT_COUNT] = {};
    for (uint32_t i = 0; i < sched_len; i++) {
        const int v = schedule[i];
        if (v < 0 || v >= VARIANT_COUNT) return BW_ERR_UNKNOWN_VARIANT;
        if (!planned[v]) {
            BW_TRY(plan_launch(ctx, g, v, side, cfg, &plans[v]));
            if (chunked(g, v, cfg)) plan_chunks(ctx, v, side, &plans[v]);
            planned[v] = true;
        }
    }
    if (time_levels) BW_TRY(ensure_level_events(ctx, 2));
    k_bfs_init_side<<<ctx->sm_count * 4, 256, 0, s>>>(levels, n, root, ctx->queue[0], ctx->bfs_ctl, max_levels,
                                                     side ? ctx->outdeg : nullptr);
    BW_CUDA(cudaGetLastError());
    BW_CUDA(cudaEventRecord(ctx->ev_start, s));
    float total_ms = 0.0f;
    uint32_t level = 0;
    uint64_t visited = 1;
    int status = BW_OK;
    bool ranges = false;                    // in ctx->heavy, until a push level's hub chunks overwrite them
    for (;;) {
        if (level >= max_levels) { status = BW_ERR_LEVEL_LIMIT; break; }
        const int v = schedule[std::min(level, sched_len - 1)];
        BfsArgs a = make_args(ctx, g, levels, static_cast<int32_t>(level), cfg);
        const bool chunks = chunked(g, v, cfg), build = chunks && !ranges;
        if (chunks) chunk_args(ctx, &a);
        else if (plans[v].k2) ranges = false;
        if (time_levels) BW_CUDA(cudaEventRecord(ctx->level_events[0], s));
        if (build) {
            BW_TRY(bfs_edge_ranges(ctx, g, ctx->heavy, s));
            ranges = true;
        }
        if (filtered(ctx, g, v, cfg, level ? ctx->mail->slot.frontier : 1, visited)) {
            BW_TRY(launch_filtered(ctx, v, side, a, s, !time_levels));
            ranges = false;                 // the filter lies where they did
        } else {
            BW_TRY(launch(plans[v], a, s, !time_levels));
        }
        if (time_levels) BW_CUDA(cudaEventRecord(ctx->level_events[1], s));
        BW_TRY(post_and_wait(ctx, static_cast<int>(level % 3), s));
        const LevelSlot sl = ctx->mail->slot;
        if (stats && level < stats_cap) {
            fill_stats(sl, v, &stats[level]);
            if (time_levels) BW_CUDA(cudaEventSynchronize(ctx->level_events[1]));
            if (time_levels)
                BW_CUDA(cudaEventElapsedTime(&stats[level].device_ms, ctx->level_events[0], ctx->level_events[1]));
        }
        visited += sl.frontier;
        level++;
        if (sl.frontier == 0) break;
    }
    BW_CUDA(cudaEventRecord(ctx->ev_stop, s));
    if (result) {
        BW_TRY(traversed_edges(ctx, g, levels, s, &result->traversed_edges));
        BW_CUDA(cudaEventSynchronize(ctx->ev_stop));
        BW_CUDA(cudaEventElapsedTime(&total_ms, ctx->ev_start, ctx->ev_stop));
        result->level_count = level;
        result->visited = visited;
        result->device_ms = total_ms;
    }
    return status;
}

// Device-loop traversal.  The level's kernels read the depth and their queue's
// length on the device, and a step kernel keeps the totals.  The first
// DEVICE_LOOP_LAUNCHED rounds are launched by the host, which only waits for
// the step's verdict: most traversals end there, and building a CUDA graph
// (0.25 ms) would cost them more than all their launches.  A traversal that
// goes on continues in a graph whose conditional WHILE node runs the same
// kernels until the step kernel clears the loop condition, with no host round
// trip per level.
constexpr uint32_t DEVICE_LOOP_LAUNCHED = 48;

int run_graph(bw_context *ctx, const bw_graph_view *g, int variant, uint32_t root,
              int32_t *levels, const bw_launch_config *cfg, uint32_t max_levels, bool side,
              bw_bfs_result *result, bw_bfs_level_stats *stats, uint32_t stats_cap,
              cudaStream_t s)
{
    const uint64_t n = g->vertex_count;
    if (max_levels == 0) max_levels = static_cast<uint32_t>(std::min<uint64_t>(n + 1, 0xffffffffULL));
    Launch plan;
    BW_TRY(plan_launch(ctx, g, variant, side, cfg, &plan));
    const bool chunks = chunked(g, variant, cfg);
    if (chunks) plan_chunks(ctx, variant, side, &plan);
    const bool cluster_path = variant == V_FRONTIER_PUSH;
    if (cluster_path) {
        BW_TRY(ensure_outdeg(ctx, g, s));   // frontier edge volumes gate the cluster path
        BW_TRY(bfs_cluster_prepare());
    }
    LevelSlot *log = nullptr;
    const uint32_t log_cap = stats ? std::min(stats_cap, max_levels) : 0;
    if (log_cap) BW_CUDA(ctx_malloc_async(ctx, reinterpret_cast<void **>(&log), log_cap * sizeof(LevelSlot), s));
    BfsArgs a = make_args(ctx, g, levels, -1, cfg);
    if (chunks) chunk_args(ctx, &a);
    if (cluster_path) {
        // small frontiers: the cluster kernel runs many levels per launch
        a.skip_check = 1;
        a.log = log;
        a.log_cap = log_cap;
    }
    auto level_kernels = [&](cudaStream_t to, bool small, bool early) -> int {
        if (cluster_path && small)
            BW_CUDA(launch_chained(bfs_cluster_kernel(side ? 1 : 0), CLUSTER_CTAS, CLUSTER_THREADS, bfs_cluster_smem(), to, early, a));
        return launch(plan, a, to, early);
    };
    BfsMail end{};                          // the last round's
    auto traverse = [&]() -> int {
        k_bfs_init_side<<<ctx->sm_count * 4, 256, 0, s>>>(levels, n, root, ctx->queue[0], ctx->bfs_ctl, max_levels,
                                                         (side || cluster_path) ? ctx->outdeg : nullptr);
        BW_CUDA(cudaGetLastError());
        BW_CUDA(cudaEventRecord(ctx->ev_start, s));
        if (chunks) BW_TRY(bfs_edge_ranges(ctx, g, ctx->heavy, s));
        for (uint32_t i = 0; i < DEVICE_LOOP_LAUNCHED && !end.stop; i++) {
            if (filtered(ctx, g, variant, cfg, i ? end.slot.frontier : 1, i ? end.visited : 1))
                BW_TRY(launch_filtered(ctx, variant, side, a, s, true));
            else
                BW_TRY(level_kernels(s, i == 0 || cluster_frontier(end.slot), true));
            const uint32_t seq = ++ctx->mail_seq;
            BW_CUDA(launch_chained(k_bfs_step_post, 1, 32, 0, s, true, ctx->bfs_ctl, log, log_cap, ctx->mail, seq));
            BW_TRY(bfs_wait(ctx, seq, s));
            end = *ctx->mail;
        }
        if (end.stop) {
            BW_CUDA(cudaEventRecord(ctx->ev_stop, s));
        } else {
            // BW_LAUNCH_L2_WINDOW: the captured kernels keep the depth array persisting in L2
            const bool window = cfg && (cfg->flags & BW_LAUNCH_L2_WINDOW);
            auto capture = [&](cudaStream_t cap, cudaGraph_t body, cudaGraphConditionalHandle handle) -> int {
                L2Window win;
                if (window) BW_TRY(l2_window_begin(ctx, cap, levels, n * sizeof(int32_t), win, false));
                BW_CUDA(cudaStreamBeginCaptureToGraph(cap, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed));
                const int launched = level_kernels(cap, true, false);
                k_bfs_step<<<1, 32, 0, cap>>>(ctx->bfs_ctl, log, log_cap, handle);
                cudaGraph_t captured = body;
                const cudaError_t e = cudaStreamEndCapture(cap, &captured);
                l2_window_end(win);                 // before its stream goes
                BW_TRY(launched);
                BW_CUDA(e);
                return BW_OK;
            };
            auto loop = [&](cudaGraph_t graph, cudaStream_t cap) -> int {
                cudaGraphConditionalHandle handle;
                BW_CUDA(cudaGraphConditionalHandleCreate(&handle, graph, 1, cudaGraphCondAssignDefault));
                cudaGraphNodeParams cp = {};
                cp.type = cudaGraphNodeTypeConditional;
                cp.conditional.handle = handle;
                cp.conditional.type = cudaGraphCondTypeWhile;
                cp.conditional.size = 1;
                cudaGraphNode_t cnode;
                BW_CUDA(cudaGraphAddNode(&cnode, graph, nullptr, nullptr, 0, &cp));
                BW_TRY(capture(cap, cp.conditional.phGraph_out[0], handle));
                cudaGraphExec_t exec = nullptr;
                BW_CUDA(cudaGraphInstantiate(&exec, graph, 0));
                cudaError_t e = cudaGraphLaunch(exec, s);
                if (e == cudaSuccess) e = cudaEventRecord(ctx->ev_stop, s);
                if (e == cudaSuccess)
                    e = cudaMemcpyAsync(ctx->bfs_ctl_host, ctx->bfs_ctl, sizeof(BfsCtl), cudaMemcpyDeviceToHost, s);
                if (e == cudaSuccess) e = cudaStreamSynchronize(s);
                cudaGraphExecDestroy(exec);
                BW_CUDA(e);
                end.status = ctx->bfs_ctl_host->status;
                end.levels_done = ctx->bfs_ctl_host->levels_done;
                end.visited = ctx->bfs_ctl_host->visited;
                return BW_OK;
            };
            cudaGraph_t graph = nullptr;
            cudaStream_t cap = nullptr;             // the caller's may be the legacy default stream
            BW_CUDA(cudaGraphCreate(&graph, 0));
            const cudaError_t e = cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking);
            const int rc = e == cudaSuccess ? loop(graph, cap) : BW_ERR_CUDA;
            if (cap) cudaStreamDestroy(cap);
            cudaGraphDestroy(graph);
            BW_CUDA(e);
            BW_TRY(rc);
        }
        return BW_OK;
    };
    const int rc = traverse();
    if (rc != BW_OK) {
        if (log) cudaFreeAsync(log, s);
        return rc;
    }
    if (log_cap) {
        BW_CUDA(cudaStreamSynchronize(s));
        const uint32_t got = std::min(end.levels_done, log_cap);
        LevelSlot *tmp = new LevelSlot[got ? got : 1];
        BW_CUDA(cudaMemcpy(tmp, log, got * sizeof(LevelSlot), cudaMemcpyDeviceToHost));
        for (uint32_t i = 0; i < got; i++) fill_stats(tmp[i], variant, &stats[i]);
        delete[] tmp;
        BW_CUDA(cudaFreeAsync(log, s));
    }
    if (result) {
        BW_TRY(traversed_edges(ctx, g, levels, s, &result->traversed_edges));
        float ms = 0.0f;
        BW_CUDA(cudaEventSynchronize(ctx->ev_stop));
        BW_CUDA(cudaEventElapsedTime(&ms, ctx->ev_start, ctx->ev_stop));
        result->level_count = end.levels_done;
        result->visited = end.visited;
        result->device_ms = ms;
    }
    return end.status ? static_cast<int>(end.status) : BW_OK;
}

int prepare(bw_context *ctx, const bw_graph_view *g, int reps, bool side, int32_t *levels,
            uint32_t root, cudaStream_t s)
{
    if (!ctx || !levels) return BW_ERR_INVALID_ARGUMENT;
    BW_TRY(validate_graph(g));
    if (root >= g->vertex_count) return BW_ERR_INVALID_ARGUMENT;
    BW_TRY(check_reps(g, reps));
    BW_TRY(ensure_bfs_scratch(ctx, g->vertex_count, g->edge_count));
    if (side) BW_TRY(ensure_outdeg(ctx, g, s));
    return BW_OK;
}

}  // namespace

// A graph without edges (the edge arrays may then be null): level 0 expands
// {root} and finds nothing, so the root gets depth 0 and every other vertex
// INT_MAX after one level (bfs/bfs.cpp:80-107); no level kernel runs.
int bfs_edgeless(bw_context *ctx, const bw_graph_view *g, int variant, uint32_t root, int32_t *levels,
                 bw_bfs_result *result, bw_bfs_level_stats *stats, uint32_t stats_capacity, cudaStream_t s)
{
    if (!ctx || !levels) return BW_ERR_INVALID_ARGUMENT;
    BW_TRY(validate_graph(g));
    if (root >= g->vertex_count) return BW_ERR_INVALID_ARGUMENT;
    if (!g->fwd_vertices && !g->rev_vertices) return BW_ERR_MISSING_REPRESENTATION;
    BW_TRY(ensure_bfs_scratch(ctx, g->vertex_count, 0));
    k_bfs_init_side<<<ctx->sm_count * 4, 256, 0, s>>>(levels, g->vertex_count, root, ctx->queue[0], ctx->bfs_ctl,
                                                     0, nullptr);
    BW_CUDA(cudaGetLastError());
    BW_CUDA(cudaStreamSynchronize(s));
    if (stats && stats_capacity) {
        stats[0] = bw_bfs_level_stats{};
        stats[0].variant = static_cast<uint32_t>(variant);
    }
    if (result) {
        result->level_count = 1;
        result->visited = 1;
        result->traversed_edges = 0;
        result->device_ms = 0.0;
    }
    return BW_OK;
}

// Shared with bw_learn.cu.
int bfs_prepare(bw_context *ctx, const bw_graph_view *g, int reps, bool side, int32_t *levels, uint32_t root,
                cudaStream_t s)
{ return prepare(ctx, g, reps, side, levels, root, s); }

int bfs_plan(const bw_context *ctx, const bw_graph_view *g, int variant, bool side, const bw_launch_config *cfg,
             BfsKernelFn *k, BfsKernelFn *k2, unsigned *block, unsigned *grid, size_t *smem, unsigned *grid2)
{
    Launch l;
    BW_TRY(plan_launch(ctx, g, variant, side, cfg, &l));
    *k = l.k; *k2 = l.k2; *block = l.block; *grid = l.grid; *smem = l.smem; *grid2 = l.grid2;
    return BW_OK;
}

BfsArgs bfs_args(bw_context *ctx, const bw_graph_view *g, int32_t *levels, int32_t depth,
                 const bw_launch_config *cfg)
{ return make_args(ctx, g, levels, depth, cfg); }

int bfs_variant_reps(int v) { return variant_reps(v); }

int bfs_read_slot(bw_context *ctx, int slot, cudaStream_t s) { return post_and_wait(ctx, slot, s); }

int bfs_traversed(bw_context *ctx, const bw_graph_view *g, int32_t *levels, cudaStream_t s, uint64_t *out)
{ return traversed_edges(ctx, g, levels, s, out); }

}  // namespace bw

using namespace bw;

extern "C" {

int bw_bfs_variant_count(void) { return VARIANT_COUNT; }

const char *bw_bfs_variant_name(int variant)
{
    return (variant >= 0 && variant < VARIANT_COUNT) ? names().names[variant].c_str() : nullptr;
}

int bw_bfs_variant_lookup(const char *name)
{
    if (!name) return -1;
    for (int i = 0; i < VARIANT_COUNT; i++)
        if (names().names[i] == name) return i;
    return -1;
}

int bw_bfs_variant_reps(int variant) { return variant_reps(variant); }

int bw_bfs_init(bw_context *ctx, uint64_t vertex_count, uint32_t root, int32_t *levels, void *stream)
{
    if (!ctx || !levels || vertex_count == 0 || root >= vertex_count) return BW_ERR_INVALID_ARGUMENT;
    BW_TRY(ensure_bfs_scratch(ctx, vertex_count, 0));
    k_bfs_init_side<<<ctx->sm_count * 4, 256, 0, as_stream(stream)>>>(levels, vertex_count, root, ctx->queue[0],
                                                                      ctx->bfs_ctl, 0, nullptr);
    BW_CUDA(cudaGetLastError());
    return BW_OK;
}

int bw_bfs_level(bw_context *ctx, const bw_graph_view *g, int variant, int32_t *levels, int32_t depth,
                 const bw_launch_config *cfg, uint32_t *frontier, void *stream)
{
    if (!ctx || !levels || depth < 0) return BW_ERR_INVALID_ARGUMENT;
    BW_TRY(validate_graph(g));
    if (variant < 0 || variant >= VARIANT_COUNT) return BW_ERR_UNKNOWN_VARIANT;
    if (!ctx->bfs_ctl || ctx->bfs_n_cap < g->vertex_count) return BW_ERR_INVALID_ARGUMENT;  // bw_bfs_init first
    if (g->edge_count == 0) {
        // no edges: the level visits nothing; its counts read as zero
        cudaStream_t s = as_stream(stream);
        BW_CUDA(cudaMemsetAsync(&ctx->bfs_ctl->slot[depth % 3], 0, sizeof(LevelSlot), s));
        BW_CUDA(cudaStreamSynchronize(s));
        if (frontier) *frontier = 0;
        return BW_OK;
    }
    BW_TRY(check_reps(g, variant_reps(variant)));
    BW_TRY(ensure_bfs_scratch(ctx, g->vertex_count, g->edge_count));
    Launch plan;
    // Queue-driven variants need the queue kept by every level: levels run
    // through this entry point always emit it.
    const bool side = g->fwd_vertices != nullptr;
    if (side) BW_TRY(ensure_outdeg(ctx, g, as_stream(stream)));
    if (!side && (variant == V_FRONTIER_PUSH)) return BW_ERR_MISSING_REPRESENTATION;
    BW_TRY(plan_launch(ctx, g, variant, side, cfg, &plan));
    cudaStream_t s = as_stream(stream);
    BfsArgs a = make_args(ctx, g, levels, depth, cfg);
    BW_TRY(launch(plan, a, s));
    BW_CUDA(cudaMemcpyAsync(&ctx->bfs_ctl_host->slot[depth % 3], &ctx->bfs_ctl->slot[depth % 3],
                            sizeof(LevelSlot), cudaMemcpyDeviceToHost, s));
    BW_CUDA(cudaStreamSynchronize(s));
    if (frontier) *frontier = ctx->bfs_ctl_host->slot[depth % 3].frontier;
    return BW_OK;
}

int bw_bfs_run(bw_context *ctx, const bw_graph_view *g, int variant, uint32_t root, int32_t *levels,
               const bw_launch_config *cfg, int loop_mode, uint32_t max_levels,
               bw_bfs_result *result, bw_bfs_level_stats *stats, uint32_t stats_capacity,
               void *stream)
{
    if (variant < 0 || variant >= VARIANT_COUNT) return BW_ERR_UNKNOWN_VARIANT;
    // frontier-push needs the queue of the level before it, which only it
    // (or a side-output level) writes; a fixed frontier-push run keeps it.
    const bool side = stats != nullptr && stats_capacity > 0;
    int reps = variant_reps(variant) | (side ? REP_FWD_CSR : 0);
    cudaStream_t s = as_stream(stream);
    if (loop_mode != BW_LOOP_GRAPH && loop_mode != BW_LOOP_HOST) return BW_ERR_INVALID_ARGUMENT;
    if (g && g->edge_count == 0) return bfs_edgeless(ctx, g, variant, root, levels, result, stats, stats_capacity, s);
    BW_TRY(prepare(ctx, g, reps, side, levels, root, s));
    L2Window win;                  // BW_LAUNCH_L2_WINDOW: the depth array persisting in L2
    if (cfg && (cfg->flags & BW_LAUNCH_L2_WINDOW))
        BW_TRY(l2_window_begin(ctx, s, levels, g->vertex_count * sizeof(int32_t), win));
    if (loop_mode == BW_LOOP_GRAPH)
        return run_graph(ctx, g, variant, root, levels, cfg, max_levels, side, result, stats, stats_capacity, s);
    if (loop_mode != BW_LOOP_HOST) return BW_ERR_INVALID_ARGUMENT;
    int32_t sched = variant;
    return run_host(ctx, g, &sched, 1, root, levels, cfg, max_levels, 0, side, result, stats,
                    stats_capacity, s);
}

int bw_bfs_run_schedule(bw_context *ctx, const bw_graph_view *g, const int32_t *schedule,
                        uint32_t schedule_len, uint32_t root, int32_t *levels,
                        const bw_launch_config *cfg, uint32_t max_levels, int time_levels,
                        bw_bfs_result *result, bw_bfs_level_stats *stats, uint32_t stats_capacity,
                        void *stream)
{
    if (!schedule || schedule_len == 0) return BW_ERR_INVALID_ARGUMENT;
    // Mixed schedules hand the frontier from one variant to the next, so
    // every level emits the queue and statistics (needs the forward CSR).
    int reps = REP_FWD_CSR;
    for (uint32_t i = 0; i < schedule_len; i++) {
        if (schedule[i] < 0 || schedule[i] >= VARIANT_COUNT) return BW_ERR_UNKNOWN_VARIANT;
        reps |= variant_reps(schedule[i]);
    }
    cudaStream_t s = as_stream(stream);
    if (g && g->edge_count == 0)
        return bfs_edgeless(ctx, g, schedule[0], root, levels, result, stats, stats_capacity, s);
    BW_TRY(prepare(ctx, g, reps, true, levels, root, s));
    return run_host(ctx, g, schedule, schedule_len, root, levels, cfg, max_levels, time_levels, true,
                    result, stats, stats_capacity, s);
}

}  // extern "C"
