// Batched persistent traversal: many graphs, or many BFS sources, in one
// launch.  Each CTA takes units from a device work queue (an atomic cursor
// over a largest-first order) and runs each unit to completion with
// CTA-level barriers between BFS levels and PageRank iterations.
//
// Per unit: BFS with CTA-wide frontier queues in global scratch (private to
// the CTA), warp-cooperative row expansion (32 frontier rows concatenated per
// warp step) and CTA-cooperative expansion of rows above BATCH_HEAVY edges;
// for whole-graph units, then `pr_iterations` PageRank iterations of that
// graph alone, each vertex summing its reverse row in row order with the
// reference's consolidation (pagerank/vertex_pull.cu:23-29,
// pagerank/pagerank.cu:131-136), so ranks are bit-identical to a
// single-graph vertex-pull run.
#include <algorithm>
#include <climits>

#include <cooperative_groups.h>

#include "bw_consolidate.h"
#include "bw_internal.cuh"
#include "bw_seqsum_warp.cuh"

namespace bw {
namespace {
namespace cg = cooperative_groups;

constexpr int BATCH_THREADS = 512;
constexpr int BATCH_WARPS = BATCH_THREADS / 32;
constexpr uint32_t BATCH_HEAVY = 1024;    // rows above this are expanded by the whole CTA
constexpr uint32_t HEAVY_SLOTS = 256;
constexpr uint32_t NO_UNIT = 0xffffffffu;
constexpr float DAMPING = 0.85f;
constexpr uint32_t BATCH_PR_LIGHT = 256;  // PageRank rows above this are summed by a whole warp
constexpr int BATCH_PR_UNROLL = 8;
constexpr int BATCH_BFS_UNROLL = 4;
constexpr uint32_t BATCH_BU_DIV = 24;     // default push/pull divisor: bottom-up above 1/24 of the unit
constexpr uint32_t BATCH_PR_L = 8;        // warp sums: windows of 32 x 8 terms
constexpr uint64_t PACKED_MAX_VERTICES = uint64_t(1) << 29;   // the work list's row ids
constexpr uint64_t MULTI_MIN_VERTICES = 98304, MULTI_MAX_VERTICES = uint64_t(1) << 31;
constexpr uint32_t PACKED_MIN_UNIT = 4096;
constexpr uint64_t PACKED_MIN_WORK = 16384;                   // vertices of the largest unit x iterations

struct BatchArgs {
    const uint32_t *fwd_v, *fwd_e, *rev_v, *rev_e;
    uint64_t n;
    int mode;
    const uint32_t *goff;
    const uint32_t *roots, *order;
    uint32_t units;
    uint32_t *cursor;
    uint32_t *queues;         // per CTA: 2 * qcap
    float *contrib;           // per CTA: 2 * qcap
    uint32_t qcap;
    int32_t *levels;
    float *ranks;
    uint32_t pr_iters;
    uint32_t vis_words;       // > 0: the unit's visited set is a shared-memory bitmap of this many words
    uint32_t bu_div;          // a level whose frontier holds more than 1/bu_div of the unit runs bottom-up
    unsigned long long *traversed;
    // Many sources that bfs_multi_source has begun: the units of pass t / pass
    // are done (MS_DONE), have their depths up to resume[t / pass], or start at
    // their roots (0).  nullptr: all start at their roots.
    const int32_t *resume;
    uint32_t pass;
};

__device__ __forceinline__ bool relax_local(int32_t *lv, uint32_t v, int32_t nd)
{ return lv[v] > nd && atomicMin(&lv[v], nd) > nd; }

// The frontier at depth `from` and the visited set from the depths of the
// vertices 0 .. n - 1, RESUME_UNROLL loads in flight a lane.
constexpr int RESUME_UNROLL = 8;
__device__ void resume_unit(const int32_t *lv, uint32_t n, int32_t from, uint32_t *vis, uint32_t *queue, uint32_t *qlen,
                            unsigned wib, unsigned lane)
{
    for (uint64_t v0 = wib * 32; v0 < n; v0 += uint64_t(BATCH_THREADS) * RESUME_UNROLL) {
        int32_t d[RESUME_UNROLL];
#pragma unroll
        for (int j = 0; j < RESUME_UNROLL; j++) {
            const uint64_t v = v0 + uint64_t(j) * BATCH_THREADS + lane;
            d[j] = v < n ? lv[v] : INF;
        }
#pragma unroll
        for (int j = 0; j < RESUME_UNROLL; j++) {
            const uint64_t w0 = v0 + uint64_t(j) * BATCH_THREADS;
            const unsigned seen = __ballot_sync(FULL_MASK, d[j] != INF), here = __ballot_sync(FULL_MASK, d[j] == from);
            if (vis && lane == 0 && w0 < n) vis[w0 / 32] = seen;
            if (here == 0) continue;
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(qlen, static_cast<uint32_t>(__popc(here)));
            base = __shfl_sync(FULL_MASK, base, 0);
            if (d[j] == from) queue[base + __popc(here & ((1u << lane) - 1u))] = static_cast<uint32_t>(w0) + lane;
        }
    }
}

// RESUME: units may have been begun (a.resume).  Its looks at that in the one
// form took 7% of a call with 16 graphs of 200 to 900 vertices (241 -> 259 us).
template<bool RESUME>
__global__ void __launch_bounds__(BATCH_THREADS, 2) k_batch(BatchArgs a)
{
    __shared__ uint32_t s_unit, s_qlen[2], s_heavy_n;
    __shared__ int32_t s_from;                         // RESUME
    __shared__ uint32_t s_heavy[HEAVY_SLOTS];
    __shared__ uint32_t s_excl[BATCH_WARPS][32], s_start[BATCH_WARPS][32];
    __shared__ double s_base;
    __shared__ uint32_t s_long_n, s_job;
    __shared__ float s_stage[BATCH_WARPS][33 * BATCH_PR_L];
    extern __shared__ uint32_t s_vis[];
    __shared__ unsigned long long s_trav;
    const unsigned tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
    uint32_t *q[2] = {a.queues + static_cast<size_t>(blockIdx.x) * 2 * a.qcap,
                      a.queues + static_cast<size_t>(blockIdx.x) * 2 * a.qcap + a.qcap};
    float *cbuf[2] = {a.contrib + static_cast<size_t>(blockIdx.x) * 2 * a.qcap,
                      a.contrib + static_cast<size_t>(blockIdx.x) * 2 * a.qcap + a.qcap};
    for (;;) {
        if (tid == 0) {
            uint32_t t;
            do t = atomicAdd(a.cursor, 1u);
            while (RESUME && a.resume && t < a.units && a.resume[t / a.pass] == MS_DONE);
            s_unit = t < a.units ? (a.order ? a.order[t] : t) : NO_UNIT;
            if constexpr (RESUME) s_from = a.resume && t < a.units ? a.resume[t / a.pass] : 0;
            s_trav = 0;
        }
        __syncthreads();
        const uint32_t unit = s_unit;
        if (unit == NO_UNIT) break;
        uint32_t vb, ve;
        int32_t *lv;
        if (a.mode == BW_BATCH_GRAPHS) {
            vb = a.goff[unit];
            ve = a.goff[unit + 1];
            lv = a.levels;
        } else {
            vb = 0;
            ve = static_cast<uint32_t>(a.n);
            lv = a.levels + static_cast<size_t>(unit) * a.n;
        }
        const int32_t from = RESUME ? s_from : 0;
        const bool bitmap = a.vis_words != 0;
        if (!RESUME || from == 0) {
            const uint32_t root = a.roots[unit];
            for (uint32_t v = vb + tid; v < ve; v += BATCH_THREADS) lv[v] = v == root ? 0 : INF;
            if (bitmap) {
                for (uint32_t w = tid; w < (ve - vb + 31) / 32; w += BATCH_THREADS) s_vis[w] = 0u;
                __syncthreads();
            }
            if (tid == 0) {
                if (bitmap) s_vis[(root - vb) >> 5] = 1u << ((root - vb) & 31);
                q[0][0] = root;
                s_qlen[0] = 1;
                s_qlen[1] = 0;
                s_heavy_n = 0;
            }
        } else {
            if (tid == 0) s_qlen[0] = s_qlen[1] = s_heavy_n = 0;
            __syncthreads();
            resume_unit(lv, ve, from, bitmap ? s_vis : nullptr, q[from & 1], &s_qlen[from & 1], wib, lane);
        }
        __syncthreads();
        // ------------------------------ BFS ------------------------------
        for (int32_t depth = from;; depth++) {
            const uint32_t len = s_qlen[depth & 1];
            if (len == 0) break;
            const int32_t nd = depth + 1;
            const uint32_t *qin = q[depth & 1];
            uint32_t *qout = q[(depth + 1) & 1];
            uint32_t *olen = &s_qlen[(depth + 1) & 1];
            // first visit of u: the shared-memory bitmap answers without a
            // global access (and its atomic is a shared one); the depth is
            // then stored once
            auto relax = [&](uint32_t u) -> bool {
                if (!bitmap) return relax_local(lv, u, nd);
                const uint32_t w = (u - vb) >> 5, bit = 1u << ((u - vb) & 31);
                if (s_vis[w] & bit) return false;
                if (atomicOr(&s_vis[w], bit) & bit) return false;
                lv[u] = nd;
                return true;
            };
            auto visit = [&](uint32_t u) {
                if (relax(u)) {
                    cg::coalesced_group g = cg::coalesced_threads();
                    uint32_t base = 0;
                    if (g.thread_rank() == 0) base = atomicAdd(olen, g.size());
                    base = g.shfl(base, 0);
                    qout[base + g.thread_rank()] = u;
                }
            };
            // A frontier above 1/bu_div of the unit's vertices: bottom-up.
            // Every vertex not yet reached looks for an in-neighbour reached
            // before this level, which is then at `depth` (one at a smaller
            // depth would have reached it already); the bitmap answers, and
            // is updated only once the level is done, so that it reads as of
            // the level's start.
            const uint32_t nunit = ve - vb;
            const bool bottom_up = bitmap && a.rev_v && len > nunit / a.bu_div;
            if (bottom_up) {
                const uint32_t words = (nunit + 31) / 32;
                for (uint32_t w = tid; w < words; w += BATCH_THREADS) {
                    uint32_t todo = ~s_vis[w];
                    if (w == words - 1 && (nunit & 31)) todo &= (1u << (nunit & 31)) - 1u;
                    while (todo) {
                        const uint32_t v = vb + w * 32 + (__ffs(todo) - 1);
                        todo &= todo - 1;
                        const uint32_t s = a.rev_v[v], e = a.rev_v[v + 1];
                        bool found = false;
                        for (uint32_t i = s; i < e && !found; i += BATCH_BFS_UNROLL) {
                            uint32_t pu[BATCH_BFS_UNROLL];
#pragma unroll
                            for (int j = 0; j < BATCH_BFS_UNROLL; j++)
                                pu[j] = i + j < e ? __ldg(a.rev_e + i + j) - vb : NO_UNIT;
#pragma unroll
                            for (int j = 0; j < BATCH_BFS_UNROLL; j++)
                                if (pu[j] != NO_UNIT) found |= ((s_vis[pu[j] >> 5] >> (pu[j] & 31)) & 1u) != 0u;
                        }
                        if (found) {
                            lv[v] = nd;
                            cg::coalesced_group g = cg::coalesced_threads();
                            uint32_t base = 0;
                            if (g.thread_rank() == 0) base = atomicAdd(olen, g.size());
                            base = g.shfl(base, 0);
                            qout[base + g.thread_rank()] = v;
                        }
                    }
                }
                __syncthreads();
                for (uint32_t i = tid; i < *olen; i += BATCH_THREADS) {
                    const uint32_t u = qout[i] - vb;
                    atomicOr(&s_vis[u >> 5], 1u << (u & 31));
                }
            }
            for (uint32_t t = wib * 32; !bottom_up && t < len; t += BATCH_THREADS) {
                const uint32_t i = t + lane;
                uint32_t v = 0, s = 0, d = 0;
                if (i < len) {
                    v = qin[i];
                    s = a.fwd_v[v];
                    d = a.fwd_v[v + 1] - s;
                }
                if (d > BATCH_HEAVY) {
                    const uint32_t slot = atomicAdd(&s_heavy_n, 1u);
                    if (slot < HEAVY_SLOTS) { s_heavy[slot] = v; d = 0; }   // else: this warp expands it
                }
                uint32_t incl = d;
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(FULL_MASK, incl, o);
                    if (lane >= static_cast<unsigned>(o)) incl += y;
                }
                const uint32_t total = __shfl_sync(FULL_MASK, incl, 31);
                s_excl[wib][lane] = incl - d;
                s_start[wib][lane] = s;
                __syncwarp();
                // edge k of the 32 concatenated rows: a per-lane cursor over
                // the rows' exclusive offsets (k grows), BATCH_BFS_UNROLL
                // neighbours' indices in flight before their visits
                uint32_t seg = 0;
                for (uint32_t k0 = 0; k0 < total; k0 += 32 * BATCH_BFS_UNROLL) {
                    uint32_t u[BATCH_BFS_UNROLL];
#pragma unroll
                    for (int j = 0; j < BATCH_BFS_UNROLL; j++) {
                        const uint32_t k = k0 + j * 32 + lane;
                        u[j] = NO_UNIT;
                        if (k < total) {
                            while (seg < 31 && s_excl[wib][seg + 1] <= k) seg++;
                            u[j] = __ldg(a.fwd_e + s_start[wib][seg] + (k - s_excl[wib][seg]));
                        }
                    }
#pragma unroll
                    for (int j = 0; j < BATCH_BFS_UNROLL; j++)
                        if (u[j] != NO_UNIT) visit(u[j]);
                }
                __syncwarp();
            }
            __syncthreads();
            const uint32_t heavy = bottom_up ? 0u : min(s_heavy_n, HEAVY_SLOTS);
            for (uint32_t h = 0; h < heavy; h++) {
                const uint32_t v = s_heavy[h];
                const uint32_t s = a.fwd_v[v], e = a.fwd_v[v + 1];
                for (uint32_t i0 = s; i0 < e; i0 += BATCH_THREADS * BATCH_BFS_UNROLL) {
                    uint32_t u[BATCH_BFS_UNROLL];
#pragma unroll
                    for (int j = 0; j < BATCH_BFS_UNROLL; j++) {
                        const uint32_t i = i0 + j * BATCH_THREADS + tid;
                        u[j] = i < e ? __ldg(a.fwd_e + i) : NO_UNIT;
                    }
#pragma unroll
                    for (int j = 0; j < BATCH_BFS_UNROLL; j++)
                        if (u[j] != NO_UNIT) visit(u[j]);
                }
            }
            __syncthreads();
            if (tid == 0) {
                s_qlen[depth & 1] = 0;
                s_heavy_n = 0;
            }
            __syncthreads();
        }
        // traversed edges: out-degrees of reached vertices
        unsigned long long trav = 0;
        for (uint32_t v = vb + tid; v < ve; v += BATCH_THREADS)
            if (lv[v] != INF) trav += a.fwd_v[v + 1] - a.fwd_v[v];
        for (int o = 16; o > 0; o >>= 1) trav += __shfl_xor_sync(FULL_MASK, trav, o);
        if (lane == 0 && trav) atomicAdd(&s_trav, trav);
        // --------------------------- PageRank -----------------------------
        // Every row is summed in row order from +0 (bit-identical to the
        // reference's loop).  Rows of at most BATCH_PR_LIGHT terms: one lane
        // each, BATCH_PR_UNROLL gathers in flight.  Longer rows: one warp
        // each (warp_sequential_continue_load: coalesced gathers staged in
        // shared memory, a serial start by one lane, then binade-map scans),
        // so that a hub's row no longer holds the CTA's iteration.  Warps take
        // jobs -- the long rows, then chunks of 32 vertices -- from a
        // shared-memory counter.
        if (a.mode == BW_BATCH_GRAPHS && a.pr_iters) {
            const uint32_t ng = ve - vb;
            if (tid == 0) {
                s_base = (1.0 - static_cast<double>(DAMPING)) / static_cast<double>(ng);
                s_long_n = 0;
                s_job = 0;
            }
            __syncthreads();
            const double base = s_base;
            const float init = __fdiv_rn(1.0f, static_cast<float>(ng));
            uint32_t *long_rows = q[0];                  // the BFS queues are free now
            for (uint32_t v = vb + tid; v < ve; v += BATCH_THREADS) {
                const uint32_t d = a.fwd_v[v + 1] - a.fwd_v[v];
                a.ranks[v] = init;
                cbuf[0][v - vb] = d ? __fdiv_rn(init, static_cast<float>(d)) : 0.0f;
                if (a.rev_v[v + 1] - a.rev_v[v] > BATCH_PR_LIGHT) long_rows[atomicAdd(&s_long_n, 1u)] = v;
            }
            __syncthreads();
            const uint32_t n_long = s_long_n, jobs = n_long + (ng + 31) / 32;
            auto finish = [&](uint32_t v, float sum, float *cout) {
                const float scaled = __fmul_rn(DAMPING, sum);
                bool ok;
                const uint32_t rb = bwcons::add_round_bits(static_cast<uint64_t>(__double_as_longlong(base)),
                                                           __float_as_uint(scaled), ok);
                const float nr = ok ? __uint_as_float(rb) : __double2float_rn(__dadd_rn(base, static_cast<double>(scaled)));
                a.ranks[v] = nr;
                const uint32_t d = a.fwd_v[v + 1] - a.fwd_v[v];
                cout[v - vb] = d ? __fdiv_rn(nr, static_cast<float>(d)) : 0.0f;
            };
            for (uint32_t it = 1; it <= a.pr_iters; it++) {
                const float *cin = cbuf[(it - 1) & 1];
                float *cout = cbuf[it & 1];
                for (;;) {
                    uint32_t job = 0;
                    if (lane == 0) job = atomicAdd(&s_job, 1u);
                    job = __shfl_sync(FULL_MASK, job, 0);
                    if (job >= jobs) break;
                    if (job < n_long) {
                        const uint32_t v = long_rows[job];
                        const uint32_t s = a.rev_v[v], len = a.rev_v[v + 1] - s;
                        auto load = [&](uint32_t i) { return cin[__ldg(a.rev_e + s + i) - vb]; };
                        uint32_t sb = 0;
                        float sum;
                        if (warp_sequential_continue_load<BATCH_PR_L>(load, 0, len, sb, s_stage[wib], lane)) {
                            sum = __uint_as_float(sb);
                        } else {                         // terms outside the maps' domain: the plain loop
                            sum = 0.0f;
                            if (lane == 0)
                                for (uint32_t i = 0; i < len; i++) sum = __fadd_rn(sum, load(i));
                        }
                        if (lane == 0) finish(v, sum, cout);
                    } else {
                        const uint32_t v = vb + (job - n_long) * 32 + lane;
                        if (v < ve) {
                            const uint32_t s = a.rev_v[v], e = a.rev_v[v + 1];
                            if (e - s <= BATCH_PR_LIGHT) {
                                float sum = 0.0f;
                                for (uint32_t i = s; i < e; i += BATCH_PR_UNROLL) {
                                    float t[BATCH_PR_UNROLL];
#pragma unroll
                                    for (int k = 0; k < BATCH_PR_UNROLL; k++)
                                        t[k] = i + k < e ? cin[__ldg(a.rev_e + i + k) - vb] : 0.0f;
#pragma unroll
                                    for (int k = 0; k < BATCH_PR_UNROLL; k++)
                                        if (i + k < e) sum = __fadd_rn(sum, t[k]);
                                }
                                finish(v, sum, cout);
                            }
                        }
                    }
                }
                __syncthreads();
                if (tid == 0) s_job = 0;
                __syncthreads();
            }
        }
        __syncthreads();
        if (tid == 0 && s_trav) atomicAdd(a.traversed, s_trav);
    }
}

// Whether the graphs' PageRank runs as one set of rows over the whole GPU
// (pagerank_run_packed) or inside k_batch, a CTA per graph.  A CTA sums about
// 0.6 G terms/s, so a large graph ends long after the rest: 512 R-MAT graphs
// of 1K-200K vertices (343M edges), BFS and 20 iterations, 109 ms in k_batch
// and 30.5 ms packed on GB300; 16 graphs of 4K-200K 75 and 3.5 ms.  Small
// graphs balance well on CTAs and need no set-up: 350 graphs of 1K-4K
// vertices 1.65 and 1.83 ms, of 200-800 0.27 and 0.76 ms.  One iteration of
// 64 graphs of up to 8K vertices: 0.19 and 0.26 ms (the set-up, 0.15 ms).
bool packed_pagerank(const bw_graph_view *g, uint32_t max_unit_vertices, uint32_t iterations)
{
    return g->vertex_count < PACKED_MAX_VERTICES && max_unit_vertices >= PACKED_MIN_UNIT &&
           uint64_t(max_unit_vertices) * iterations >= PACKED_MIN_WORK;
}

// Whether many sources run together, a bit each (bfs_multi_source), or each on
// a CTA.  A level costs two launches and at least 20 us, so small graphs stay
// on CTAs.  Measured on GB300, together / on CTAs, ms for 4 and 512 sources:
// 30,000 vertices R-MAT 0.26 / 0.21 and 0.40 / 0.46, ER 0.26 / 0.17 and
// 0.43 / 0.48; 60,000 R-MAT 0.31 / 0.52 and 0.45 / 0.83, BA 0.34 / 0.25 and
// 0.57 / 0.76; 120,000 R-MAT 0.30 / 0.48 and 0.47 / 1.64, ER 0.28 / 0.82 and
// 0.50 / 2.09, BA 0.36 / 0.46 and 0.63 / 1.57.  A traversal of more than 31
// levels is finished on CTAs from there: 4 and 512 sources on R-MAT-18
// symmetrised with a path of 60 vertices 1.1 and 2.1 ms (all on CTAs 3.0 and
// 4.9, without the path 0.50 and 0.94).  What is given back as a mesh costs
// 0.2 to 0.9 ms first: 1 and 512 sources on the 512 x 512 grid 3.43 and 8.21
// (3.20 and 7.77 on CTAs alone), on the 1024 x 1024 grid 10.1 and 44.1 (9.7 and
// 43.2).
bool multi_source(const bw_graph_view *g, int mode)
{
    return mode == BW_BATCH_SOURCES && g->rev_vertices && g->rev_edges && g->vertex_count >= MULTI_MIN_VERTICES &&
           g->vertex_count <= MULTI_MAX_VERTICES;
}

}  // namespace
}  // namespace bw

using namespace bw;

extern "C" int bw_batch_run(bw_context *ctx, const bw_graph_view *g, int mode, const uint32_t *graph_offsets,
                            uint32_t graph_count, const uint32_t *roots, const uint32_t *order, uint32_t unit_count,
                            uint32_t max_unit_vertices, uint32_t pr_iterations, int32_t *levels, float *ranks,
                            const bw_launch_config *cfg, bw_batch_result *result, void *stream)
{
    if (!ctx || !g || !roots || !levels || !g->fwd_vertices || !g->fwd_edges) return BW_ERR_INVALID_ARGUMENT;
    if (mode != BW_BATCH_GRAPHS && mode != BW_BATCH_SOURCES) return BW_ERR_INVALID_ARGUMENT;
    if (mode == BW_BATCH_GRAPHS) {
        if (!graph_offsets || graph_count == 0 || unit_count != graph_count) return BW_ERR_INVALID_ARGUMENT;
        if (pr_iterations && (!ranks || !g->rev_vertices || !g->rev_edges)) return BW_ERR_MISSING_REPRESENTATION;
    } else if (graph_count != 1 || g->vertex_count > max_unit_vertices) {
        return BW_ERR_INVALID_ARGUMENT;
    }
    if (max_unit_vertices == 0 || g->vertex_count > 0xffffffffULL) return BW_ERR_INVALID_ARGUMENT;
    if (unit_count == 0) {
        if (result) *result = bw_batch_result{};
        return BW_OK;
    }
    cudaStream_t s = as_stream(stream);
    // the visited bitmap of the largest unit in shared memory when it fits
    // beside the kernel's static shared memory; CTAs per SM as it allows
    cudaFuncAttributes fa{};
    const auto kernel = multi_source(g, mode) ? k_batch<true> : k_batch<false>;
    BW_CUDA(cudaFuncGetAttributes(&fa, kernel));
    const uint64_t words = (static_cast<uint64_t>(max_unit_vertices) + 31) / 32;
    const bool bitmap = fa.sharedSizeBytes + words * 4 + 1024 <= static_cast<uint64_t>(ctx->max_smem_optin);
    const size_t dyn = bitmap ? words * 4 : 0;
    BW_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(dyn)));
    int per_sm = 0;
    BW_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, BATCH_THREADS, dyn));
    unsigned grid = static_cast<unsigned>(ctx->sm_count) * static_cast<unsigned>(std::max(1, std::min(per_sm, 2)));
    if (cfg && cfg->grid_size) grid = cfg->grid_size;
    if (cfg && cfg->block_size && cfg->block_size != BATCH_THREADS) return BW_ERR_INVALID_ARGUMENT;
    BW_CUDA(cudaEventRecord(ctx->ev_start, s));         // device_ms: also of a pass that is given back
    uint64_t traversed = 0;                             // of units that need no CTA
    std::vector<int32_t> resume;
    BatchArgs a{};
    if (multi_source(g, mode)) {
        BW_TRY(bfs_multi_source(ctx, g, roots, order, unit_count, levels, &traversed, &a.pass, resume, s));
        if (!resume.empty() && std::all_of(resume.begin(), resume.end(), [](int32_t d) { return d == MS_DONE; })) {
            BW_CUDA(cudaEventRecord(ctx->ev_stop, s));
            BW_CUDA(cudaEventSynchronize(ctx->ev_stop));
            if (result) {
                float ms = 0.0f;
                BW_CUDA(cudaEventElapsedTime(&ms, ctx->ev_start, ctx->ev_stop));
                result->units = unit_count;
                result->traversed_edges = traversed;
                result->device_ms = ms;
            }
            return BW_OK;
        }
    }
    a.fwd_v = g->fwd_vertices; a.fwd_e = g->fwd_edges; a.rev_v = g->rev_vertices; a.rev_e = g->rev_edges;
    a.n = g->vertex_count;
    a.mode = mode;
    a.goff = graph_offsets;
    a.roots = roots;
    a.order = order;
    a.units = unit_count;
    a.qcap = max_unit_vertices;
    a.levels = levels;
    a.ranks = ranks;
    const uint32_t pr = mode == BW_BATCH_GRAPHS ? pr_iterations : 0;
    a.pr_iters = pr;
    if (pr && packed_pagerank(g, max_unit_vertices, pr)) {
        const int rc = pagerank_run_packed(ctx, g, graph_offsets, graph_count, pr, ranks, s);
        if (rc == BW_OK) {
            a.pr_iters = 0;
        } else if (rc == BW_ERR_OUT_OF_MEMORY) {
            cudaGetLastError();                  // its scratch (about 5 bytes per edge) does not fit: a CTA per graph
        } else {
            return rc;
        }
    }
    a.vis_words = bitmap ? static_cast<uint32_t>(words) : 0u;
    a.bu_div = (cfg && cfg->chunk_size) ? cfg->chunk_size : BATCH_BU_DIV;
    const size_t per_cta = static_cast<size_t>(2) * max_unit_vertices;
    char *scratch = nullptr;
    const size_t head = 64 + ((resume.size() * sizeof(int32_t) + 63) & ~size_t(63));
    const size_t bytes = head + grid * per_cta * sizeof(uint32_t) + (a.pr_iters ? grid * per_cta * sizeof(float) : 0);
    BW_CUDA(ctx_malloc_async(ctx, reinterpret_cast<void **>(&scratch), bytes, s));
    BW_CUDA(cudaMemsetAsync(scratch, 0, 64, s));
    a.cursor = reinterpret_cast<uint32_t *>(scratch);
    a.traversed = reinterpret_cast<unsigned long long *>(scratch + 8);
    if (!resume.empty()) {
        BW_CUDA(cudaMemcpyAsync(scratch + 64, resume.data(), resume.size() * sizeof(int32_t), cudaMemcpyHostToDevice, s));
        a.resume = reinterpret_cast<const int32_t *>(scratch + 64);
    }
    a.queues = reinterpret_cast<uint32_t *>(scratch + head);
    a.contrib = a.pr_iters ? reinterpret_cast<float *>(scratch + head + grid * per_cta * sizeof(uint32_t)) : nullptr;
    kernel<<<grid, BATCH_THREADS, dyn, s>>>(a);
    BW_CUDA(cudaGetLastError());
    BW_CUDA(cudaEventRecord(ctx->ev_stop, s));
    unsigned long long trav = 0;
    BW_CUDA(cudaMemcpyAsync(&trav, a.traversed, sizeof trav, cudaMemcpyDeviceToHost, s));
    BW_CUDA(cudaFreeAsync(scratch, s));
    BW_CUDA(cudaStreamSynchronize(s));
    if (result) {
        float ms = 0.0f;
        BW_CUDA(cudaEventElapsedTime(&ms, ctx->ev_start, ctx->ev_stop));
        result->units = unit_count;
        result->traversed_edges = traversed + trav;
        result->device_ms = ms;
    }
    return BW_OK;
}
