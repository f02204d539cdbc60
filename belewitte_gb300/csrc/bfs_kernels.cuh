// BFS level kernels.  One template per reference kernel family
// (bfs/edgelist.cu, rev_edgelist.cu, struct_edgelist.cu,
// rev_struct_edgelist.cu, vertex_push.cu, vertex_pull.cu,
// vertex_push_warp.cu, vertex_pull_warp.cu), parameterised on the
// frontier-count reduction of bfs/bfs.hpp:32-116 and on SIDE (emit the next
// frontier queue and the frontier statistics, needed when levels of
// different variants follow each other), plus the GB300 variants
// frontier-push and frontier-pull.
//
// Every variant computes the same level relation (exact BFS depths): a
// vertex at `depth` gives each unvisited out-neighbour depth + 1, and the
// frontier counter counts each newly visited vertex exactly once.
#pragma once

#include <cooperative_groups.h>
#include "bw_internal.cuh"

namespace bw {
namespace cg = cooperative_groups;

enum Reduction { RED_NORMAL = 0, RED_BULK = 1, RED_WARP = 2, RED_BLOCK = 3 };
enum EdgeLayout { FWD_SOA = 0, REV_SOA = 1, FWD_AOS = 2, REV_AOS = 3 };

// Hub handling of frontier-push: vertices above HEAVY_DEGREE edges are cut
// into HUB_CHUNK-edge chunks that any warp of a second kernel can take.
constexpr uint32_t HEAVY_DEGREE = 256;
constexpr uint32_t HUB_CHUNK = 256;

__device__ __forceinline__ int level_depth(const BfsArgs &a)
{ return a.depth >= 0 ? a.depth : *((volatile int32_t *) &a.ctl->depth); }

__device__ __forceinline__ void reset_slot(LevelSlot *s)
{
    s->frontier = 0; s->qlen = 0; s->fedges = 0; s->lsum = 0; s->lsq = 0;
    s->lmax_bits = 0; s->heavy = 0;
}

// Frontier counter with the four reference strategies
// (bfs/bfs.hpp:32-116).  finish() must be reached by every thread.
template<int RED>
struct Counter {
    uint32_t c = 0;
    __device__ __forceinline__ void hit(uint32_t *g)
    {
        if constexpr (RED == RED_NORMAL) atomicAdd(g, 1u);
        else c++;
    }
    __device__ __forceinline__ void finish(uint32_t *g)
    {
        if constexpr (RED == RED_BULK) {
            if (c) atomicAdd(g, c);
        } else if constexpr (RED == RED_WARP) {
            uint32_t s = __reduce_add_sync(FULL_MASK, c);
            if ((threadIdx.x & 31) == 0 && s) atomicAdd(g, s);
        } else if constexpr (RED == RED_BLOCK) {
            __shared__ uint32_t part[32];
            const unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
            uint32_t s = __reduce_add_sync(FULL_MASK, c);
            if (lane == 0) part[wid] = s;
            __syncthreads();
            if (wid == 0) {
                s = lane < (blockDim.x >> 5) ? part[lane] : 0u;
                s = __reduce_add_sync(FULL_MASK, s);
                if (lane == 0 && s) atomicAdd(g, s);
            }
        }
    }
};

// Warp-aggregated append of `v` to a queue; safe in divergent code.
__device__ __forceinline__ void queue_append(uint32_t *q, uint32_t *len, uint32_t v)
{
    cg::coalesced_group g = cg::coalesced_threads();
    uint32_t base = 0;
    if (g.thread_rank() == 0) base = atomicAdd(len, g.size());
    base = g.shfl(base, 0);
    q[base + g.thread_rank()] = v;
}

// Side outputs: next frontier queue + frontier degree statistics.
template<bool SIDE>
struct Side {
    unsigned long long fe = 0;
    unsigned long long ls = 0, lq = 0;     // fixed point (lsum_fx, lsq_fx)
    float lm = 0.f;
    __device__ __forceinline__ void visit(const BfsArgs &a, uint32_t *qnext, LevelSlot *s, uint32_t v)
    {
        if constexpr (SIDE) {
            if (qnext) queue_append(qnext, &s->qlen, v);   // null: statistics only
            const uint32_t d = a.outdeg[v];
            const float l = __log2f(1.0f + static_cast<float>(d));
            fe += d; ls += lsum_fx(l); lq += lsq_fx(l); lm = fmaxf(lm, l);
        }
    }
    __device__ __forceinline__ void finish(LevelSlot *s)
    {
        if constexpr (SIDE) {
            for (int o = 16; o > 0; o >>= 1) {
                fe += __shfl_xor_sync(FULL_MASK, fe, o);
                ls += __shfl_xor_sync(FULL_MASK, ls, o);
                lq += __shfl_xor_sync(FULL_MASK, lq, o);
                lm = fmaxf(lm, __shfl_xor_sync(FULL_MASK, lm, o));
            }
            if ((threadIdx.x & 31) == 0 && fe) {
                atomicAdd(&s->fedges, fe);
                atomicAdd(&s->lsum, ls);
                atomicAdd(&s->lsq, lq);
                atomicMax(&s->lmax_bits, __float_as_uint(lm));
            }
        }
    }
    // The same, one set of atomics per block (every thread of the block
    // calls): the level's slot is one address per counter, and per-warp
    // atomics from every warp of a large level serialise there.
    __device__ __forceinline__ void finish_block(LevelSlot *s)
    {
        if constexpr (SIDE) {
            __shared__ unsigned long long b_fe[32];
            __shared__ unsigned long long b_ls[32], b_lq[32];
            __shared__ float b_lm[32];
            const unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
            for (int o = 16; o > 0; o >>= 1) {
                fe += __shfl_xor_sync(FULL_MASK, fe, o);
                ls += __shfl_xor_sync(FULL_MASK, ls, o);
                lq += __shfl_xor_sync(FULL_MASK, lq, o);
                lm = fmaxf(lm, __shfl_xor_sync(FULL_MASK, lm, o));
            }
            if (lane == 0) { b_fe[wid] = fe; b_ls[wid] = ls; b_lq[wid] = lq; b_lm[wid] = lm; }
            __syncthreads();
            if (wid == 0) {
                const bool in = lane < (blockDim.x >> 5);
                fe = in ? b_fe[lane] : 0ull; ls = in ? b_ls[lane] : 0ull; lq = in ? b_lq[lane] : 0ull;
                lm = in ? b_lm[lane] : 0.f;
                for (int o = 16; o > 0; o >>= 1) {
                    fe += __shfl_xor_sync(FULL_MASK, fe, o);
                    ls += __shfl_xor_sync(FULL_MASK, ls, o);
                    lq += __shfl_xor_sync(FULL_MASK, lq, o);
                    lm = fmaxf(lm, __shfl_xor_sync(FULL_MASK, lm, o));
                }
                if (lane == 0 && fe) {
                    atomicAdd(&s->fedges, fe);
                    atomicAdd(&s->lsum, ls);
                    atomicAdd(&s->lsq, lq);
                    atomicMax(&s->lmax_bits, __float_as_uint(lm));
                }
            }
        }
    }
};

// Next-queue appends staged per warp in shared memory: the whole warp calls
// add() at a convergent point; a full stage goes to the queue with one
// global atomic and coalesced stores.  One counter address takes every
// append of a level, so a large level otherwise serialises on it.
constexpr uint32_t WARP_STAGE = 256;
struct WarpQueue {
    uint32_t *stage;      // this warp's WARP_STAGE entries of shared memory
    uint32_t n = 0;       // staged (warp-uniform)
    __device__ __forceinline__ void add(bool hit, uint32_t v, uint32_t *q, uint32_t *len)
    {
        const unsigned lane = threadIdx.x & 31;
        const unsigned m = __ballot_sync(FULL_MASK, hit);
        if (hit) stage[n + __popc(m & ((1u << lane) - 1u))] = v;
        n += __popc(m);
        if (n > WARP_STAGE - 32) flush(q, len);
    }
    __device__ __forceinline__ void flush(uint32_t *q, uint32_t *len)
    {
        __syncwarp();
        uint32_t base = 0;
        if ((threadIdx.x & 31) == 0 && n) base = atomicAdd(len, n);
        base = __shfl_sync(FULL_MASK, base, 0);
        for (uint32_t i = threadIdx.x & 31; i < n; i += 32) q[base + i] = stage[i];
        n = 0;
        __syncwarp();
    }
};

// Hint that the 128-byte line holding p will be read soon (L2 only).
// Callers pass addresses inside their arrays.
__device__ __forceinline__ void prefetch_l2(const void *p)
{
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// Relax v to nd; true for exactly one caller per newly visited vertex.
// The plain pre-check only filters: a stale read can only be INF or nd.
__device__ __forceinline__ bool relax(int32_t *levels, uint32_t v, int32_t nd)
{
    return levels[v] > nd && atomicMin(&levels[v], nd) > nd;
}

// Warp-reduce an out-edge count into slot->fedges (every lane must call).
__device__ __forceinline__ void flush_edges(LevelSlot *s, unsigned long long fe)
{
    for (int o = 16; o > 0; o >>= 1) fe += __shfl_xor_sync(FULL_MASK, fe, o);
    if ((threadIdx.x & 31) == 0 && fe) atomicAdd(&s->fedges, fe);
}

__device__ __forceinline__ uint64_t gtid()
{ return blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; }
__device__ __forceinline__ uint64_t gthreads()
{ return uint64_t(gridDim.x) * blockDim.x; }

// Relaxes up to U neighbours (NO_VERTEX: none): their depths are all in
// flight before the first relaxation, the relaxations' atomics before the
// first result, and only a neighbour not yet visited costs an atomic.
constexpr uint32_t NO_VERTEX = 0xffffffffu;
template<int U>
__device__ __forceinline__ void claim_all(int32_t *lv, int32_t nd, const uint32_t (&u)[U], bool (&won)[U])
{
    int32_t d[U];
#pragma unroll
    for (int j = 0; j < U; j++) d[j] = u[j] != NO_VERTEX ? lv[u[j]] : nd;
#pragma unroll
    for (int j = 0; j < U; j++) d[j] = d[j] > nd ? atomicMin(&lv[u[j]], nd) : nd;
#pragma unroll
    for (int j = 0; j < U; j++) won[j] = d[j] > nd;
}
template<int U, class Visit>
__device__ __forceinline__ void relax_all(int32_t *lv, int32_t nd, const uint32_t (&u)[U], Visit visit)
{
    bool won[U];
    claim_all(lv, nd, u, won);
#pragma unroll
    for (int j = 0; j < U; j++)
        if (won[j]) visit(u[j]);
}

// ---------------------------------------------------------------------------
// Edge-list families (bfs/edgelist.cu:3-22, rev_edgelist.cu:3-21,
// struct_edgelist.cu:3-22, rev_struct_edgelist.cu:3-22).  Every level
// streams all M edges; edges are read 4 per thread with 16-byte streaming
// loads (evict-first, so the depth array keeps L2).  The reverse families
// test the sequential destination first, which skips the random source
// gather for already-visited destinations.
// ---------------------------------------------------------------------------
template<int RED, bool SIDE, int LAYOUT>
__global__ void __launch_bounds__(512) k_bfs_edge(BfsArgs a)
{
    chain_wait();
    const int32_t depth = level_depth(a), nd = depth + 1;
    LevelSlot *slot = &a.ctl->slot[depth % 3];
    if (blockIdx.x == 0 && threadIdx.x == 0) reset_slot(&a.ctl->slot[(depth + 1) % 3]);
    uint32_t *qnext = (depth & 1) ? a.q0 : a.q1;
    int32_t *lv = a.levels;
    Counter<RED> cnt;
    Side<SIDE> side;

    auto edge = [&](uint32_t row, uint32_t col) {
        // FWD: row = source, col = destination.  REV: row = destination,
        // col = source.
        if constexpr (LAYOUT == FWD_SOA || LAYOUT == FWD_AOS) {
            if (lv[row] == depth && relax(lv, col, nd)) { cnt.hit(&slot->frontier); side.visit(a, qnext, slot, col); }
        } else {
            if (lv[row] > nd && lv[col] == depth && atomicMin(&lv[row], nd) > nd) {
                cnt.hit(&slot->frontier);
                side.visit(a, qnext, slot, row);
            }
        }
    };

    // Four edges.  Forward: their depths in flight together (ER(1M, 8M)
    // edge-list 320 -> 286 us a traversal, R-MAT-16 struct-edge-list 113 -> 105);
    // the reverse lists, whose quads are mostly one row, lose by it (BA(8.4M, 8)
    // 4.25 -> 4.47 ms).
    auto edges = [&](const uint4 &r, const uint4 &c) {
        if constexpr (LAYOUT == FWD_SOA || LAYOUT == FWD_AOS) {
            const uint32_t row[4] = {r.x, r.y, r.z, r.w}, col[4] = {c.x, c.y, c.z, c.w};
            bool want[4];
            uint32_t u[4];
#pragma unroll
            for (int k = 0; k < 4; k++) want[k] = lv[row[k]] == depth;
#pragma unroll
            for (int k = 0; k < 4; k++) u[k] = want[k] ? col[k] : NO_VERTEX;
            relax_all(lv, nd, u, [&](uint32_t w) { cnt.hit(&slot->frontier); side.visit(a, qnext, slot, w); });
        } else {
            edge(r.x, c.x); edge(r.y, c.y); edge(r.z, c.z); edge(r.w, c.w);
        }
    };

    const uint64_t m = a.m;
    bool aligned;
    if constexpr (LAYOUT == FWD_SOA) aligned = !((reinterpret_cast<uintptr_t>(a.fwd_in) | reinterpret_cast<uintptr_t>(a.fwd_e)) & 15);
    else if constexpr (LAYOUT == REV_SOA) aligned = !((reinterpret_cast<uintptr_t>(a.rev_in) | reinterpret_cast<uintptr_t>(a.rev_e)) & 15);
    else if constexpr (LAYOUT == FWD_AOS) aligned = !(reinterpret_cast<uintptr_t>(a.fwd_s) & 15);
    else aligned = !(reinterpret_cast<uintptr_t>(a.rev_s) & 15);
    const uint64_t groups = aligned ? m >> 2 : 0;
    const uint64_t stride = gthreads();
    for (uint64_t g = gtid(); g < groups; g += stride) {
        if constexpr (LAYOUT == FWD_SOA || LAYOUT == REV_SOA) {
            const uint32_t *rows = LAYOUT == FWD_SOA ? a.fwd_in : a.rev_in;
            const uint32_t *cols = LAYOUT == FWD_SOA ? a.fwd_e : a.rev_e;
            const uint4 r = __ldcs(reinterpret_cast<const uint4 *>(rows) + g);
            const uint4 c = __ldcs(reinterpret_cast<const uint4 *>(cols) + g);
            edges(r, c);
        } else {
            const uint2 *pairs = LAYOUT == FWD_AOS ? a.fwd_s : a.rev_s;
            const uint4 p0 = __ldcs(reinterpret_cast<const uint4 *>(pairs) + 2 * g);
            const uint4 p1 = __ldcs(reinterpret_cast<const uint4 *>(pairs) + 2 * g + 1);
            edges(make_uint4(p0.x, p0.z, p1.x, p1.z), make_uint4(p0.y, p0.w, p1.y, p1.w));
        }
    }
    for (uint64_t e = (groups << 2) + gtid(); e < m; e += stride) {
        if constexpr (LAYOUT == FWD_SOA) edge(a.fwd_in[e], a.fwd_e[e]);
        else if constexpr (LAYOUT == REV_SOA) edge(a.rev_in[e], a.rev_e[e]);
        else if constexpr (LAYOUT == FWD_AOS) edge(a.fwd_s[e].x, a.fwd_s[e].y);
        else edge(a.rev_s[e].x, a.rev_s[e].y);
    }
    cnt.finish(&slot->frontier);
    side.finish_block(slot);
}

// edge-list over chunks of EDGE_CHUNK edges, for lists that L2 does not hold.
// k_edge_ranges reads the sources once per traversal and writes each chunk's
// least and largest one.  A level looks at the depths between them first
// (k_edge_active) and reads the edges of those chunks only where a source of
// this level is (k_bfs_edge_chunks), shared by all warps, as a hub's edges
// may be the level.  In a list sorted by source a chunk's range is a few
// dozen depths; chunks with a range too wide for that are read as before.
// (The reverse lists have work in nearly every chunk until their last levels.)
// GB300, BA(8.4M, 8), 134M edges, a traversal from a hub: 1289 us with every
// level streamed whole, 1029 by chunk (a quiet level 171 -> 25 us, the ranges
// 80; the two large levels are 60M gathers each).  R-MAT-22 with no launch
// shape asked for 696 -> 687, a root without edges there 94 -> 91.
constexpr uint32_t ACTIVE_BATCH = 4;                // chunks a warp looks at, 128 depths each in flight

static __global__ void __launch_bounds__(256) k_edge_active(BfsArgs a)
{
    chain_wait();
    constexpr uint32_t RANGE = 2 * EDGE_CHUNK;
    __shared__ uint32_t s_count[8], s_base;
    const int32_t depth = level_depth(a);
    LevelSlot *slot = &a.ctl->slot[depth % 3];
    const int32_t *lv = a.levels;
    const uint32_t lane = threadIdx.x & 31, wib = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const uint64_t chunks = (a.m + EDGE_CHUNK - 1) / EDGE_CHUNK, step = uint64_t(gridDim.x) * warps * ACTIVE_BATCH;
    for (uint64_t b0 = uint64_t(blockIdx.x) * warps * ACTIVE_BATCH; b0 < chunks; b0 += step) {
        const uint64_t first = b0 + wib * ACTIVE_BATCH;
        const uint2 mine = lane < ACTIVE_BATCH && first + lane < chunks ? a.ranges[first + lane] : make_uint2(1u, 0u);
        bool hit[ACTIVE_BATCH];
#pragma unroll
        for (uint32_t j = 0; j < ACTIVE_BATCH; j++) {
            const uint32_t lo = __shfl_sync(FULL_MASK, mine.x, j), hi = __shfl_sync(FULL_MASK, mine.y, j);
            const uint64_t v = uint64_t(lo) + lane;
            const int32_t d0 = v <= hi ? lv[v] : -1, d1 = v + 32 <= hi ? lv[v + 32] : -1;
            const int32_t d2 = v + 64 <= hi ? lv[v + 64] : -1, d3 = v + 96 <= hi ? lv[v + 96] : -1;
            hit[j] = d0 == depth || d1 == depth || d2 == depth || d3 == depth;
        }
        unsigned found = 0;
#pragma unroll
        for (uint32_t j = 0; j < ACTIVE_BATCH; j++) {
            const uint32_t lo = __shfl_sync(FULL_MASK, mine.x, j), hi = __shfl_sync(FULL_MASK, mine.y, j);
            bool any = __any_sync(FULL_MASK, hit[j]) || (hi > lo && hi - lo >= RANGE);
            for (uint64_t v = uint64_t(lo) + 128 + lane; !any && v - lane <= hi; v += 256) {
                int32_t d[8];
#pragma unroll
                for (uint32_t k = 0; k < 8; k++) d[k] = v + 32 * k <= hi ? lv[v + 32 * k] : -1;
                bool here = false;
#pragma unroll
                for (uint32_t k = 0; k < 8; k++) here = here || d[k] == depth;
                any = __any_sync(FULL_MASK, here);
            }
            if (any) found |= 1u << j;
        }
        // append, one atomic per block
        if (lane == 0) s_count[wib] = __popc(found);
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t total = 0;
            for (uint32_t w = 0; w < warps; w++) {
                const uint32_t c = s_count[w];
                s_count[w] = total;
                total += c;
            }
            s_base = total ? atomicAdd(&slot->heavy, total) : 0u;
        }
        __syncthreads();
        if (found >> lane & 1)
            a.active[s_base + s_count[wib] + __popc(found & ((1u << lane) - 1))] = static_cast<uint32_t>(first + lane);
        __syncthreads();
    }
}

template<int RED, bool SIDE>
__global__ void __launch_bounds__(256, SIDE ? 4 : 5) k_bfs_edge_chunks(BfsArgs a)
{
    chain_wait();
    constexpr uint32_t STEPS = EDGE_CHUNK / 128;
    const int32_t depth = level_depth(a), nd = depth + 1;
    LevelSlot *slot = &a.ctl->slot[depth % 3];
    if (blockIdx.x == 0 && threadIdx.x == 0) reset_slot(&a.ctl->slot[(depth + 1) % 3]);
    uint32_t *qnext = (depth & 1) ? a.q0 : a.q1;
    int32_t *lv = a.levels;
    Counter<RED> cnt;
    Side<SIDE> side;
    const uint32_t lane = threadIdx.x & 31;
    auto edge = [&](uint32_t row, uint32_t col) {
        if (lv[row] == depth && relax(lv, col, nd)) { cnt.hit(&slot->frontier); side.visit(a, qnext, slot, col); }
    };
    const uint64_t m = a.m, steps = uint64_t(slot->heavy) * STEPS, warps = gthreads() >> 5;
    for (uint64_t t0 = (gtid() >> 5) * 2; t0 < steps; t0 += warps * 2) {      // (STEPS is even)
        const uint64_t e = uint64_t(__ldca(a.active + t0 / STEPS)) * EDGE_CHUNK + (t0 % STEPS) * 128 + 4 * lane;
        if (e + 128 + 4 <= m) {
            const uint4 r0 = __ldcs(reinterpret_cast<const uint4 *>(a.fwd_in + e)), r1 = __ldcs(reinterpret_cast<const uint4 *>(a.fwd_in + e + 128));
            const uint4 q0 = __ldcs(reinterpret_cast<const uint4 *>(a.fwd_e + e)), q1 = __ldcs(reinterpret_cast<const uint4 *>(a.fwd_e + e + 128));
            const uint32_t row[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w}, col[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
            uint32_t u[8];
#pragma unroll
            for (int k = 0; k < 8; k++) u[k] = lv[row[k]] == depth ? col[k] : NO_VERTEX;
            relax_all(lv, nd, u, [&](uint32_t w) { cnt.hit(&slot->frontier); side.visit(a, qnext, slot, w); });
        } else {
            for (uint64_t i = e; i < m && i < e + 4; i++) edge(a.fwd_in[i], a.fwd_e[i]);
            for (uint64_t i = e + 128; i < m && i < e + 132; i++) edge(a.fwd_in[i], a.fwd_e[i]);
        }
    }
    cnt.finish(&slot->frontier);
    side.finish_block(slot);
}

// A warp per chunk, the chunk's 4 KB in flight; `in` is 16-byte aligned.
static __global__ void __launch_bounds__(256) k_edge_ranges(const uint32_t *__restrict__ in, uint64_t m,
                                                            uint2 *__restrict__ ranges)
{
    constexpr uint32_t STEPS = EDGE_CHUNK / 128;
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t chunks = (m + EDGE_CHUNK - 1) / EDGE_CHUNK;
    for (uint64_t c = gtid() >> 5; c < chunks; c += gthreads() >> 5) {
        uint32_t least = 0xffffffffu, most = 0u;
        auto take = [&](uint32_t r) { least = min(least, r); most = max(most, r); };
        const uint64_t e0 = c * EDGE_CHUNK + 4 * lane;
        if (c * EDGE_CHUNK + EDGE_CHUNK <= m) {
            uint4 r[STEPS];
#pragma unroll
            for (uint32_t k = 0; k < STEPS; k++) r[k] = __ldcs(reinterpret_cast<const uint4 *>(in + e0 + k * 128));
#pragma unroll
            for (uint32_t k = 0; k < STEPS; k++) { take(r[k].x); take(r[k].y); take(r[k].z); take(r[k].w); }
        } else {
            for (uint64_t e = c * EDGE_CHUNK + lane; e < m; e += 32) take(in[e]);
        }
        least = __reduce_min_sync(FULL_MASK, least);
        most = __reduce_max_sync(FULL_MASK, most);
        if (lane == 0) ranges[c] = make_uint2(least, most);
    }
}

// ---------------------------------------------------------------------------
// vertex-push (bfs/vertex_push.cu:3-26): thread per vertex; a frontier
// vertex's owner walks its CSR row.  Depths are scanned 4 per thread.  The
// rows of a warp's frontier vertices are expanded as one concatenation, an
// edge per lane, BFS_PUSH_UNROLL in flight: neighbours in id are hubs
// together on R-MAT, and one row after the other a warp's chain of
// relaxations holds the level.  A whole traversal on GB300 (host loop, rows
// one by one before): R-MAT-16 371 -> 157 us, R-MAT-22 symmetrised 1719 ->
// 1127, BA(2M, 8) 1778 -> 785.
// ---------------------------------------------------------------------------
constexpr int BFS_PUSH_UNROLL = 8;
// Rows above BFS_PUSH_GIANT edges are cut into HUB_CHUNK chunks for
// k_bfs_hub_chunks (the level's second kernel), as frontier-push does: one
// warp expanding a hub of R-MAT's lowest ids would hold the level.
constexpr uint32_t BFS_PUSH_GIANT = 256;

__device__ __forceinline__ void queue_hub_chunks(const BfsArgs &a, LevelSlot *slot, uint32_t v, uint32_t s,
                                                 uint32_t e)
{
    const uint32_t chunks = (e - s + HUB_CHUNK - 1) / HUB_CHUNK;
    const uint32_t base = atomicAdd(&slot->heavy, chunks);
    for (uint32_t c = 0; c < chunks; c++) a.heavy[base + c] = make_uint2(v, s + c * HUB_CHUNK);
}

// The row that edge k of a warp's concatenated rows belongs to: the last lane
// whose exclusive prefix is <= k (that lane's row is not empty).  Every lane
// calls.
__device__ __forceinline__ uint32_t concat_row(uint32_t excl, uint32_t k)
{
    uint32_t l = 0;
#pragma unroll
    for (uint32_t b = 16; b > 0; b >>= 1)
        if (__shfl_sync(FULL_MASK, excl, l + b) <= k) l += b;
    return l;
}

// Relaxes the neighbours E[first + k * step] (k < BFS_PUSH_UNROLL, below
// `end`): their indices, then their depths, are all in flight before the
// relaxations, and only a neighbour not yet visited costs an atomic.
template<int RED, bool SIDE>
__device__ __forceinline__ void relax_neighbours(const BfsArgs &a, const uint32_t *E, int32_t *lv, int32_t nd,
                                                 uint32_t first, uint32_t step, uint32_t end, Counter<RED> &cnt,
                                                 Side<SIDE> &side, uint32_t *qnext, LevelSlot *slot)
{
    uint32_t u[BFS_PUSH_UNROLL];
#pragma unroll
    for (int k = 0; k < BFS_PUSH_UNROLL; k++) {
        const uint32_t i = first + k * step;
        u[k] = i < end ? __ldg(E + i) : NO_VERTEX;
    }
    relax_all(lv, nd, u, [&](uint32_t w) { cnt.hit(&slot->frontier); side.visit(a, qnext, slot, w); });
}

template<int RED, bool SIDE>
__global__ void __launch_bounds__(512) k_bfs_vertex_push(BfsArgs a)
{
    chain_wait();
    const int32_t depth = level_depth(a), nd = depth + 1;
    LevelSlot *slot = &a.ctl->slot[depth % 3];
    if (blockIdx.x == 0 && threadIdx.x == 0) reset_slot(&a.ctl->slot[(depth + 1) % 3]);
    uint32_t *qnext = (depth & 1) ? a.q0 : a.q1;
    int32_t *lv = a.levels;
    Counter<RED> cnt;
    Side<SIDE> side;
    const unsigned lane = threadIdx.x & 31;
    const uint64_t n = a.n, stride = gthreads();
    // every lane calls it; rows [s, e) of frontier vertices, empty for the others
    auto expand = [&](uint32_t v, uint32_t s, uint32_t e) {
        if (e - s > BFS_PUSH_GIANT) {
            queue_hub_chunks(a, slot, v, s, e);
            e = s;
        }
        if (!__any_sync(FULL_MASK, e > s)) return;
        uint32_t incl = e - s;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL_MASK, incl, o);
            if (lane >= static_cast<unsigned>(o)) incl += y;
        }
        const uint32_t total = __shfl_sync(FULL_MASK, incl, 31), excl = incl - (e - s), from = s - excl;
        for (uint32_t k0 = 0; k0 < total; k0 += 32 * BFS_PUSH_UNROLL) {
            uint32_t u[BFS_PUSH_UNROLL];
#pragma unroll
            for (int j = 0; j < BFS_PUSH_UNROLL; j++) {
                const uint32_t k = k0 + j * 32 + lane, row = concat_row(excl, k);
                const uint32_t at = __shfl_sync(FULL_MASK, from, row) + k;
                u[j] = k < total ? __ldg(a.fwd_e + at) : NO_VERTEX;
            }
            relax_all(lv, nd, u, [&](uint32_t w) { cnt.hit(&slot->frontier); side.visit(a, qnext, slot, w); });
        }
    };
    const uint64_t groups = (reinterpret_cast<uintptr_t>(lv) & 15) ? 0 : n >> 2;
    for (uint64_t g0 = gtid() - lane; g0 < groups; g0 += stride) {
        const uint64_t g = g0 + lane;
        int4 l = make_int4(-1, -1, -1, -1);
        if (g < groups) l = reinterpret_cast<const int4 *>(lv)[g];
        const int32_t d4[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            uint32_t s = 0, e = 0;
            if (d4[k] == depth) {
                s = a.fwd_v[4 * g + k];
                e = a.fwd_v[4 * g + k + 1];
            }
            expand(static_cast<uint32_t>(4 * g + k), s, e);
        }
    }
    for (uint64_t v0 = (groups << 2) + gtid() - lane; v0 < n; v0 += stride) {
        const uint64_t v = v0 + lane;
        uint32_t s = 0, e = 0;
        if (v < n && lv[v] == depth) {
            s = a.fwd_v[v];
            e = a.fwd_v[v + 1];
        }
        expand(static_cast<uint32_t>(v), s, e);
    }
    cnt.finish(&slot->frontier);
    side.finish_block(slot);
}

// ---------------------------------------------------------------------------
// vertex-pull (bfs/vertex_pull.cu:3-31): thread per vertex; an unvisited
// vertex scans its reverse row and stops at the first parent at `depth`.
// The row is scanned BFS_PULL_UNROLL edges at a time: their indices, then
// their depths, are in flight together (a chain of dependent loads per
// edge would otherwise bound the thread); the few loads past the first
// parent are the price of the early exit.
// ---------------------------------------------------------------------------
constexpr int BFS_PULL_UNROLL = 4;

template<int RED, bool SIDE>
__global__ void __launch_bounds__(512) k_bfs_vertex_pull(BfsArgs a)
{
    chain_wait();
    const int32_t depth = level_depth(a), nd = depth + 1;
    LevelSlot *slot = &a.ctl->slot[depth % 3];
    if (blockIdx.x == 0 && threadIdx.x == 0) reset_slot(&a.ctl->slot[(depth + 1) % 3]);
    uint32_t *qnext = (depth & 1) ? a.q0 : a.q1;
    int32_t *lv = a.levels;
    Counter<RED> cnt;
    Side<SIDE> side;
    __shared__ uint32_t s_stage[SIDE ? 16 : 1][SIDE ? WARP_STAGE : 1];
    WarpQueue wq;
    wq.stage = s_stage[SIDE ? (threadIdx.x >> 5) : 0];
    const unsigned lane = threadIdx.x & 31;
    const uint64_t n = a.n, stride = gthreads();
    // whole-warp steps (the next queue is staged with one ballot per step)
    for (uint64_t v0 = gtid() - lane; v0 < n; v0 += stride) {
        const uint64_t v = v0 + lane;
        bool found = false;
        if (v < n && lv[v] > nd) {
            const uint32_t s = a.rev_v[v], e = a.rev_v[v + 1];
            for (uint32_t i = s; i < e && !found; i += BFS_PULL_UNROLL) {
                uint32_t p[BFS_PULL_UNROLL];
#pragma unroll
                for (int k = 0; k < BFS_PULL_UNROLL; k++) p[k] = i + k < e ? __ldg(a.rev_e + i + k) : 0u;
#pragma unroll
                for (int k = 0; k < BFS_PULL_UNROLL; k++) found |= i + k < e && lv[p[k]] == depth;
            }
            if (found) {
                lv[v] = nd;
                cnt.hit(&slot->frontier);
                side.visit(a, nullptr, slot, static_cast<uint32_t>(v));   // statistics; the queue below
            }
        }
        if constexpr (SIDE) if (qnext) wq.add(found, static_cast<uint32_t>(v), qnext, &slot->qlen);
    }
    if constexpr (SIDE) if (qnext) wq.flush(qnext, &slot->qlen);
    cnt.finish(&slot->frontier);
    side.finish_block(slot);
}

// vertex-pull while the frontier is small and most vertices are open: nearly
// every open vertex then looks at its whole in-row in vain, an L1TEX tag for
// each index and one for each depth.  The frontier's bits (k_bfs_filter; folded
// to FILTER_BITS where the graph has more vertices) go to every block's shared
// memory, and a warp streams the in-rows of 32 neighbouring vertices (a
// window), one contiguous range, 32 edges a load: an edge costs a bit test, and
// only those whose bit is set look for their row and at the depth.  Windows of
// more than FILTER_PIECE edges (R-MAT's hubs are neighbours in id) are cut into
// pieces of so many, listed by k_bfs_filter: as one task of one warp such a
// window held the level, R-MAT-20 symmetrised from its hub 2020 us.
static __global__ void __launch_bounds__(256) k_bfs_filter(BfsArgs a)
{
    const unsigned lane = threadIdx.x & 31;
    const uint64_t words = (uint64_t(a.filter_mask) + 1) / 32, n = a.n, windows = (n + 31) / 32;
    auto edges_of = [&](uint64_t j) {
        return j < windows ? __ldg(a.rev_v + min(32 * j + 32, n)) - __ldg(a.rev_v + 32 * j) : 0u;
    };
    uint32_t total = edges_of(gtid());                 // before the wait: the graph is older than the run
    chain_wait();
    const int32_t depth = level_depth(a);
    const int32_t *lv = a.levels;
    // the heavy windows' pieces
    for (uint64_t j0 = gtid() - lane; j0 < windows; j0 += gthreads(), total = edges_of(j0 + lane)) {
        for (unsigned heavy = __ballot_sync(FULL_MASK, total > FILTER_PIECE); heavy; heavy &= heavy - 1) {
            const int l = __ffs(heavy) - 1;
            const uint32_t count = __shfl_sync(FULL_MASK, (total - 1) / FILTER_PIECE + 1, l);
            uint32_t at = 0;
            if (lane == 0) at = atomicAdd(&a.ctl->slot[depth % 3].heavy, count);
            at = __shfl_sync(FULL_MASK, at, 0);
            for (uint32_t c = lane; c < count; c += 32)
                a.pieces[at + c] = make_uint2(static_cast<uint32_t>(j0) + l, c * FILTER_PIECE);
        }
    }
    for (uint64_t w = gtid() >> 5; w < words; w += gthreads() >> 5) {
        uint32_t bits = 0;
#pragma unroll 4
        for (uint64_t v0 = w * 32; v0 < n; v0 += uint64_t(a.filter_mask) + 1) {
            const uint64_t v = v0 + lane;
            bits |= __ballot_sync(FULL_MASK, v < n && lv[v] == depth);
        }
        if (lane == 0) a.filter[w] = bits;
    }
}

constexpr int FILTER_UNROLL = 8;

template<int RED, bool SIDE>
__global__ void __launch_bounds__(1024, 1) k_bfs_pull_filter(BfsArgs a)
{
    extern __shared__ __align__(16) uint32_t s_filter[];
    chain_wait();
    const int32_t depth = level_depth(a), nd = depth + 1;
    LevelSlot *slot = &a.ctl->slot[depth % 3];
    if (blockIdx.x == 0 && threadIdx.x == 0) reset_slot(&a.ctl->slot[(depth + 1) % 3]);
    uint32_t *qnext = (depth & 1) ? a.q0 : a.q1;
    int32_t *lv = a.levels;
    Counter<RED> cnt;
    Side<SIDE> side;
    const unsigned lane = threadIdx.x & 31;
    const uint64_t n = a.n, windows = (n + 31) / 32, tasks = windows + slot->heavy, warps = gthreads() >> 5;
    // the windows, then the pieces of the heavy ones; the next task's rows'
    // bounds and depths are loaded one task ahead
    uint32_t next_off = 0, next_end = 0, next_k0 = 0, next_v0 = 0;
    int32_t next_depth = 0;
    auto fetch = [&](uint64_t t) {
        if (t >= tasks) return;
        uint64_t w = t;
        if (t >= windows) {
            const uint2 piece = a.pieces[t - windows];
            w = piece.x;
            next_k0 = piece.y;
        }
        const uint64_t v = 32 * w + lane;
        next_v0 = static_cast<uint32_t>(32 * w);
        next_off = __ldg(a.rev_v + min(v, n));
        next_end = __ldg(a.rev_v + min(32 * w + 32, n));
        next_depth = v < n ? lv[v] : 0;
    };
    fetch(gtid() >> 5);
    const uint32_t mask = a.filter_mask, quads = (mask + 1) / 128;
    for (uint32_t i = threadIdx.x; i < quads; i += blockDim.x)
        reinterpret_cast<uint4 *>(s_filter)[i] = __ldcg(reinterpret_cast<const uint4 *>(a.filter) + i);
    __syncthreads();
    // up to FILTER_UNROLL in-edges a lane: in-neighbour p of the row that
    // row_of gives for load u (every lane calls it, where some lane has a hit)
    auto test = [&](const uint32_t (&p)[FILTER_UNROLL], auto row_of) {
        bool hit[FILTER_UNROLL];
        bool any = false;
#pragma unroll
        for (int u = 0; u < FILTER_UNROLL; u++) {
            hit[u] = p[u] != NO_VERTEX && (s_filter[(p[u] & mask) >> 5] >> (p[u] & 31) & 1u);
            any = any || hit[u];
        }
        if (!__any_sync(FULL_MASK, any)) return;
        int32_t d[FILTER_UNROLL];
#pragma unroll
        for (int u = 0; u < FILTER_UNROLL; u++) d[u] = hit[u] ? lv[p[u]] : nd;
#pragma unroll
        for (int u = 0; u < FILTER_UNROLL; u++) {
            if (!__any_sync(FULL_MASK, d[u] == depth)) continue;
            const uint32_t w = row_of(u);
            if (d[u] == depth && lv[w] > nd && atomicMin(&lv[w], nd) > nd) {
                cnt.hit(&slot->frontier);
                side.visit(a, qnext, slot, w);
            }
        }
    };
    for (uint64_t t = gtid() >> 5; t < tasks; t += warps) {
        const uint32_t off = next_off, end = next_end, v0 = next_v0, k0 = next_k0;
        const bool open = next_depth > nd;
        fetch(t + warps);
        const uint32_t base = __shfl_sync(FULL_MASK, off, 0), excl = off - base, total = end - base;
        if (t < windows && total > FILTER_PIECE) continue;
        const uint32_t k1 = k0 + min(total - k0, FILTER_PIECE);
        const uint32_t below = __shfl_down_sync(FULL_MASK, off, 1);
        const uint32_t s = max(off, base + k0), e = min(lane == 31 ? end : below, base + k1);
        const uint32_t len = open && e > s ? e - s : 0u, wanted = __reduce_add_sync(FULL_MASK, len);
        if (wanted == 0) continue;
        if (wanted >= (k1 - k0) / 2) {
            for (uint32_t b = k0; b < k1; b += 32 * FILTER_UNROLL) {
                uint32_t p[FILTER_UNROLL];
#pragma unroll
                for (int u = 0; u < FILTER_UNROLL; u++) {
                    const uint32_t k = b + u * 32 + lane;
                    p[u] = k < k1 ? __ldcs(a.rev_e + base + k) : NO_VERTEX;
                }
                test(p, [&](int u) { return v0 + concat_row(excl, b + u * 32 + lane); });
            }
        } else {
            // mostly rows already reached: the open ones' edges one after the other
            uint32_t incl = len;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(FULL_MASK, incl, o);
                if (lane >= static_cast<unsigned>(o)) incl += y;
            }
            const uint32_t before = incl - len, from = s - before;
            for (uint32_t b = 0; b < wanted; b += 32 * FILTER_UNROLL) {
                uint32_t p[FILTER_UNROLL];
#pragma unroll
                for (int u = 0; u < FILTER_UNROLL; u++) {
                    const uint32_t k = b + u * 32 + lane;
                    const uint32_t i = __shfl_sync(FULL_MASK, from, concat_row(before, k)) + k;
                    p[u] = k < wanted ? __ldcs(a.rev_e + i) : NO_VERTEX;
                }
                test(p, [&](int u) { return v0 + concat_row(before, b + u * 32 + lane); });
            }
        }
    }
    cnt.finish(&slot->frontier);
    side.finish_block(slot);
}

// ---------------------------------------------------------------------------
// Virtual-warp families (bfs/vertex_push_warp.cu:19-60,
// vertex_pull_warp.cu:17-71): a virtual warp of W lanes (W | 32) takes a
// chunk of C vertices, stages their depths and row offsets in shared memory
// ((W-lane group) x (C + C + 1) words, ImplementationTemplate.hpp:166-167)
// and expands / scans each row with its W lanes.  The pull form stops a
// row as soon as any lane has found a parent (the reference scans the
// whole row) and writes back only the depths it changed.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned subwarp_mask(uint32_t W)
{
    if (W >= 32) return FULL_MASK;
    const unsigned lane = threadIdx.x & 31;
    return ((1u << W) - 1u) << (lane & ~(W - 1u));
}

// Push, without statistics: three blocks an SM, the claims of 8 edges in 40
// registers.  Left to itself the compiler takes 56, and a quiet level, one scan
// of the depths, waits on fewer warps.  Whole traversals on GB300: R-MAT-23
// symmetrised 3152 -> 2758 us, BA(4.2M, 12) 1661 -> 1471.
template<int RED, bool SIDE, bool PULL>
__global__ void __launch_bounds__(512, SIDE ? 0 : 3) k_bfs_vwarp(BfsArgs a)
{
    chain_wait();
    extern __shared__ uint32_t smem[];
    const int32_t depth = level_depth(a), nd = depth + 1;
    LevelSlot *slot = &a.ctl->slot[depth % 3];
    if (blockIdx.x == 0 && threadIdx.x == 0) reset_slot(&a.ctl->slot[(depth + 1) % 3]);
    uint32_t *qnext = (depth & 1) ? a.q0 : a.q1;
    int32_t *lv = a.levels;
    Counter<RED> cnt;
    Side<SIDE> side;

    const uint32_t W = a.warp_size, C = a.chunk_size;
    const uint32_t per_block = blockDim.x / W;
    const uint32_t vw = threadIdx.x / W, lane = threadIdx.x % W;
    const unsigned mask = subwarp_mask(W);
    int32_t *my_lv = reinterpret_cast<int32_t *>(smem) + vw * C;
    uint32_t *my_off = smem + per_block * C + vw * (C + 1);
    const uint32_t *V = PULL ? a.rev_v : a.fwd_v;
    const uint32_t *E = PULL ? a.rev_e : a.fwd_e;
    const uint64_t n = a.n;
    const uint64_t total_vw = uint64_t(gridDim.x) * per_block;

    for (uint64_t chunk = blockIdx.x * uint64_t(per_block) + vw; chunk * C < n; chunk += total_vw) {
        const uint64_t v0 = chunk * C;
        const uint32_t cntv = static_cast<uint32_t>(min(uint64_t(C), n - v0));
        for (uint32_t i = lane; i < cntv; i += W) my_lv[i] = lv[v0 + i];
        for (uint32_t i = lane; i < cntv + 1; i += W) my_off[i] = V[v0 + i];
        __syncwarp(mask);
        for (uint32_t v = 0; v < cntv; v++) {
            const uint32_t s = my_off[v], e = my_off[v + 1];
            if constexpr (!PULL) {
                if (my_lv[v] == depth) {
                    if (e - s > BFS_PUSH_GIANT) {             // to k_bfs_hub_chunks
                        if (lane == 0) queue_hub_chunks(a, slot, static_cast<uint32_t>(v0 + v), s, e);
                    } else {
                        for (uint32_t base = s; base < e; base += W * BFS_PUSH_UNROLL)
                            relax_neighbours(a, E, lv, nd, base + lane, W, e, cnt, side, qnext, slot);
                    }
                }
            } else {
                if (my_lv[v] > depth) {
                    bool found = false;
                    for (uint32_t base = s; base < e; base += W) {
                        const uint32_t i = base + lane;
                        const bool hit = i < e && lv[__ldg(E + i)] == depth;
                        if (__any_sync(mask, hit)) { found = true; break; }
                    }
                    if (found && lane == 0) my_lv[v] = nd;
                }
            }
        }
        __syncwarp(mask);
        if constexpr (PULL) {
            for (uint32_t i = lane; i < cntv; i += W) {
                if (my_lv[i] == nd && lv[v0 + i] != nd) {
                    lv[v0 + i] = nd;
                    cnt.hit(&slot->frontier);
                    side.visit(a, qnext, slot, static_cast<uint32_t>(v0 + i));
                }
            }
            __syncwarp(mask);
        }
    }
    cnt.finish(&slot->frontier);
    side.finish_block(slot);
}

// ---------------------------------------------------------------------------
// frontier-push (GB300 variant): top-down over the frontier queue only.
// A warp takes up to 32 queue entries; their rows are concatenated (warp
// prefix sum of degrees) and the warp's lanes sweep the concatenation,
// FRONTIER_UNROLL edges in flight each, so every lane does the same amount
// of edge work and reads within a row coalesce.  A level is a chain of
// dependent accesses per step (index, depth, claim): with one edge in flight
// per lane a traversal of BA(2M, 8) took 714 us on GB300 and takes 399 with
// four, and the whole of a hub chunk in flight.
// Rows above HEAVY_DEGREE are cut into HUB_CHUNK chunks queued for
// k_bfs_hub_chunks, which spreads a hub over the whole GPU.
// Always emits the next queue.
// ---------------------------------------------------------------------------
constexpr int FRONTIER_UNROLL = 4;

template<bool SIDE>
__global__ void __launch_bounds__(256) k_bfs_frontier_push(BfsArgs a)
{
    chain_wait();
    __shared__ uint32_t s_stage[8][WARP_STAGE];
    if (a.skip_check && *((volatile uint32_t *) &a.ctl->skip)) return;
    const int32_t depth = level_depth(a), nd = depth + 1;
    LevelSlot *slot = &a.ctl->slot[depth % 3];
    if (blockIdx.x == 0 && threadIdx.x == 0) reset_slot(&a.ctl->slot[(depth + 1) % 3]);
    const uint32_t *qin = (depth & 1) ? a.q1 : a.q0;
    uint32_t *qnext = (depth & 1) ? a.q0 : a.q1;
    const uint32_t qlen = *((volatile uint32_t *) &a.ctl->slot[(depth + 2) % 3].qlen);
    int32_t *lv = a.levels;
    Counter<RED_BLOCK> cnt;
    Side<SIDE> side;
    const unsigned lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const uint64_t warp = gtid() >> 5, warps = gthreads() >> 5;
    unsigned long long fe = 0;   // next-frontier out-edges (cluster-path gating)
    WarpQueue wq;
    wq.stage = s_stage[wib];

    // a short queue is spread over the warps, down to a row each
    const uint32_t per = static_cast<uint32_t>(min(uint64_t(32), (qlen + warps - 1) / warps));
    for (uint64_t t = warp * per; t < qlen; t += warps * per) {
        const uint64_t i = t + lane;
        uint32_t v = 0, s = 0, d = 0;
        if (lane < per && i < qlen) {
            v = qin[i];
            s = a.fwd_v[v];
            d = a.fwd_v[v + 1] - s;
        }
        if (d > HEAVY_DEGREE) {
            queue_hub_chunks(a, slot, v, s, s + d);
            d = 0;
        }
        uint32_t incl = d;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL_MASK, incl, o);
            if (lane >= static_cast<unsigned>(o)) incl += y;
        }
        const uint32_t total = __shfl_sync(FULL_MASK, incl, 31), excl = incl - d, from = s - excl;
        // whole-warp steps, so that the new vertices are staged with one
        // ballot each
        for (uint32_t k0 = 0; k0 < total; k0 += 32 * FRONTIER_UNROLL) {
            uint32_t u[FRONTIER_UNROLL];
            bool won[FRONTIER_UNROLL];
#pragma unroll
            for (int j = 0; j < FRONTIER_UNROLL; j++) {
                const uint32_t k = k0 + j * 32 + lane, row = concat_row(excl, k);
                const uint32_t at = __shfl_sync(FULL_MASK, from, row) + k;
                u[j] = k < total ? __ldg(a.fwd_e + at) : NO_VERTEX;
            }
            claim_all(lv, nd, u, won);
#pragma unroll
            for (int j = 0; j < FRONTIER_UNROLL; j++) {
                if (won[j]) {
                    cnt.hit(&slot->frontier);
                    if constexpr (SIDE) side.visit(a, nullptr, nullptr, u[j]);
                    else if (a.skip_check) fe += a.outdeg[u[j]];
                }
                wq.add(won[j], u[j], qnext, &slot->qlen);
            }
        }
    }
    wq.flush(qnext, &slot->qlen);
    cnt.finish(&slot->frontier);
    side.finish_block(slot);
    if constexpr (!SIDE) flush_edges(slot, fe);
}

template<bool SIDE>
__global__ void __launch_bounds__(256) k_bfs_hub_chunks(BfsArgs a)
{
    chain_wait();
    __shared__ uint32_t s_stage[8][WARP_STAGE];
    if (a.skip_check && *((volatile uint32_t *) &a.ctl->skip)) return;
    const int32_t depth = level_depth(a), nd = depth + 1;
    LevelSlot *slot = &a.ctl->slot[depth % 3];
    uint32_t *qnext = (depth & 1) ? a.q0 : a.q1;
    const uint32_t chunks = *((volatile uint32_t *) &slot->heavy);
    int32_t *lv = a.levels;
    Counter<RED_BLOCK> cnt;
    Side<SIDE> side;
    const unsigned lane = threadIdx.x & 31;
    const uint64_t warp = gtid() >> 5, warps = gthreads() >> 5;
    unsigned long long fe = 0;
    WarpQueue wq;
    wq.stage = s_stage[threadIdx.x >> 5];
    for (uint64_t c = warp; c < chunks; c += warps) {
        const uint2 h = a.heavy[c];
        const uint32_t end = min(h.y + HUB_CHUNK, a.fwd_v[h.x + 1]);
        // the whole chunk in flight
        uint32_t u[HUB_CHUNK / 32];
        bool won[HUB_CHUNK / 32];
#pragma unroll
        for (int j = 0; j < static_cast<int>(HUB_CHUNK / 32); j++) {
            const uint32_t i = h.y + j * 32 + lane;
            u[j] = i < end ? __ldcs(a.fwd_e + i) : NO_VERTEX;
        }
        claim_all(lv, nd, u, won);
#pragma unroll
        for (int j = 0; j < static_cast<int>(HUB_CHUNK / 32); j++) {
            if (won[j]) {
                cnt.hit(&slot->frontier);
                if constexpr (SIDE) side.visit(a, nullptr, nullptr, u[j]);
                else if (a.skip_check) fe += a.outdeg[u[j]];
            }
            wq.add(won[j], u[j], qnext, &slot->qlen);
        }
    }
    wq.flush(qnext, &slot->qlen);
    cnt.finish(&slot->frontier);
    side.finish_block(slot);
    if constexpr (!SIDE) flush_edges(slot, fe);
}

// ---------------------------------------------------------------------------
// frontier-pull (GB300 variant): bottom-up.  Each lane owns one unvisited
// vertex and checks up to 8 in-neighbours on its own; vertices still
// unresolved with longer rows are then swept by the whole warp 32
// in-neighbours at a time with a ballot early exit, so skewed in-degrees
// do not serialise a lane.  Emits the next queue when SIDE.
// ---------------------------------------------------------------------------
template<bool SIDE>
__global__ void __launch_bounds__(256) k_bfs_frontier_pull(BfsArgs a)
{
    chain_wait();
    __shared__ uint32_t s_stage[8][WARP_STAGE];
    const int32_t depth = level_depth(a), nd = depth + 1;
    LevelSlot *slot = &a.ctl->slot[depth % 3];
    if (blockIdx.x == 0 && threadIdx.x == 0) reset_slot(&a.ctl->slot[(depth + 1) % 3]);
    uint32_t *qnext = (depth & 1) ? a.q0 : a.q1;
    int32_t *lv = a.levels;
    Counter<RED_BLOCK> cnt;
    Side<SIDE> side;
    const unsigned lane = threadIdx.x & 31;
    const uint64_t warp = gtid() >> 5, warps = gthreads() >> 5;
    const uint64_t n = a.n;
    constexpr uint32_t SOLO = 8;
    WarpQueue wq;
    wq.stage = s_stage[threadIdx.x >> 5];

    for (uint64_t t = warp * 32; t < n; t += warps * 32) {
        const uint64_t v = t + lane;
        bool open = v < n && lv[v] > nd;
        bool found = false;
        uint32_t s = 0, e = 0;
        if (open) {
            s = a.rev_v[v];
            e = a.rev_v[v + 1];
            const uint32_t lim = min(e, s + SOLO);
            for (uint32_t i = s; i < lim; i++) {
                if (lv[__ldg(a.rev_e + i)] == depth) { found = true; break; }
            }
            open = !found && e > lim;
            s = lim;
        }
        unsigned pending = __ballot_sync(FULL_MASK, open);
        while (pending) {
            const int owner = __ffs(pending) - 1;
            pending &= pending - 1;
            const uint32_t rs = __shfl_sync(FULL_MASK, s, owner);
            const uint32_t re = __shfl_sync(FULL_MASK, e, owner);
            bool got = false;
            for (uint32_t b = rs; b < re; b += 32) {
                const uint32_t i = b + lane;
                const bool hit = i < re && lv[__ldg(a.rev_e + i)] == depth;
                if (__any_sync(FULL_MASK, hit)) { got = true; break; }
            }
            if (lane == static_cast<unsigned>(owner)) found = got;
        }
        if (found) {
            lv[v] = nd;
            cnt.hit(&slot->frontier);
            side.visit(a, nullptr, slot, static_cast<uint32_t>(v));   // statistics; the queue below
        }
        if constexpr (SIDE) wq.add(found, static_cast<uint32_t>(v), qnext, &slot->qlen);
    }
    if constexpr (SIDE) wq.flush(qnext, &slot->qlen);
    cnt.finish(&slot->frontier);
    side.finish_block(slot);
}

// ---------------------------------------------------------------------------
// frontier-push, small-frontier path (device loop only): one cluster of
// CLUSTER_CTAS blocks keeps expanding levels while the frontier stays small
// -- the high-diameter case (2-D grids, BFS tails) where one launch per
// level would dominate.  A level is then a short chain of dependent
// accesses, so the kernel keeps all else on chip:
//  * each block holds its part of the frontier in shared memory as {row
//    start, row end}: a level reads no queue and no offsets from global
//    memory, and where no row of a warp's 32 is longer than CLUSTER_UNROLL
//    (meshes) each lane takes its own row, without the search for an edge's
//    row in the concatenation;
//  * a neighbour is claimed with one atomicMin on its depth, issued with
//    its row bounds' loads and the lane's other claims; the winner puts the
//    bounds in its block's next list;
//  * warps add their counts to their block's in shared memory, and after the
//    level's one cluster barrier every warp reads the blocks' counts for
//    itself.  Lists of up to CLUSTER_KEEP rows stay with their block; longer
//    ones are shared out equally, read from the other blocks' shared memory.
//    The next lists alternate between two buffers, the counts between three,
//    so nothing needs a second cluster barrier.
// Bound by the latency of that chain: on GB300 a level of the 2048 x 2048 grid
// took 4.5 to 5.0 us and takes 3.1 to 4.1, of a 300 x 300 grid 4.0 and 2.6.
// More threads a block than the frontier fills only make the barriers dearer
// (1024 instead of 512: 3.1 and 4.4 us), fewer leave wide frontiers behind
// (256: 2.5 us on 300 x 300, but 7.4 instead of 6.8 on 5000 x 5000); 16 blocks
// of 256 in place of 8 of 512: 3.0 and 6.2.
// Rows above CLUSTER_HEAVY edges are left to the full-GPU kernels (their
// hub chunks spread such a row over every SM): a frontier with one is not
// taken on, and a level that finds one hands over.  So do a frontier above
// the caps and a block list overflow (the overflow went to the global queue
// already): the blocks write their lists to the global queue after the
// overflow, the leader fills the level's slot as the regular kernels would
// have, sets ctl->skip so that the regular frontier-push kernels of the loop
// iteration return at once, and leaves that level's bookkeeping to the step
// kernel.  The leader does the bookkeeping of the levels it completes.
// ---------------------------------------------------------------------------
constexpr uint32_t CLUSTER_HEAVY = 1024;           // rows above: the full-GPU kernels
constexpr int CLUSTER_UNROLL = 4;
constexpr uint32_t CLUSTER_KEEP = 256;             // next lists up to this long stay with their block
// dynamic shared memory: the level's share {row start, row end} and two next
// lists {row start, row end}, {vertex}
constexpr size_t CLUSTER_SMEM = (3 * 2 + 2) * CLUSTER_LIST * sizeof(uint32_t);

// A block's counts of one level, added up by its warps; read by the others.
struct __align__(16) ClusterCounts {
    uint32_t frontier;            // new vertices found (those past CLUSTER_LIST went to the global queue)
    uint32_t fedges;              // their out-edges (each vertex once: at most M < 2^32 in all)
    uint32_t heavy;               // != 0: one of them has a row above CLUSTER_HEAVY
    uint32_t lm_bits;             // STATS == 1: largest log degree
    unsigned long long ls, lq;    // STATS == 1: log-degree sums, fixed point
};

// STATS: 0 none; 1 the log-degree statistics of every level (accumulated
// per claim, for a level log); 2 only those of a level handed over (what
// the next level's choice reads), computed from its frontier at handover.
template<int STATS>
__global__ void __cluster_dims__(CLUSTER_CTAS, 1, 1) __launch_bounds__(CLUSTER_THREADS, 1)
k_bfs_cluster(BfsArgs a)
{
    chain_wait();
    extern __shared__ __align__(16) uint32_t cl_lists[];
    __shared__ ClusterCounts s_cnt[3];             // by level
    __shared__ unsigned long long r_ls[CLUSTER_THREADS / 32], r_lq[CLUSTER_THREADS / 32];
    __shared__ float r_lm[CLUSTER_THREADS / 32];
    __shared__ unsigned long long s_hand[3];       // this block's part of a handed-over frontier's statistics
    cg::cluster_group cl = cg::this_cluster();
    BfsCtl *ctl = a.ctl;
    const unsigned rank = cl.block_rank(), tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
    const bool leader = rank == 0 && tid == 0;
    int32_t L = *((volatile int32_t *) &ctl->depth);
    const uint32_t max_levels = *((volatile uint32_t *) &ctl->max_levels);
    const uint32_t qlen = *((volatile uint32_t *) &ctl->slot[(L + 2) % 3].qlen);
    const unsigned long long fedges = *((volatile unsigned long long *) &ctl->slot[(L + 2) % 3].fedges);
    // same values in every block: a large or edge-heavy frontier is left to
    // the full-GPU kernels
    if (qlen == 0 || qlen > CLUSTER_CAP || fedges > CLUSTER_EDGE_CAP) return;
    int32_t *lv = a.levels;
    uint2 *const share = reinterpret_cast<uint2 *>(cl_lists);
    uint2 *const next_se[2] = {share + CLUSTER_LIST, share + 2 * CLUSTER_LIST};
    uint32_t *const next_v[2] = {cl_lists + 6 * CLUSTER_LIST, cl_lists + 7 * CLUSTER_LIST};
    uint32_t ncur;                                 // rows in `cur`, this block's part of the level
    const uint2 *cur = share;
    {   // this block's share of the level's queue, with the rows' bounds
        const uint32_t *qin = (L & 1) ? a.q1 : a.q0;
        const uint32_t per = (qlen + CLUSTER_CTAS - 1) / CLUSTER_CTAS;
        const uint32_t b = min(qlen, rank * per), cnt = min(per, qlen - b);   // cnt <= CLUSTER_LIST
        uint32_t heavy = 0;
        for (uint32_t i = tid; i < cnt; i += CLUSTER_THREADS) {
            const uint32_t v = __ldcg(qin + b + i);
            const uint32_t rs = a.fwd_v[v], re = a.fwd_v[v + 1];
            share[i] = make_uint2(rs, re);
            heavy |= re - rs > CLUSTER_HEAVY ? 1u : 0u;
        }
        if (tid < 3) s_cnt[tid] = ClusterCounts{};
        heavy = __syncthreads_or(heavy);
        if (tid == 0) s_cnt[(L + 2) % 3].heavy = heavy;
        ncur = cnt;
        cl.sync();
        uint32_t any = 0;
        if (tid < CLUSTER_CTAS) any = cl.map_shared_rank(&s_cnt[(L + 2) % 3], tid)->heavy;
        any = __syncthreads_or(any);
        cl.sync();                                   // nobody leaves while its flag may be read
        if (any) return;                             // a hub row: the full-GPU kernels take this level
        // (the flag is zero then, as the counts of level L + 2 begin)
    }
    unsigned long long visited = 0, traversed = 0;   // of the completed levels (the leader's)
    int p = 0;                                       // the next list being filled
    for (;;) {
        const int32_t nd = L + 1;
        LevelSlot *slot = &ctl->slot[L % 3];
        ClusterCounts *const cnt = &s_cnt[L % 3];
        uint32_t *qnext = (L & 1) ? a.q0 : a.q1;
        if (leader) reset_slot(&ctl->slot[(L + 1) % 3]);
        uint2 *const nse = next_se[p];
        uint32_t *const nv = next_v[p];
        uint32_t fe = 0, heavy = 0;
        unsigned long long ls = 0, lq = 0;
        float lm = 0.f;
        // Next-line prefetch: where vertex ids follow the graph's geometry
        // (grids, meshes, road networks) the wavefront reaches a claimed
        // vertex's id neighbours within a few levels, and the first touch of
        // their lines would put an HBM miss on a level's critical path.  Done
        // for a lane's last claims, while the cluster barrier waits (300 x 300
        // grid 2.77 -> 2.60 us a level, 20,000 x 50 2.66 -> 2.31).
        uint32_t claimed[CLUSTER_UNROLL], claimed_end[CLUSTER_UNROLL];
#pragma unroll
        for (int jj = 0; jj < CLUSTER_UNROLL; jj++) claimed[jj] = NO_VERTEX;
        auto prefetch = [&]() {
#pragma unroll
            for (int jj = 0; jj < CLUSTER_UNROLL; jj++) {
                if (claimed[jj] == NO_VERTEX) continue;
                const uint64_t v = claimed[jj], e = claimed_end[jj];
                if (e + 32 < a.m) prefetch_l2(a.fwd_e + e + 32);
                if (v + 33 <= a.n) prefetch_l2(a.fwd_v + v + 33);
                if (v + 32 < a.n) prefetch_l2(lv + v + 32);
            }
        };
        // Claims up to CLUSTER_UNROLL neighbours a lane.  A level is a chain
        // of dependent accesses, so every lane's neighbours go out together:
        // their row bounds (loaded whether or not the claim wins) and their
        // atomics are all in flight before any result is used.
        auto claim = [&](const uint32_t (&u)[CLUSTER_UNROLL]) {
            uint32_t us[CLUSTER_UNROLL], ue[CLUSTER_UNROLL];
            int32_t old[CLUSTER_UNROLL];
#pragma unroll
            for (int jj = 0; jj < CLUSTER_UNROLL; jj++)
                old[jj] = u[jj] != NO_VERTEX ? atomicMin(&lv[u[jj]], nd) : nd;
#pragma unroll
            for (int jj = 0; jj < CLUSTER_UNROLL; jj++) {
                us[jj] = ue[jj] = 0;
                if (u[jj] != NO_VERTEX) {
                    us[jj] = __ldg(a.fwd_v + u[jj]);
                    ue[jj] = __ldg(a.fwd_v + u[jj] + 1);
                }
            }
            // the winners' entries: one shared atomic per warp
            unsigned wm[CLUSTER_UNROLL];
            uint32_t total = 0;
#pragma unroll
            for (int jj = 0; jj < CLUSTER_UNROLL; jj++) {
                wm[jj] = __ballot_sync(FULL_MASK, old[jj] > nd);
                total += __popc(wm[jj]);
            }
            if (total == 0) return;
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(&cnt->frontier, total);
            base = __shfl_sync(FULL_MASK, base, 0);
            const unsigned below = (1u << lane) - 1u;
#pragma unroll
            for (int jj = 0; jj < CLUSTER_UNROLL; jj++) {
                if (old[jj] > nd) {
                    const uint32_t k = base + __popc(wm[jj] & below);
                    if (k < CLUSTER_LIST) {
                        nse[k] = make_uint2(us[jj], ue[jj]);
                        nv[k] = u[jj];
                    } else {                             // overflow: straight to the global queue
                        qnext[atomicAdd(&slot->qlen, 1u)] = u[jj];
                    }
                    fe += ue[jj] - us[jj];
                    heavy |= ue[jj] - us[jj] > CLUSTER_HEAVY ? 1u : 0u;
                    if constexpr (STATS == 1) {
                        const float l = __log2f(1.0f + static_cast<float>(ue[jj] - us[jj]));
                        ls += lsum_fx(l); lq += lsq_fx(l); lm = fmaxf(lm, l);
                    }
                    claimed[jj] = u[jj];
                    claimed_end[jj] = ue[jj];
                }
                base += __popc(wm[jj]);
            }
        };
        // 32 rows per warp step
        for (uint32_t t = wib * 32; t < ncur; t += CLUSTER_THREADS) {
            const uint32_t i = t + lane;
            const uint2 se = i < ncur ? cur[i] : make_uint2(0u, 0u);
            const uint32_t s = se.x, d = se.y - se.x;
            uint32_t u[CLUSTER_UNROLL];
            if (__reduce_max_sync(FULL_MASK, d) <= CLUSTER_UNROLL) {
                // short rows (meshes): a lane's own row
#pragma unroll
                for (uint32_t jj = 0; jj < CLUSTER_UNROLL; jj++) u[jj] = jj < d ? __ldg(a.fwd_e + s + jj) : NO_VERTEX;
                claim(u);
                continue;
            }
            // the rows concatenated
            uint32_t incl = d;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(FULL_MASK, incl, o);
                if (lane >= static_cast<unsigned>(o)) incl += y;
            }
            const uint32_t total = __shfl_sync(FULL_MASK, incl, 31), excl = incl - d, from = s - excl;
            for (uint32_t k0 = 0; k0 < total; k0 += 32 * CLUSTER_UNROLL) {
#pragma unroll
                for (int jj = 0; jj < CLUSTER_UNROLL; jj++) {
                    const uint32_t k = k0 + jj * 32 + lane, row = concat_row(excl, k);
                    const uint32_t at = __shfl_sync(FULL_MASK, from, row) + k;
                    u[jj] = k < total ? __ldg(a.fwd_e + at) : NO_VERTEX;
                }
                claim(u);
            }
        }
        // the warp's counts
        fe = __reduce_add_sync(FULL_MASK, fe);
        if (fe) {
            heavy = __any_sync(FULL_MASK, heavy);
            if (lane == 0) {
                atomicAdd(&cnt->fedges, fe);
                if (heavy) cnt->heavy = 1;
            }
        }
        if constexpr (STATS == 1) {
            for (int o = 16; o > 0; o >>= 1) {
                ls += __shfl_xor_sync(FULL_MASK, ls, o);
                lq += __shfl_xor_sync(FULL_MASK, lq, o);
                lm = fmaxf(lm, __shfl_xor_sync(FULL_MASK, lm, o));
            }
            if (lane == 0 && ls) {
                atomicAdd(&cnt->ls, ls);
                atomicAdd(&cnt->lq, lq);
                atomicMax(&cnt->lm_bits, __float_as_uint(lm));
            }
        }
        // every block's counts, list and overflow are out
        asm volatile("barrier.cluster.arrive.release;" ::: "memory");
        prefetch();
        asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
        // The cluster's totals, read by every warp for itself: lane q holds
        // block q's list length and the exclusive prefix of the lists.
        if (tid == 0) s_cnt[(L + 2) % 3] = ClusterCounts{};     // last read before this barrier, next used after another
        uint4 c = make_uint4(0u, 0u, 0u, 0u);
        if (lane < CLUSTER_CTAS) c = *reinterpret_cast<const uint4 *>(cl.map_shared_rank(cnt, lane));
        const uint32_t listed = min(c.x, CLUSTER_LIST);
        uint32_t pre = listed;
#pragma unroll
        for (uint32_t o = 1; o < CLUSTER_CTAS; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL_MASK, pre, o);
            if (lane >= o) pre += y;
        }
        const uint32_t listed_all = __shfl_sync(FULL_MASK, pre, CLUSTER_CTAS - 1);
        pre -= listed;
        const uint32_t f = __reduce_add_sync(FULL_MASK, c.x), longest = __reduce_max_sync(FULL_MASK, listed);
        const unsigned long long fe_all = __reduce_add_sync(FULL_MASK, c.y);
        const uint32_t any_heavy = __reduce_or_sync(FULL_MASK, c.z), mine = __shfl_sync(FULL_MASK, listed, rank);
        unsigned long long ls_all = 0, lq_all = 0;
        float lm_all = 0.f;
        if constexpr (STATS == 1) {
            if (leader) {
                for (unsigned q = 0; q < CLUSTER_CTAS; q++) {
                    const ClusterCounts *h = cl.map_shared_rank(cnt, q);
                    ls_all += h->ls; lq_all += h->lq;
                    lm_all = fmaxf(lm_all, __uint_as_float(h->lm_bits));
                }
            }
        }
        if (f == 0 || f > CLUSTER_CAP || fe_all > CLUSTER_EDGE_CAP || listed_all < f || any_heavy ||
            static_cast<uint32_t>(L) + 2 > max_levels) {
            // hand level L to the step kernel: the next queue (overflow first,
            // then the blocks' lists) and the level's slot
            const uint32_t at = (f - listed_all) + __shfl_sync(FULL_MASK, pre, rank);
            for (uint32_t i = tid; i < mine; i += CLUSTER_THREADS) qnext[at + i] = nv[i];
            unsigned long long hls = ls_all, hlq = lq_all;
            float hlm = lm_all;
            if constexpr (STATS == 2) {
                // The handed-over frontier's log-degree statistics: this
                // block's list entries and its slice of the overflow, which
                // the other blocks wrote to the global queue before the
                // counts' cluster barrier (read past L1).
                unsigned long long ls = 0, lq = 0;
                float lm = 0.f;
                auto add = [&](uint32_t deg) {
                    const float l = __log2f(1.0f + static_cast<float>(deg));
                    ls += lsum_fx(l); lq += lsq_fx(l); lm = fmaxf(lm, l);
                };
                for (uint32_t i = tid; i < mine; i += CLUSTER_THREADS) add(nse[i].y - nse[i].x);
                const uint32_t ov = f - listed_all, per = (ov + CLUSTER_CTAS - 1) / CLUSTER_CTAS;
                const uint32_t ob = min(ov, rank * per), oe = min(ov, ob + per);
                for (uint32_t i = ob + tid; i < oe; i += CLUSTER_THREADS) {
                    const uint32_t v = __ldcg(qnext + i);
                    add(a.fwd_v[v + 1] - a.fwd_v[v]);
                }
                for (int o = 16; o > 0; o >>= 1) {
                    ls += __shfl_xor_sync(FULL_MASK, ls, o);
                    lq += __shfl_xor_sync(FULL_MASK, lq, o);
                    lm = fmaxf(lm, __shfl_xor_sync(FULL_MASK, lm, o));
                }
                if (lane == 0) { r_ls[wib] = ls; r_lq[wib] = lq; r_lm[wib] = lm; }
                __syncthreads();
                if (wib == 0) {
                    constexpr unsigned WARPS = CLUSTER_THREADS / 32;
                    ls = lane < WARPS ? r_ls[lane] : 0; lq = lane < WARPS ? r_lq[lane] : 0; lm = lane < WARPS ? r_lm[lane] : 0.f;
                    for (int o = 16; o > 0; o >>= 1) {
                        ls += __shfl_xor_sync(FULL_MASK, ls, o);
                        lq += __shfl_xor_sync(FULL_MASK, lq, o);
                        lm = fmaxf(lm, __shfl_xor_sync(FULL_MASK, lm, o));
                    }
                    if (lane == 0) { s_hand[0] = ls; s_hand[1] = lq; s_hand[2] = __float_as_uint(lm); }
                }
                cl.sync();                               // every block's part is out
                if (leader) {
                    hls = hlq = 0;
                    hlm = 0.f;
                    for (unsigned q = 0; q < CLUSTER_CTAS; q++) {
                        const unsigned long long *h = cl.map_shared_rank(s_hand, q);
                        hls += h[0]; hlq += h[1];
                        hlm = fmaxf(hlm, __uint_as_float(static_cast<uint32_t>(h[2])));
                    }
                }
            }
            if (leader) {
                slot->frontier = f;
                slot->qlen = f;
                slot->fedges = fe_all;
                slot->lsum = hls;
                slot->lsq = hlq;
                slot->lmax_bits = __float_as_uint(hlm);
                slot->heavy = 0;
                ctl->skip = 1;
                ctl->visited += visited;                 // the step kernel's bookkeeping for the levels before
                ctl->traversed += traversed;
                ctl->levels_done = static_cast<uint32_t>(L);
                ctl->depth = L;
            }
            cl.sync();                                   // no block leaves while others may read its shared memory
            return;
        }
        if (leader) {
            if (a.log && static_cast<uint32_t>(L) < a.log_cap) {
                LevelSlot sl;
                sl.frontier = f;
                sl.qlen = f;
                sl.fedges = fe_all;
                sl.lsum = ls_all;
                sl.lsq = lq_all;
                sl.lmax_bits = __float_as_uint(lm_all);
                sl.heavy = static_cast<uint32_t>(ctl->variant);
                a.log[L] = sl;
            }
            visited += f;
            traversed += fe_all;
        }
        if (longest <= CLUSTER_KEEP) {                   // short lists stay where they were found
            cur = nse;
            ncur = mine;
        } else {
            // this block's equal share of the next frontier, gathered from the
            // blocks' next lists (rank order)
            const uint32_t per = (f + CLUSTER_CTAS - 1) / CLUSTER_CTAS;
            const uint32_t b = min(f, rank * per);
            ncur = min(per, f - b);
            for (uint32_t i0 = wib * 32; i0 < ncur; i0 += CLUSTER_THREADS) {
                const uint32_t i = i0 + lane, j = b + i;
                unsigned q = 0;
#pragma unroll
                for (unsigned r = 1; r < CLUSTER_CTAS; r++)
                    if (__shfl_sync(FULL_MASK, pre, r) <= j) q = r;
                const uint32_t k = j - __shfl_sync(FULL_MASK, pre, q);
                if (i < ncur) share[i] = *cl.map_shared_rank(nse + k, q);
            }
            __syncthreads();
            cur = share;
        }
        p ^= 1;
        L++;
    }
}

}  // namespace bw
