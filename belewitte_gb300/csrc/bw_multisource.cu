// BFS from many sources of one graph at once (bw_batch_run,
// BW_BATCH_SOURCES): one bit per source and vertex, so that a level reads
// the adjacency once for all sources of a pass instead of once per source
// (Then et al., "The More the Merrier: Efficient Multi-Source Graph
// Traversal", VLDB 2014, in its bottom-up form).
//
// A vertex has W words (32 W >= sources of the pass, W a power of two up to
// 32).  Level L ORs the frontier words of a vertex's in-neighbours; what it
// had not visited is its part of the next frontier, at depth L + 1.  A
// frontier buffer is not cleared between the levels that use it: a stale
// word's bits reached every out-neighbour one level after they were set, so
// they add nothing.  Depths are kept as MS_PLANES bit planes and written out
// once at the end, a 128-byte line per source and 32 vertices.  Where the
// planes end before the traversal does, the caller goes on from the depths
// written by then, a CTA per source; a pass that has reached little after many
// levels (a mesh) is given back as it came.
//
// Work split: a warp takes 32 consecutive vertices and sweeps the in-row of
// each that misses a bit some frontier still carries, 32 edges at a time, W
// lanes per edge, until it misses none.  A row is a chain of dependent loads
// (index, words), so the next row's indices are loaded a row ahead.  While few
// vertices are in the frontier, the rows of the 32 are first tested together,
// an edge per lane, against the active-vertex bitmap (128 KB per million
// vertices, in L1/L2), and only those that meet the frontier are swept.  Rows
// above MS_HEAVY edges would hold their warp for the level, so they are cut
// into chunks for a kernel of their own, which ORs them into one accumulator
// per heavy vertex first.
//
// 512 sources of R-MAT scale 20 symmetrised (31M edges) on GB300: 2.6 ms,
// where a CTA per source took 20.9 ms; the depths alone (2.1 GB) take 0.35 ms
// of HBM.  The first big level is bound by the frontier words' L2 sectors,
// the others by the rows' latency.
#include <algorithm>
#include <climits>

#include "bw_internal.cuh"

namespace bw {
namespace {

constexpr int MS_THREADS = 256;
constexpr int MS_WARPS = MS_THREADS / 32;
constexpr int MS_BLOCKS_PER_SM = 8;
constexpr uint32_t MS_PLANES = 5;                  // depths 1 .. 31
constexpr uint32_t MS_LEVELS = (1u << MS_PLANES) - 1;
// Longer rows: chunks of as many edges.  Measured, the case above: 512 edges
// 3.5 ms (32 rows of one warp are 16K edges), 256 2.81, 128 2.78, 64 2.89.
constexpr uint32_t MS_HEAVY = 128;
constexpr uint32_t MS_GROUP = 4;                   // levels launched between two looks at the counters
constexpr uint32_t MS_PASS = 1024;                 // sources of a pass at most
// A pass's words at most, unless one word a vertex takes more already (from
// 805M vertices on).  The heavy rows' accumulators and chunks come on top,
// about 1.1 bytes an edge with 32 words, and 4 bytes a vertex.  The context's
// pool keeps at most this much of a call's scratch; what it took beyond goes
// back to the device.
constexpr uint64_t MS_BYTES = uint64_t(24) << 30;
constexpr int MS_UNROLL = 8;                       // frontier words in flight per lane
constexpr int MS_TEST = 4;                         // edges per lane and step of the bitmap test
constexpr int MS_OUT = 4;                          // lines of a source's depths written together

struct MsCtl {
    uint32_t active[MS_LEVELS + 1];                // vertices of the frontier that level L reads
    uint32_t heavy, chunks;                        // heavy vertices, their chunks
    unsigned long long bits;                       // (vertex, source) pairs visited
    unsigned long long traversed;
    uint32_t live[2][32];                          // by level parity: the sources with a frontier
};

struct MsArgs {
    const uint32_t *off, *src;                     // reverse CSR
    const uint32_t *fwd_off;
    uint32_t n;
    const uint32_t *roots;                         // by unit
    const uint32_t *order;                         // the units to run, as bw_batch_run takes them; nullptr: 0, 1, ..
    uint32_t first, sources;                       // of this pass
    uint32_t *visited;                             // [n][W]
    uint32_t *front[2];                            // [n][W] by level parity
    uint32_t *bitmap[2];                           // a bit per vertex: in that frontier
    uint32_t *planes;                              // [MS_PLANES][n][W]
    uint32_t *heavy_of;                            // heavy vertices' accumulator (by vertex)
    uint32_t *heavy_acc;                           // [heavy][W]
    uint2 *chunk;                                  // {vertex, first edge}
    MsCtl *ctl;
    int32_t *levels;                               // [unit][n]
};

// The unit of the pass's source i.
__device__ __forceinline__ uint32_t unit_of(const MsArgs &a, uint32_t i)
{
    return a.order ? a.order[a.first + i] : a.first + i;
}

// Bits of word w that belong to sources.
__device__ __forceinline__ uint32_t valid_bits(uint32_t sources, uint32_t w)
{
    if (sources >= 32 * (w + 1)) return 0xffffffffu;
    return sources > 32 * w ? (1u << (sources - 32 * w)) - 1u : 0u;
}

template<uint32_t W>
__global__ void k_ms_roots(MsArgs a)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.sources) return;
    const uint32_t r = a.roots[unit_of(a, i)], bit = 1u << (i & 31);
    atomicOr(&a.visited[uint64_t(r) * W + (i >> 5)], bit);
    atomicOr(&a.front[0][uint64_t(r) * W + (i >> 5)], bit);
    atomicOr(&a.ctl->live[0][i >> 5], bit);
    const uint32_t old = atomicOr(&a.bitmap[0][r >> 5], 1u << (r & 31));
    if (!(old >> (r & 31) & 1u)) atomicAdd(&a.ctl->active[0], 1u);
    atomicAdd(&a.ctl->bits, 1ull);
}

// Heavy vertices numbered and their rows cut into chunks, once per call.
__global__ void k_ms_chunks(MsArgs a)
{
    for (uint64_t v = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; v < a.n; v += uint64_t(gridDim.x) * blockDim.x) {
        const uint32_t s = a.off[v], d = a.off[v + 1] - s;
        if (d <= MS_HEAVY) continue;
        a.heavy_of[v] = atomicAdd(&a.ctl->heavy, 1u);
        const uint32_t cnt = (d + MS_HEAVY - 1) / MS_HEAVY, base = atomicAdd(&a.ctl->chunks, cnt);
        for (uint32_t c = 0; c < cnt; c++) a.chunk[base + c] = make_uint2(static_cast<uint32_t>(v), s + c * MS_HEAVY);
    }
}

// Index i + lane of a row that ends at e, and whether that in-neighbour may be
// in the frontier.
__device__ __forceinline__ uint32_t row_index(const MsArgs &a, uint32_t i, uint32_t e)
{
    const uint32_t at = i + (threadIdx.x & 31);
    return at < e ? __ldg(a.src + at) : 0u;
}

// The OR of the frontier words of in-neighbours [s, e), in every slot of W
// lanes; stops when no bit of `need` is missing.  u: row_index(s, e); `buf`:
// 32 words of shared memory per warp.
template<uint32_t W>
__device__ __forceinline__ uint32_t sweep_row(const MsArgs &a, const uint32_t *front, const uint32_t *bitmap, bool dense,
                                              uint32_t s, uint32_t e, uint32_t u, uint32_t need, uint32_t acc, uint32_t *buf)
{
    constexpr uint32_t R = 32 / W;                 // edges a warp reads at a time
    const uint32_t lane = threadIdx.x & 31, word = lane % W, slot = lane / W;
    for (uint32_t i = s; i < e; i += 32) {
        bool on = i + lane < e;
        if (on && !dense) on = (__ldg(bitmap + (u >> 5)) >> (u & 31)) & 1u;
        const uint32_t m = __ballot_sync(FULL_MASK, on), cnt = __popc(m);
        if (on) buf[__popc(m & ((1u << lane) - 1u))] = u;
        if (i + 32 < e) u = row_index(a, i + 32, e);
        if (cnt == 0) continue;
        __syncwarp();
        for (uint32_t k = slot; k < cnt; k += R * MS_UNROLL) {
            uint32_t f[MS_UNROLL];
#pragma unroll
            for (int j = 0; j < MS_UNROLL; j++)
                f[j] = k + j * R < cnt ? __ldg(front + uint64_t(buf[k + j * R]) * W + word) : 0u;
#pragma unroll
            for (int j = 0; j < MS_UNROLL; j++) acc |= f[j];
        }
        __syncwarp();
#pragma unroll
        for (uint32_t o = W; o < 32; o <<= 1) acc |= __shfl_xor_sync(FULL_MASK, acc, o);
        if (!__any_sync(FULL_MASK, (need & ~acc) != 0u)) break;
    }
    return acc;
}

// Whether the level has a frontier at all, and whether most rows will meet
// it: then testing the bitmap first only adds a load per edge.
__device__ __forceinline__ bool level_runs(const MsArgs &a, uint32_t level, bool &dense)
{
    const uint32_t active = *reinterpret_cast<volatile uint32_t *>(&a.ctl->active[level]);
    dense = active > a.n / 8;
    return active != 0;
}

template<uint32_t W>
__global__ void __launch_bounds__(MS_THREADS, 6) k_ms_heavy(MsArgs a, uint32_t level)
{
    __shared__ uint32_t s_buf[MS_WARPS][32];
    bool dense;
    if (!level_runs(a, level, dense)) return;
    const uint32_t lane = threadIdx.x & 31, wib = threadIdx.x >> 5, word = lane % W;
    const uint32_t *front = a.front[level & 1], *bitmap = a.bitmap[level & 1];
    const uint32_t valid = valid_bits(a.sources, word) & a.ctl->live[level & 1][word], chunks = a.ctl->chunks;
    if (blockIdx.x == 0 && threadIdx.x < 32) a.ctl->live[(level + 1) & 1][threadIdx.x] = 0;     // for k_ms_level
    const uint64_t warps = uint64_t(gridDim.x) * MS_WARPS;
    for (uint64_t c = blockIdx.x * uint64_t(MS_WARPS) + wib; c < chunks; c += warps) {
        const uint2 q = a.chunk[c];
        uint32_t *sum = a.heavy_acc + uint64_t(a.heavy_of[q.x]) * W + word;
        const uint32_t need = valid & ~a.visited[uint64_t(q.x) * W + word];
        const uint32_t have = *reinterpret_cast<volatile uint32_t *>(sum);       // what other chunks found
        if (!__any_sync(FULL_MASK, (need & ~have) != 0u)) continue;
        const uint32_t e = min(q.y + MS_HEAVY, a.off[q.x + 1]);
        const uint32_t acc = sweep_row<W>(a, front, bitmap, dense, q.y, e, row_index(a, q.y, e), need, have, s_buf[wib]);
        if (lane < W && (acc & need & ~have)) atomicOr(sum, acc & need);
    }
}

template<uint32_t W>
__global__ void __launch_bounds__(MS_THREADS, 6) k_ms_level(MsArgs a, uint32_t level)
{
    __shared__ uint32_t s_buf[MS_WARPS][32];
    __shared__ uint32_t s_hit[MS_WARPS];
    __shared__ uint32_t s_live[32];
    bool dense;
    if (!level_runs(a, level, dense)) return;
    const uint32_t lane = threadIdx.x & 31, wib = threadIdx.x >> 5, word = lane % W;
    const uint32_t *front = a.front[level & 1], *bitmap = a.bitmap[level & 1];
    uint32_t *next = a.front[(level + 1) & 1], *next_map = a.bitmap[(level + 1) & 1];
    const uint32_t valid = valid_bits(a.sources, word) & a.ctl->live[level & 1][word], depth = level + 1;
    const uint64_t plane = uint64_t(a.n) * W;
    const uint32_t batches = (a.n + 31) / 32;
    uint32_t found = 0, live = 0;
    unsigned long long bits = 0;
    if (threadIdx.x < 32) s_live[threadIdx.x] = 0;
    __syncthreads();
    for (uint32_t b = blockIdx.x * MS_WARPS + wib; b < batches; b += gridDim.x * MS_WARPS) {
        const uint32_t v0 = b * 32, mine = v0 + lane;
        uint32_t s = 0, e = 0;
        if (mine < a.n) {
            s = a.off[mine];
            e = a.off[mine + 1];
        }
        unsigned todo = __ballot_sync(FULL_MASK, e > s);
        {
            // the vertices that miss a live bit: 32 W words in order, R vertices a step
            constexpr uint32_t R = 32 / W;
            uint32_t w[W];
            unsigned lacks = 0;
#pragma unroll
            for (uint32_t k = 0; k < W; k++) {
                const uint32_t v = v0 + k * R + lane / W;
                w[k] = v < a.n ? a.visited[uint64_t(v) * W + word] : 0xffffffffu;
            }
#pragma unroll
            for (uint32_t k = 0; k < W; k++) {
                const unsigned m = __ballot_sync(FULL_MASK, (valid & ~w[k]) != 0u);
#pragma unroll
                for (uint32_t r = 0; r < R; r++)
                    if (m & ((W == 32 ? 0xffffffffu : (1u << W) - 1u) << (r * W % 32))) lacks |= 1u << (k * R + r);
            }
            todo &= lacks;
        }
        const unsigned heavy = __ballot_sync(FULL_MASK, e - s > MS_HEAVY);
        if (!dense && (todo & ~heavy)) {
            // which rows meet the frontier: their edges one after the other, an edge per lane
            const uint32_t d = (todo & ~heavy) >> lane & 1u ? e - s : 0u;
            uint32_t incl = d;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(FULL_MASK, incl, o);
                if (lane >= static_cast<unsigned>(o)) incl += y;
            }
            const uint32_t total = __shfl_sync(FULL_MASK, incl, 31), excl = incl - d, from = s - excl;
            if (lane == 0) s_hit[wib] = 0;
            __syncwarp();
            for (uint32_t k0 = 0; k0 < total; k0 += 32 * MS_TEST) {
                uint32_t u[MS_TEST], row[MS_TEST];
#pragma unroll
                for (int j = 0; j < MS_TEST; j++) {
                    const uint32_t k = k0 + j * 32 + lane;
                    uint32_t l = 0;                // the last lane whose row starts at k or before
#pragma unroll
                    for (uint32_t o = 16; o > 0; o >>= 1)
                        if (__shfl_sync(FULL_MASK, excl, l + o) <= k) l += o;
                    row[j] = l;
                    const uint32_t at = __shfl_sync(FULL_MASK, from, l) + k;
                    u[j] = k < total ? __ldg(a.src + at) : 0xffffffffu;
                }
#pragma unroll
                for (int j = 0; j < MS_TEST; j++)
                    if (u[j] != 0xffffffffu && (__ldg(bitmap + (u[j] >> 5)) >> (u[j] & 31) & 1u))
                        atomicOr(&s_hit[wib], 1u << row[j]);
            }
            __syncwarp();
            todo &= heavy | s_hit[wib];
        }
        uint32_t map = 0;
        uint32_t first = todo ? __ffs(todo) - 1 : 0;
        uint32_t vis = todo ? a.visited[uint64_t(v0 + first) * W + word] : 0u;
        uint32_t u = row_index(a, __shfl_sync(FULL_MASK, s, first), todo ? __shfl_sync(FULL_MASK, e, first) : 0u);
        while (todo) {
            const uint32_t j = __ffs(todo) - 1, v = v0 + j;
            todo &= todo - 1;
            const uint32_t was = vis, need = valid & ~was, u_now = u;
            const uint32_t rs = __shfl_sync(FULL_MASK, s, j), re = __shfl_sync(FULL_MASK, e, j);
            if (todo) {
                const uint32_t nx = __ffs(todo) - 1;
                vis = a.visited[uint64_t(v0 + nx) * W + word];
                u = row_index(a, __shfl_sync(FULL_MASK, s, nx), __shfl_sync(FULL_MASK, e, nx));
            }
            uint32_t acc;
            if (re - rs > MS_HEAVY) {              // k_ms_heavy has swept it
                uint32_t *sum = a.heavy_acc + uint64_t(a.heavy_of[v]) * W + word;
                acc = *sum;
                __syncwarp();
                if (lane < W) *sum = 0;
            } else {
                acc = sweep_row<W>(a, front, bitmap, dense, rs, re, u_now, need, 0u, s_buf[wib]);
            }
            const uint32_t got = acc & need;
            if (!__any_sync(FULL_MASK, got != 0u)) continue;
            map |= 1u << j;
            live |= got;
            if (lane < W) {
                const uint64_t at = uint64_t(v) * W + word;
                next[at] = got;
                a.visited[at] = was | got;
                if (got) {
#pragma unroll
                    for (uint32_t k = 0; k < MS_PLANES; k++)
                        if (depth >> k & 1u) a.planes[k * plane + at] |= got;
                    bits += __popc(got);
                }
            }
        }
        if (lane == 0) next_map[b] = map;
        found += __popc(map);
    }
    for (int o = 16; o > 0; o >>= 1) bits += __shfl_xor_sync(FULL_MASK, bits, o);
    if (lane == 0 && found) {
        atomicAdd(&a.ctl->active[level + 1], found);
        atomicAdd(&a.ctl->bits, bits);
    }
    if (live) atomicOr(&s_live[word], live);
    __syncthreads();
    if (threadIdx.x < W && s_live[threadIdx.x]) atomicOr(&a.ctl->live[(level + 1) & 1][threadIdx.x], s_live[threadIdx.x]);
}

// The depths: one warp per MS_OUT x 32 vertices, word by word, so that a row
// of the result is written MS_OUT whole lines at a time.  Also, where the
// pass is `whole`, the out-edges of every reached (vertex, source) pair.
// ORDERED: the rows are those of a.order.  (A test per row instead took 0.1 ms
// of the 2.75 ms of 512 sources on R-MAT-20.)
template<uint32_t W, bool ORDERED>
__global__ void __launch_bounds__(MS_THREADS) k_ms_depths(MsArgs a, bool whole)
{
    const uint32_t lane = threadIdx.x & 31, wib = threadIdx.x >> 5, words = (a.sources + 31) / 32;
    const uint64_t plane = uint64_t(a.n) * W;
    const uint64_t tasks = uint64_t((a.n + 32 * MS_OUT - 1) / (32 * MS_OUT)) * words, warps = uint64_t(gridDim.x) * MS_WARPS;
    unsigned long long trav = 0;
    for (uint64_t t = blockIdx.x * uint64_t(MS_WARPS) + wib; t < tasks; t += warps) {
        const uint32_t v0 = static_cast<uint32_t>(t / words) * (32 * MS_OUT) + lane, w = static_cast<uint32_t>(t % words);
        uint32_t vis[MS_OUT], p[MS_OUT][MS_PLANES];
#pragma unroll
        for (int q = 0; q < MS_OUT; q++) {
            const uint32_t v = v0 + 32 * q;
            if (v >= a.n) continue;
            const uint64_t at = uint64_t(v) * W + w;
            vis[q] = a.visited[at];
#pragma unroll
            for (uint32_t k = 0; k < MS_PLANES; k++) p[q][k] = a.planes[k * plane + at];
            trav += static_cast<unsigned long long>(__popc(vis[q])) * (a.fwd_off[v + 1] - a.fwd_off[v]);
        }
        const uint32_t cnt = min(32u, a.sources - 32 * w);
        int32_t *out = a.levels + uint64_t(a.first + 32 * w) * a.n + v0;
        for (uint32_t b = 0; b < cnt; b++, out += a.n) {
            if constexpr (ORDERED) out = a.levels + uint64_t(unit_of(a, 32 * w + b)) * a.n + v0;
#pragma unroll
            for (int q = 0; q < MS_OUT; q++) {
                int32_t d = 0;
#pragma unroll
                for (uint32_t k = 0; k < MS_PLANES; k++) d |= static_cast<int32_t>((p[q][k] >> b & 1u) << k);
                if (v0 + 32 * q < a.n) __stcs(out + 32 * q, (vis[q] >> b & 1u) ? d : INF);
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) trav += __shfl_xor_sync(FULL_MASK, trav, o);
    if (lane == 0 && trav && whole) atomicAdd(&a.ctl->traversed, trav);
}

// One pass.  resume: MS_DONE, or the depth up to which its sources' depths are
// written, their frontiers being the vertices at that depth; 0 with nothing
// written where `mesh` says that little had been reached (going on from there
// instead: 512 sources on the 1024 x 1024 grid 45.0 ms, from the roots 43.7).
template<uint32_t W>
int run_pass(bw_context *ctx, const MsArgs &a, int32_t &resume, bool &mesh, cudaStream_t s)
{
    const unsigned grid = static_cast<unsigned>(ctx->sm_count) * MS_BLOCKS_PER_SM;
    bool done = false;
    BW_CUDA(cudaMemsetAsync(a.visited, 0, uint64_t(a.n) * W * sizeof(uint32_t) * (3 + MS_PLANES), s));   // with the frontiers and planes
    BW_CUDA(cudaMemsetAsync(a.bitmap[0], 0, (a.n + 31) / 32 * sizeof(uint32_t), s));
    BW_CUDA(cudaMemsetAsync(a.ctl->active, 0, sizeof a.ctl->active, s));
    BW_CUDA(cudaMemsetAsync(&a.ctl->bits, 0, sizeof a.ctl->bits, s));
    BW_CUDA(cudaMemsetAsync(a.ctl->live, 0, sizeof a.ctl->live, s));
    k_ms_roots<W><<<(a.sources + 255) / 256, 256, 0, s>>>(a);
    MsCtl h;
    uint32_t level = 0;
    while (level < MS_LEVELS && !done && !mesh) {
        for (uint32_t end = std::min(level + MS_GROUP, MS_LEVELS); level < end; level++) {
            k_ms_heavy<W><<<grid, MS_THREADS, 0, s>>>(a, level);
            k_ms_level<W><<<grid, MS_THREADS, 0, s>>>(a, level);
        }
        BW_CUDA(cudaGetLastError());
        BW_CUDA(cudaMemcpyAsync(&h, a.ctl, sizeof h, cudaMemcpyDeviceToHost, s));
        BW_CUDA(cudaStreamSynchronize(s));
        done = h.active[level] == 0;
        // little reached after many levels (a mesh, a chain): not worth going on.  Random graphs of average
        // degree 4 have reached 1/16 of a million vertices by level 8.  Four levels say nothing yet: a source
        // at the end of a short path comes to the rest of its graph after them (one source, a path of 6 on
        // R-MAT-19 symmetrised: 1.05 ms, 2.72 when given back at level 4).
        mesh = !done && level >= 2 * MS_GROUP &&
               h.bits < uint64_t(a.n) * a.sources / (level < 4 * MS_GROUP ? 64 : 16);
    }
    if (mesh) {
        resume = 0;
        return BW_OK;
    }
    if (a.order) k_ms_depths<W, true><<<grid, MS_THREADS, 0, s>>>(a, done);
    else k_ms_depths<W, false><<<grid, MS_THREADS, 0, s>>>(a, done);
    BW_CUDA(cudaGetLastError());
    resume = done ? MS_DONE : static_cast<int32_t>(level);
    return BW_OK;
}

}  // namespace

// BFS from `count` sources in passes of *pass.  resume[p]: how far pass p got,
// MS_DONE or the depth to go on from (0: nothing written); empty when memory
// is short, with nothing written.  traversed: out-edges of the reached
// vertices, summed over the sources of the finished passes.
int bfs_multi_source(bw_context *ctx, const bw_graph_view *g, const uint32_t *roots, const uint32_t *order,
                     uint32_t count, int32_t *levels, uint64_t *traversed, uint32_t *pass,
                     std::vector<int32_t> &resume, cudaStream_t s)
{
    resume.clear();
    *traversed = 0;
    const uint32_t n = static_cast<uint32_t>(g->vertex_count);
    uint32_t W = 1;                                // words per vertex: all sources, while the scratch stays bounded
    while (W < MS_PASS / 32 && 32 * W < count && uint64_t(n) * 2 * W * 4 * (3 + MS_PLANES) <= MS_BYTES) W *= 2;
    auto al = [](uint64_t b) { return (b + 255) & ~uint64_t(255); };
    const uint64_t hcap = g->edge_count / (MS_HEAVY + 1) + 1, ccap = g->edge_count / MS_HEAVY + hcap;
    const uint64_t o_vis = al(sizeof(MsCtl)), per = uint64_t(n) * W * 4, o_map = o_vis + al(per * (3 + MS_PLANES)),
                   map = al((uint64_t(n) + 31) / 32 * 4), o_of = o_map + 2 * map, o_acc = o_of + al(uint64_t(n) * 4),
                   o_chunk = o_acc + al(hcap * W * 4), bytes = o_chunk + al(ccap * sizeof(uint2));
    char *mem = nullptr;
    const cudaError_t e = ctx_malloc_async(ctx, reinterpret_cast<void **>(&mem), bytes, s);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        return BW_OK;
    }
    BW_CUDA(e);
    MsArgs a{};
    a.off = g->rev_vertices; a.src = g->rev_edges; a.fwd_off = g->fwd_vertices;
    a.n = n;
    a.roots = roots; a.order = order; a.levels = levels;
    a.ctl = reinterpret_cast<MsCtl *>(mem);
    a.visited = reinterpret_cast<uint32_t *>(mem + o_vis);
    a.front[0] = a.visited + uint64_t(n) * W;
    a.front[1] = a.front[0] + uint64_t(n) * W;
    a.planes = a.front[1] + uint64_t(n) * W;
    a.bitmap[0] = reinterpret_cast<uint32_t *>(mem + o_map);
    a.bitmap[1] = reinterpret_cast<uint32_t *>(mem + o_map + map);
    a.heavy_of = reinterpret_cast<uint32_t *>(mem + o_of);
    a.heavy_acc = reinterpret_cast<uint32_t *>(mem + o_acc);
    a.chunk = reinterpret_cast<uint2 *>(mem + o_chunk);
    auto passes = [&]() -> int {
        BW_CUDA(cudaMemsetAsync(a.ctl, 0, sizeof(MsCtl), s));
        BW_CUDA(cudaMemsetAsync(a.heavy_acc, 0, hcap * W * 4, s));
        k_ms_chunks<<<ctx->sm_count * 4, 256, 0, s>>>(a);
        *pass = 32 * W;
        resume.assign((count + 32 * W - 1) / (32 * W), 0);
        bool mesh = false;                         // then the passes that follow are left to the caller
        for (uint32_t first = 0; first < count && !mesh; first += 32 * W) {
            a.first = first;
            a.sources = std::min(count - first, 32 * W);
            int32_t &at = resume[first / (32 * W)];
            int rc = BW_ERR_INVALID_ARGUMENT;
            switch (W) {
              case 1: rc = run_pass<1>(ctx, a, at, mesh, s); break;
              case 2: rc = run_pass<2>(ctx, a, at, mesh, s); break;
              case 4: rc = run_pass<4>(ctx, a, at, mesh, s); break;
              case 8: rc = run_pass<8>(ctx, a, at, mesh, s); break;
              case 16: rc = run_pass<16>(ctx, a, at, mesh, s); break;
              case 32: rc = run_pass<32>(ctx, a, at, mesh, s); break;
            }
            BW_TRY(rc);
        }
        unsigned long long t = 0;
        BW_CUDA(cudaMemcpyAsync(&t, &a.ctl->traversed, sizeof t, cudaMemcpyDeviceToHost, s));
        BW_CUDA(cudaStreamSynchronize(s));
        *traversed = t;
        return BW_OK;
    };
    const int rc = passes();
    cudaFreeAsync(mem, s);
    if (bytes > MS_BYTES && ctx->pool && cudaStreamSynchronize(s) == cudaSuccess) cudaMemPoolTrimTo(ctx->pool, MS_BYTES);
    return rc;
}

}  // namespace bw
