// The context's scratch arrays, grown on demand (host code only).
#include <cstring>

#include "bw_internal.cuh"

namespace bw {

// `cap` is what the array holds: nothing from the moment its memory goes until
// the new one is there, so that after a failed allocation no later, smaller
// call takes the array for one of the old size.
template<typename T, typename Cap>
static int grow(T **ptr, uint64_t count, Cap &cap)
{
    cap = 0;
    if (*ptr) { cudaFree(*ptr); *ptr = nullptr; }
    if (count == 0) count = 1;
    BW_CUDA(cudaMalloc(reinterpret_cast<void **>(ptr), count * sizeof(T)));
    return BW_OK;
}

// The control block on the device and, in one pinned allocation, its mirror
// and the mailbox.  ctx->bfs_ctl is set last: where it is, all three are.
static int make_bfs_ctl(bw_context *ctx)
{
    constexpr size_t at = (sizeof(BfsCtl) + 127) & ~size_t(127);       // the mail on lines of its own
    if (!ctx->bfs_ctl_host)
        BW_CUDA(cudaMallocHost(reinterpret_cast<void **>(&ctx->bfs_ctl_host), at + sizeof(BfsMail)));
    ctx->mail = reinterpret_cast<BfsMail *>(reinterpret_cast<char *>(ctx->bfs_ctl_host) + at);
    std::memset(ctx->mail, 0, sizeof(BfsMail));
    ctx->mail_seq = 0;
    BfsCtl *ctl = nullptr;
    BW_CUDA(cudaMalloc(reinterpret_cast<void **>(&ctl), sizeof(BfsCtl)));
    const cudaError_t e = cudaMemset(ctl, 0, sizeof(BfsCtl));
    if (e != cudaSuccess) cudaFree(ctl);
    BW_CUDA(e);
    ctx->bfs_ctl = ctl;
    return BW_OK;
}

int ensure_bfs_scratch(bw_context *ctx, uint64_t n, uint64_t m)
{
    if (!ctx->bfs_ctl) BW_TRY(make_bfs_ctl(ctx));
    if (n > ctx->bfs_n_cap) {
        BW_TRY(grow(&ctx->queue[0], n, ctx->bfs_n_cap));
        BW_TRY(grow(&ctx->queue[1], n, ctx->bfs_n_cap));
        ctx->bfs_n_cap = n;
    }
    // Hub chunks: every queued vertex has degree > 256 and yields at most
    // 2*deg/256 chunks of 256 edges, so 2M/256 + N/256 bounds a level.
    uint64_t hcap = 2 * m / 256 + n / 256 + 1024;
    if (hcap > ctx->heavy_cap) {
        BW_TRY(grow(&ctx->heavy, hcap, ctx->heavy_cap));
        ctx->heavy_cap = hcap;
    }
    return BW_OK;
}

int ensure_outdeg_scratch(bw_context *ctx, uint64_t n)
{
    if (n > ctx->outdeg_cap) {
        BW_TRY(grow(&ctx->outdeg, n, ctx->outdeg_cap));
        ctx->outdeg_cap = n;
    }
    return BW_OK;
}

int ensure_pr_scratch(bw_context *ctx, uint64_t n, uint32_t iterations)
{
    if (n > ctx->pr_n_cap) {
        BW_TRY(grow(&ctx->pr_acc, n, ctx->pr_n_cap));
        // both contribution buffers in one allocation, so one L2
        // access-policy window covers the vector every iteration gathers;
        // the second starts on a 256-byte boundary (the kernels read both
        // with 16-byte vector loads)
        const uint64_t stride = (n + 63) & ~uint64_t(63);
        BW_TRY(grow(&ctx->pr_buf[0], 2 * stride, ctx->pr_n_cap));
        ctx->pr_buf[1] = ctx->pr_buf[0] + stride;
        BW_TRY(grow(&ctx->pr_deg, n, ctx->pr_n_cap));
        ctx->pr_n_cap = n;
    }
    uint32_t need = iterations + 1;
    if (need > ctx->pr_diff_cap) {
        BW_TRY(grow(&ctx->pr_diffs, need, ctx->pr_diff_cap));
        ctx->pr_diff_cap = need;
    }
    return BW_OK;
}

}  // namespace bw
