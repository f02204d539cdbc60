"""The context's scratch arrays (csrc/bw_scratch.cu) when an allocation fails:
the call reports it, and a later call that needs less finds arrays of the size
it asks for, whichever allocation failed.  The unit is host code; it is built
here against an allocator that fails on request."""
import shutil
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "belewitte_gb300" / "csrc"

CHECK = r"""
#include <cstdio>
#include <cstdlib>
#include <map>
#include "bw_scratch.cu"

static std::map<void *, size_t> live;
static long countdown = -1;                        // allocations until one fails; < 0: never
static bool fails() { return countdown >= 0 && countdown-- == 0; }
static cudaError_t give(void **p, size_t bytes)
{
    if (fails()) return cudaErrorMemoryAllocation;  // *p stays as it was
    *p = std::malloc(1);                            // an address; the size is what counts
    live[*p] = bytes;
    return cudaSuccess;
}
static cudaError_t take(void *p) { if (p && !live.erase(p)) std::abort(); std::free(p); return cudaSuccess; }
extern "C" {
cudaError_t cudaMalloc(void **p, size_t b) { return give(p, b); }
cudaError_t cudaFree(void *p) { return take(p); }
cudaError_t cudaMemset(void *, int, size_t) { return fails() ? cudaErrorUnknown : cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { return take(p); }
cudaError_t cudaMallocHost(void **p, size_t b)
{
    if (fails()) return cudaErrorMemoryAllocation;
    *p = std::calloc(1, b);                         // the mailbox is cleared on the host
    live[*p] = b;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
}
namespace bw { void set_last_error(cudaError_t, const char *) {} }
using namespace bw;

static int bad = 0;
static size_t size_of(const void *p) { auto it = live.find(const_cast<void *>(p)); return p && it != live.end() ? it->second : 0; }
static void holds(const char *what, const void *p, size_t bytes)
{
    if (size_of(p) < bytes) { bad++; std::printf("%s: %zu of %zu bytes\n", what, size_of(p), bytes); }
}
static void capacities(const bw_context &c)          // never more than is there
{
    holds("queue 0", c.queue[0], c.bfs_n_cap * 4); holds("queue 1", c.queue[1], c.bfs_n_cap * 4);
    holds("heavy", c.heavy, c.heavy_cap * sizeof(uint2));
    holds("outdeg", c.outdeg, c.outdeg_cap * 4);
    holds("acc", c.pr_acc, c.pr_n_cap * 4); holds("deg", c.pr_deg, c.pr_n_cap * 4);
    holds("buf", c.pr_buf[0], 2 * c.pr_n_cap * 4); holds("diffs", c.pr_diffs, size_t(c.pr_diff_cap) * 4);
}
static int all(bw_context &c, uint64_t n, uint64_t m, uint32_t it)
{
    const int a = ensure_bfs_scratch(&c, n, m), b = ensure_outdeg_scratch(&c, n), p = ensure_pr_scratch(&c, n, it);
    return a != BW_OK ? a : b != BW_OK ? b : p;
}
static void serves(bw_context &c, uint64_t n, uint64_t m, uint32_t it)
{
    if (all(c, n, m, it) != BW_OK) { bad++; std::printf("refused\n"); return; }
    capacities(c);
    holds("queue 0", c.queue[0], n * 4); holds("queue 1", c.queue[1], n * 4);
    holds("heavy", c.heavy, (2 * m / 256 + n / 256 + 1024) * sizeof(uint2));
    holds("control block", c.bfs_ctl, sizeof(BfsCtl));
    holds("host block", c.bfs_ctl_host, sizeof(BfsCtl) + sizeof(BfsMail));
    const char *mail = reinterpret_cast<const char *>(c.mail), *host = reinterpret_cast<const char *>(c.bfs_ctl_host);
    if (!mail || mail < host + sizeof(BfsCtl) || mail + sizeof(BfsMail) > host + size_of(host)) { bad++; std::printf("mailbox\n"); }
    holds("outdeg", c.outdeg, n * 4);
    holds("acc", c.pr_acc, n * 4); holds("deg", c.pr_deg, n * 4); holds("diffs", c.pr_diffs, (it + 1) * 4);
    holds("buf", c.pr_buf[0], 2 * n * 4);
    if (c.pr_buf[1] < c.pr_buf[0] + n) { bad++; std::printf("second buffer\n"); }
}

int main()
{
    long failures = 0;
    for (const bool warm : {false, true}) {           // a first use, or arrays that grow
        for (long k = 0; k < 100; k++) {
            bw_context c;
            if (warm) serves(c, 1000, 5000, 10);
            countdown = k;
            const int rc = all(c, 1000000, 400000000, 300);
            const bool failed = countdown < 0;
            countdown = -1;
            if (failed && rc == BW_OK) { bad++; std::printf("failure %ld not reported\n", k); }
            capacities(c);
            serves(c, 500, 2000, 5);
            serves(c, 900000, 300000000, 250);
            if (!failed) break;
            failures++;
        }
    }
    std::printf("failures %ld bad %d\n", failures, bad);
    return bad || failures < 16 ? 1 : 0;
}
"""


def test_a_failed_allocation_leaves_no_stale_capacity(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda = Path(nvcc).resolve().parent.parent
    src = tmp_path / "scratch.cpp"
    src.write_text(CHECK)
    exe = tmp_path / "scratch"
    subprocess.run(["g++", "-O1", "-std=c++17", f"-I{CSRC}", f"-I{ROOT / 'include'}", f"-I{cuda / 'include'}",
                    "-I/usr/local/cuda/include", str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout[-3000:]
