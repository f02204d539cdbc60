"""The float form of the consolidation (csrc/bw_consolidate.h,
add_round_split) against real double arithmetic on the CPU: wherever it says
that it has decided, the bits are those of fl32(fl64(B + x)); it decides nearly
every ordinary product and none out of its domain."""
import subprocess
from pathlib import Path

HEADER = Path(__file__).resolve().parent.parent / "belewitte_gb300" / "csrc" / "bw_consolidate.h"

CHECK = r"""
#include <cstdio>
#include <cmath>
#include <initializer_list>
#include <limits>
#include "bw_consolidate.h"
using namespace bwcons;
static uint64_t rng = 0x9e3779b97f4a7c15ULL;
static uint64_t nxt() { rng ^= rng << 13; rng ^= rng >> 7; rng ^= rng << 17; return rng; }
static long tested = 0, decided = 0, bad = 0;
static void check(double B, float x) {
    volatile double sum = B + static_cast<double>(x);
    volatile float want = static_cast<float>(sum);
    bool ok;
    const float got = add_round_split(split_base(B), x, ok);
    tested++;
    if (!ok) return;
    decided++;
    if (f32_bits(got) != f32_bits(want)) { if (bad++ < 5) std::printf("B=%a x=%a got=%a want=%a\n", B, x, got, want); }
}
int main() {
    const float inf = std::numeric_limits<float>::infinity();
    // ordinary products: x from 2^-40 to 2^20 of B, every N in geometric steps
    for (double n = 1; n < 5e9; n = n * 1.21 + 1) {
        const double B = (1.0 - static_cast<double>(0.85f)) / std::floor(n);
        check(B, 0.0f);
        for (int i = 0; i < 60000; i++) {
            const uint64_t r = nxt();
            check(B, static_cast<float>(B * std::ldexp(1.0, static_cast<int>(r % 60) - 40)) *
                         (1.0f + static_cast<float>((r >> 8) & 0xffffff) / 16777216.0f));
        }
    }
    const long ordinary = tested, ordinary_decided = decided;
    // sums at and next to float rounding boundaries and powers of two
    for (int i = 0; i < 20000000; i++) {
        const uint64_t r = nxt();
        const double B = std::ldexp(1.0 + static_cast<double>(r & ((1ULL << 52) - 1)) / 4503599627370496.0,
                                    -static_cast<int>((r >> 52) % 40));
        const float y = f32_of(f32_bits(static_cast<float>(B)) + static_cast<uint32_t>(nxt() % 5000)) *
                        static_cast<float>(1u << (nxt() % 12));
        const float near_power = std::ldexp(1.0f, static_cast<int>(nxt() % 12) - static_cast<int>((r >> 52) % 40));
        const double half = std::ldexp(1.0, std::ilogb(y) - 24);
        const double aim = i % 3 == 0 ? static_cast<double>(y) + half : i % 3 == 1 ? static_cast<double>(y) - half
                                                                                   : static_cast<double>(near_power);
        float x = static_cast<float>(aim - B);
        if (!(x >= 0.0f)) continue;
        check(B, x);
        check(B, std::nextafter(x, inf));
        check(B, std::nextafter(x, 0.0f));
    }
    const double b0 = 1e-8;
    long wrong = 0;
    for (float x : {-1.0f, inf, -inf, std::nanf(""), 3e38f}) { bool ok; add_round_split(split_base(b0), x, ok); wrong += ok; }
    for (double b : {0.0, -1.0, 1e-40, 1e300}) { bool ok; add_round_split(split_base(b), 1.0f, ok); wrong += ok; }
    std::printf("tested %ld decided %ld ordinary %ld of %ld bad %ld wrong %ld\n", tested, decided, ordinary_decided, ordinary, bad, wrong);
    return bad || wrong || ordinary - ordinary_decided > ordinary / 100;
}
"""


def test_split_form(tmp_path):
    src = tmp_path / "split.cpp"
    src.write_text(CHECK)
    exe = tmp_path / "split"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{HEADER.parent}", str(src), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout
