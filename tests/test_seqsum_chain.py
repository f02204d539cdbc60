"""A run's binade map from two float chains (csrc/bw_seqsum.h, Chain) against
the plain loop and the term-by-term maps: from every kind of start (smallest,
largest, random; even and odd) the map gives the loop's sum while it stays in
the binade, and leaves the binade where the loop does."""
import subprocess
from pathlib import Path

HEADER = Path(__file__).resolve().parent.parent / "belewitte_gb300" / "csrc" / "bw_seqsum.h"

CHECK = r"""
#include <cstdio>
#include "bw_seqsum.h"
using namespace bwseq;
static uint64_t rng = 0x9e3779b97f4a7c15ULL;
static uint64_t nxt() { rng ^= rng << 13; rng ^= rng >> 7; rng ^= rng << 17; return rng; }
int main() {
    long bad = 0, stayed = 0, left = 0, ties = 0;
    const uint32_t ks[] = {1, 2, 24, 25, 26, 100, 127, 252, 253, 254};
    for (long i = 0; i < 400000; i++) {
        const uint32_t k = i % 3 ? 1 + nxt() % 254 : ks[nxt() % 10];
        const uint32_t len = 1 + nxt() % 32, shift = nxt() % 28;
        uint32_t x[32];
        for (uint32_t u = 0; u < len; u++) {
            const uint64_t r = nxt();
            const int32_t kx = static_cast<int32_t>(k) - static_cast<int32_t>(shift) - static_cast<int32_t>(r % 3);
            uint32_t mant = static_cast<uint32_t>(nxt()) & 0x7fffffu;
            const uint32_t d = k - static_cast<uint32_t>(kx);
            if (r % 5 == 0 && kx > 0 && d >= 1 && d <= 23)           // a constructed tie
                mant = ((mant >> d) << d | (1u << (d - 1))) & 0x7fffffu, ties++;
            x[u] = kx > 0 ? static_cast<uint32_t>(kx) << 23 | mant : (r % 2 ? mant : 0u);   // subnormal or zero
            if (r % 97 == 0) x[u] = 0;
            if (r % 211 == 0) x[u] = 0x7f7fffffu;                    // the largest finite term
        }
        Chain c = chain_start(k);
        Map t = identity();
        bool normal = true;
        for (uint32_t u = 0; u < len; u++) {
            chain_add(c, float_of(x[u]));
            Map s = identity();
            normal = step(x[u], k, s) && normal;
            t = compose(t, s);
        }
        const Map m = chain_map(c, k);
        for (int trial = 0; trial < 8; trial++) {
            uint32_t a = trial == 0 ? ONE : trial == 1 ? ONE + 1 : trial == 2 ? TOP - 1 : trial == 3 ? TOP - 2
                         : ONE + static_cast<uint32_t>(nxt() % ONE);
            float s = float_of(bits_of(k, a));
            bool in = true;
            for (uint32_t u = 0; u < len && in; u++) {
                volatile float v = s + float_of(x[u]);
                s = v;
                in = exponent_of(float_bits(s)) == k;
            }
            const uint32_t got = apply(m, a);
            if (in ? got != significand_of(float_bits(s)) : got < TOP) bad++;
            if (normal && in && apply(t, a) != got) bad++;
            (in ? stayed : left)++;
        }
    }
    std::printf("bad %ld stayed %ld left %ld ties %ld\n", bad, stayed, left, ties);
    return bad || stayed < 100000 || left < 100000 || ties < 100000;
}
"""


def test_chain_map(tmp_path):
    src = tmp_path / "chain.cpp"
    src.write_text(CHECK)
    exe = tmp_path / "chain"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{HEADER.parent}", str(src), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout
