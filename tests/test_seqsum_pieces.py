"""The long-row sums as the kernels evaluate them, against the plain loop
s = fl(s + x[i]) on the CPU, bit for bit: bw_seqsum_warp.cuh's windows (a lane's
run as two float chains, the lanes' maps scanned, a binade crossing found by
plain additions) and k_pr_long_sums' giant rows (a start of one 512-term piece
in order, a record per later piece under a guessed running sum, the records
combined in order in groups of 32, runs of them with one scan).  The guesses
are the kernels' own (float sums of the pieces before), or made wrong at
random: a record may only be applied where it holds, whatever it was made for,
so the sum must not change."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "belewitte_gb300" / "csrc"

CHECK = r"""
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "bw_seqsum.h"
using namespace bwseq;

static uint64_t rng = 0x9e3779b97f4a7c15ULL;
static uint64_t nxt() { rng ^= rng << 13; rng ^= rng >> 7; rng ^= rng << 17; return rng; }
static double unit() { return (nxt() >> 11) * (1.0 / 9007199254740992.0); }
static uint32_t fb(float f) { return float_bits(f); }
static float plus(float a, float b) { volatile float s = a + b; return s; }

constexpr uint32_t PIECE = 512, PIECE_L = 16, SERIAL = 1024;
static uint32_t L = PIECE_L;                                   // terms a lane holds of a window

struct Lanes { Map m[32]; };
static Lanes scanned(Lanes a)                                   // Kogge-Stone, inclusive
{
    for (int o = 1; o < 32; o <<= 1) {
        const Lanes was = a;
        for (int l = o; l < 32; l++) a.m[l] = compose(was.m[l - o], was.m[l]);
    }
    return a;
}

// warp_sequential_continue over [b, e); false: outside the maps' domain.
static bool window_sum(const std::vector<float> &v, uint32_t b, uint32_t e, uint32_t &sb)
{
    const uint32_t WIN = 32 * L;
    for (uint32_t w = b; w < e; w += WIN) {
        const uint32_t lim = std::min(WIN, e - w);
        uint32_t pos = 0;
        auto term = [&](uint32_t k) { return w + k < e ? fb(v[w + k]) : 0u; };
        if (w < SERIAL) {
            const uint32_t upto = std::min(lim, SERIAL - w);
            float acc = float_of(sb);
            for (uint32_t i = 0; i < upto; i++) acc = plus(acc, v[w + i]);
            sb = fb(acc);
            pos = upto;
        }
        for (uint32_t guard = 0; pos < lim; guard++) {
            if (guard > WIN + 1) return false;
            if (sb == 0) {
                uint32_t k = pos;
                while (k < lim && !(term(k) & 0x7fffffffu)) k++;
                if (k == lim) break;
                sb = term(k);
                pos = k + 1;
                if (!in_domain(sb)) return false;
                continue;
            }
            if (!in_domain(sb)) return false;
            const uint32_t K = exponent_of(sb), A = significand_of(sb);
            Lanes m;
            uint32_t worst = 0;
            for (uint32_t l = 0; l < 32; l++) {
                Chain c = chain_start(K);
                for (uint32_t u = 0; u < L; u++) {
                    const uint32_t k = l * L + u, x = k >= pos && k < lim ? term(k) : 0u;
                    worst = std::max(worst, x);
                    chain_add(c, float_of(x));
                }
                m.m[l] = chain_map(c, K);
            }
            if (worst > CHAIN_TERM_MAX) return false;
            const Lanes incl = scanned(m);
            uint32_t f = 32, a0 = 0, a1 = 0;
            for (uint32_t l = 0; l < 32; l++) {
                const uint32_t at = apply(l ? incl.m[l - 1] : identity(), A);
                a1 = apply(m.m[l], at);
                if (a1 >= TOP) { f = l; a0 = at; break; }
            }
            if (f == 32) { sb = bits_of(K, a1); break; }
            float acc = float_of(bits_of(K, a0));
            uint32_t np = 0;
            for (uint32_t u = 0; u < L && np == 0; u++) {
                const uint32_t k = f * L + u;
                if (k < pos || k >= lim) continue;
                acc = plus(acc, v[w + k]);
                if (exponent_of(fb(acc)) != K) np = k + 1;
            }
            sb = fb(acc);
            if (np <= pos || exponent_of(sb) == 0xffu) return false;
            pos = np;
        }
    }
    return true;
}

enum { NONE, BINADE, STATE, CROSS };
struct Rec { uint32_t kind = NONE, K = 0, K2 = 0, tg = 0, xb = 0; Map m1{0, 0}, m2{0, 0}; };

static Map lane_map(const std::vector<float> &t, uint32_t K, uint32_t first, uint32_t from, uint32_t &worst)
{
    Chain c = chain_start(K);
    for (uint32_t u = 0; u < PIECE_L; u++) {
        const float x = first + u >= from ? t[first + u] : 0.0f;
        worst = std::max(worst, fb(x));
        chain_add(c, x);
    }
    return chain_map(c, K);
}

// record_of_terms: t holds the piece's terms, past its end +0.
static Rec record(const std::vector<float> &t, uint32_t guess)
{
    Rec r;
    if (!in_domain(guess)) return r;
    const uint32_t K = exponent_of(guess);
    uint32_t worst = 0;
    Lanes m;
    for (uint32_t l = 0; l < 32; l++) m.m[l] = lane_map(t, K, l * PIECE_L, 0, worst);
    if (worst > CHAIN_TERM_MAX) return r;
    const Lanes incl = scanned(m);
    uint32_t f = 32, a0 = 0;
    for (uint32_t l = 0; l < 32 && f == 32; l++) {
        a0 = apply(l ? incl.m[l - 1] : identity(), significand_of(guess));
        if (apply(m.m[l], a0) >= TOP) f = l;
    }
    if (f == 32) { r.kind = BINADE; r.K = K; r.m1 = incl.m[31]; return r; }
    Chain before = chain_start(K);
    float acc = float_of(bits_of(K, a0));
    uint32_t tg = 0, xb = 0, nb = 0;
    for (uint32_t u = 0; u < PIECE_L; u++) {
        const float x = t[f * PIECE_L + u];
        acc = plus(acc, x);
        nb = fb(acc); tg = f * PIECE_L + u; xb = fb(x);
        if (exponent_of(nb) != K) break;
        chain_add(before, x);
    }
    const Map m1 = compose(f ? incl.m[f - 1] : identity(), chain_map(before, K));
    if (!in_domain(nb)) return r;
    const uint32_t K2 = exponent_of(nb);
    Lanes after;                                              // the terms after tg, composed as a tree
    for (uint32_t l = 0; l < 32; l++) after.m[l] = lane_map(t, K2, l * PIECE_L, tg + 1, worst);
    for (uint32_t o = 1; o < 32; o <<= 1)
        for (uint32_t l = 0; l + o < 32; l += 2 * o) after.m[l] = compose(after.m[l], after.m[l + o]);
    r.kind = CROSS; r.K = K; r.K2 = K2; r.tg = tg; r.xb = xb; r.m1 = m1; r.m2 = after.m[0];
    return r;
}

static long applied = 0, crossed = 0, exact = 0;
static bool advance(const std::vector<float> &v, uint32_t q, const Rec &r, uint32_t &sb)   // piece_advance
{
    if ((r.kind == BINADE || r.kind == CROSS) && in_domain(sb) && exponent_of(sb) == r.K) {
        const uint32_t a1 = apply(r.m1, significand_of(sb));
        if (r.kind == BINADE && a1 < TOP) { sb = bits_of(r.K, a1); applied++; return true; }
        if (r.kind == CROSS && a1 < TOP) {
            const uint32_t nb = fb(plus(float_of(bits_of(r.K, a1)), float_of(r.xb)));
            if (in_domain(nb) && exponent_of(nb) == r.K2) {
                const uint32_t a3 = apply(r.m2, significand_of(nb));
                if (a3 < TOP) { sb = bits_of(r.K2, a3); crossed++; return true; }
            }
        }
    }
    exact++;
    return window_sum(v, q * PIECE, std::min<uint32_t>(v.size(), (q + 1) * PIECE), sb);
}

static int wrong = 0;                                          // guesses made wrong
static bool giant_sum(const std::vector<float> &v, uint32_t &out)
{
    const uint32_t n = v.size(), P = (n + PIECE - 1) / PIECE;
    std::vector<float> sums(P, 0.0f);
    for (uint32_t p = 0; p < P; p++)
        for (uint32_t i = p * PIECE; i < std::min(n, (p + 1) * PIECE); i++) sums[p] = plus(sums[p], v[i]);
    std::vector<Rec> rec(P);
    for (uint32_t q = 1; q < P; q++) {
        float pre = 0.0f;
        for (uint32_t i = 0; i < q; i++) pre = plus(pre, sums[i]);
        uint32_t g = fb(pre);
        if (wrong) {
            const uint32_t r = nxt() % 6;
            if (r == 1 && exponent_of(g) > 1) g -= 1u << 23;
            if (r == 2 && exponent_of(g) < 0xfdu) g += 1u << 23;
            if (r == 3) g = 0;
            if (r == 4) g ^= static_cast<uint32_t>(nxt()) & 0x7fffffu;
            if (r == 5) g |= 0x7fff00u;                        // next to the binade's end: a crossing recorded
        }
        std::vector<float> t(PIECE, 0.0f);
        std::copy(v.begin() + q * PIECE, v.begin() + std::min(n, (q + 1) * PIECE), t.begin());
        rec[q] = record(t, g);
    }
    float start = 0.0f;
    for (uint32_t i = 0; i < std::min(n, PIECE); i++) start = plus(start, v[i]);
    uint32_t sb = fb(start);
    for (uint32_t g = 1; g < P; g += 32) {                     // combine_records
        const uint32_t cnt = std::min(32u, P - g);
        for (uint32_t pos = 0; pos < cnt;) {
            const uint32_t K = exponent_of(sb);
            Lanes m;
            bool simple[32], live[32];
            for (uint32_t l = 0; l < 32; l++) {
                live[l] = l >= pos && l < cnt;
                simple[l] = live[l] && in_domain(sb) && rec[g + l].kind == BINADE && rec[g + l].K == K;
                m.m[l] = simple[l] ? rec[g + l].m1 : identity();
            }
            const Lanes incl = scanned(m);
            uint32_t s = cnt;
            for (uint32_t l = 0; l < 32 && s == cnt; l++)
                if (live[l] && (!simple[l] || apply(incl.m[l], significand_of(sb)) >= TOP)) s = l;
            if (s > pos) { sb = bits_of(K, apply(incl.m[s - 1], significand_of(sb))); applied += s - pos; }
            if (s >= cnt) break;
            if (!advance(v, g + s, rec[g + s], sb)) return false;
            pos = s + 1;
        }
    }
    out = sb;
    return true;
}

static bool giants = false;
static long tested = 0, fallback = 0, bad = 0;
static void check(const std::vector<float> &v, bool domain = true)
{
    uint32_t got = 0;
    const bool ok = giants ? giant_sum(v, got) : window_sum(v, 0, v.size(), got);
    tested++;
    if (!ok) { fallback++; if (domain) { bad++; std::printf("fallback n=%zu\n", v.size()); } return; }
    float want = 0.0f;
    for (float x : v) want = plus(want, x);
    if (got != fb(want)) { if (bad++ < 10) std::printf("n=%zu got %08x want %08x\n", v.size(), got, fb(want)); }
}

static void rows(uint32_t least, uint32_t span)
{
    auto length = [&]() { return least + static_cast<uint32_t>(nxt() % span); };
    for (int t = 0; t < 200; t++) {                            // log-uniform magnitudes
        std::vector<float> x(length());
        const int s = 1 + nxt() % 40;
        for (auto &f : x) f = static_cast<float>(std::ldexp(1.0 + unit(), -static_cast<int>(nxt() % s) - 10));
        check(x);
    }
    for (int t = 0; t < 80; t++)                               // equal terms: ties, exact powers of two
        check(std::vector<float>(length(), static_cast<float>(std::ldexp(1.0 + (nxt() % 8) / 8.0, -static_cast<int>(nxt() % 30)))));
    for (int t = 0; t < 80; t++) {                             // contributions of about 1/N over small degrees
        std::vector<float> x(length());
        const float base = 1.0f / static_cast<float>(1u << (10 + nxt() % 14));
        for (auto &f : x) f = base / static_cast<float>(1 + nxt() % 64);
        check(x);
    }
    for (int t = 0; t < 80; t++) {                             // growing and shrinking: crossings in most pieces
        std::vector<float> x(length());
        const uint32_t each = x.size() / 100 + 1 + nxt() % 600;
        for (uint32_t i = 0; i < x.size(); i++) x[i] = static_cast<float>(std::ldexp(1.0 + unit(), static_cast<int>(i / each) - 60));
        check(x);
        check(std::vector<float>(x.rbegin(), x.rend()));
    }
    for (int t = 0; t < 60; t++) {                             // zeros through the start and beyond
        std::vector<float> x(length());
        const uint32_t lead = nxt() % x.size();
        for (uint32_t i = 0; i < x.size(); i++) x[i] = i < lead ? 0.0f : static_cast<float>(std::ldexp(1.0 + unit(), -20));
        check(x);
    }
    for (int t = 0; t < 60; t++) {                             // one huge term: later guesses far off
        std::vector<float> x(length(), 1e-6f);
        x[nxt() % x.size()] = 1e3f;
        check(x);
    }
    for (int t = 0; t < 200; t++) {                            // ties and near-ties against the running sum
        std::vector<float> x(length());
        float s = 0.0f;
        for (auto &f : x) {
            f = static_cast<float>(std::ldexp(1.0 + unit(), -static_cast<int>(nxt() % 30)));
            if (s > 0.0f && nxt() % 2) {
                const int sh = nxt() % 20;
                double h = std::ldexp(nxt() % (1u << sh) + 0.5, static_cast<int>(exponent_of(fb(s))) - 150);
                if (nxt() % 3 == 0) h = std::nextafter(h, 0.0);
                f = static_cast<float>(h);
            }
            s = plus(s, f);
        }
        check(x);
    }
    for (int t = 0; t < 20; t++) {                             // subnormal terms stay inside the chains' domain
        std::vector<float> x(length(), 1.0f);
        x[nxt() % x.size()] = 1e-40f;
        check(x);
    }
    for (const float f : {-1.0f, static_cast<float>(INFINITY), static_cast<float>(NAN)}) {   // reported, never summed wrongly
        std::vector<float> x(least + 5000, 1.0f);
        x[least + 4000] = f;
        check(x, false);
    }
    check(std::vector<float>(least + 5000, 3e38f), false);
}

int main(int argc, char **argv)
{
    giants = std::atoi(argv[1]) != 0;
    wrong = std::atoi(argv[2]);
    if (giants) {
        rows(512, 1700);                                       // from the shortest giant row
        rows(4097, 50000);
    } else {
        for (const uint32_t l : {8u, 16u}) { L = l; rows(1024, 9000); }
    }
    std::printf("tested %ld fallback %ld bad %ld applied %ld crossed %ld exact %ld\n", tested, fallback, bad, applied, crossed, exact);
    return bad ? 1 : 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("pieces")
    (d / "pieces.cpp").write_text(CHECK)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{CSRC}", str(d / "pieces.cpp"), "-o",
                    str(d / "pieces")], check=True)
    return d / "pieces"


@pytest.mark.parametrize("giants,wrong", [(0, 0), (1, 0), (1, 1)], ids=["windows", "giant rows", "giant rows, wrong guesses"])
def test_sums_match_the_loop(program, giants, wrong):
    out = subprocess.run([str(program), str(giants), str(wrong)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout[-3000:]
    print(out.stdout)
    said = out.stdout.split()
    n = {said[i]: int(said[i + 1]) for i in range(0, 12, 2)}
    assert n["bad"] == 0 and n["fallback"] == 8                # the terms out of the domain, at both lengths
    if giants:
        assert n["applied"] > n["exact"] // (4 if wrong else 1) and n["crossed"] > 0


def test_the_constants_are_the_kernels():
    """The sizes the check above is written for."""
    pr, warp = (CSRC / "pagerank.cu").read_text(), (CSRC / "bw_seqsum_warp.cuh").read_text()
    assert "constexpr uint32_t SEG_EDGES = 512" in pr
    assert "constexpr uint32_t PIECE_L = SEG_EDGES / 32" in pr
    assert "constexpr uint32_t START_PIECES = 1" in pr and "constexpr uint32_t GIANT_LEAST = 512" in pr
    assert "constexpr uint32_t SERIAL_TERMS = 1024" in warp
