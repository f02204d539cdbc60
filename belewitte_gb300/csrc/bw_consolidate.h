// The reference's PageRank consolidation adds a double base term to a float
// product and rounds to float:
//     new_rank = (float)(((1.0 - d) / N) + (double)(d * acc))
// (pagerank/pagerank.cu:132).  GB300 runs FP64 instructions at a small
// fraction of the FP32 rate, so this header performs the same two IEEE
// round-to-nearest-even steps -- double addition, then conversion to float --
// with 64-bit integer arithmetic.  Valid for a positive normal double B and a
// float x >= 0 (zero or normal); the result is bit-identical to the FP64 path
// (checked exhaustively on edge cases and randomly in tests).
#pragma once
#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define BWC_HD __host__ __device__ __forceinline__
#else
#define BWC_HD inline
#endif

namespace bwcons {

// Unpacked positive double: value = m * 2^(e - 1075), m in [2^52, 2^53).
struct Unpacked {
    uint64_t m;
    int32_t e;
};

BWC_HD Unpacked unpack_double(uint64_t bits)
{
    return Unpacked{(bits & ((uint64_t(1) << 52) - 1)) | (uint64_t(1) << 52), static_cast<int32_t>((bits >> 52) & 0x7ff)};
}

// fl32(fl64(B + x)) for B = double with bits `b_bits` (positive, normal) and
// x >= 0 normal float or zero.  `ok` is false for inputs outside that domain
// (subnormal x or a result outside the normal float range).
BWC_HD uint32_t add_round_bits(uint64_t b_bits, uint32_t x_bits, bool &ok)
{
    ok = true;
    const Unpacked B = unpack_double(b_bits);
    uint64_t M;
    int32_t E;
    const uint32_t ex = (x_bits >> 23) & 0xff, fx = x_bits & 0x7fffff;
    if ((x_bits & 0x7fffffff) == 0) {
        M = B.m;
        E = B.e;
    } else {
        if (ex == 0 || ex == 0xff || (x_bits >> 31)) { ok = false; return 0; }
        const Unpacked X{(static_cast<uint64_t>(fx) | (uint64_t(1) << 23)) << 29, static_cast<int32_t>(ex) - 127 + 1023};
        const Unpacked &hi = B.e >= X.e ? B : X;
        const Unpacked &lo = B.e >= X.e ? X : B;
        const uint32_t d = static_cast<uint32_t>(hi.e - lo.e);
        const uint64_t a = hi.m << 10;                    // 63 bits: 53 significant + 10 guard
        const uint64_t full = lo.m << 10;
        uint64_t b;
        bool sticky;
        if (d >= 63) {
            b = 0;
            sticky = full != 0;
        } else {
            b = full >> d;
            sticky = d ? (full & ((uint64_t(1) << d) - 1)) != 0 : false;
        }
        uint64_t s = a + b;
        int32_t e = hi.e;
        if (s >> 63) {                                    // carry: renormalise
            sticky = sticky || (s & 1);
            s >>= 1;
            e += 1;
        }
        // round the 53-bit significand (bits 62..10) to nearest even
        const uint64_t low = s & 0x3ff, half = 0x200;
        const uint64_t lsb = (s >> 10) & 1;
        const bool up = low > half || (low == half && (sticky || lsb));
        M = (s >> 10) + (up ? 1 : 0);
        if (M >> 53) {
            M >>= 1;
            e += 1;
        }
        E = e;
        if (E >= 0x7ff) { ok = false; return 0; }
    }
    // double (M, E) -> float, round to nearest even on the 29 dropped bits
    const uint64_t low29 = M & ((uint64_t(1) << 29) - 1), half29 = uint64_t(1) << 28;
    const uint64_t lsb = (M >> 29) & 1;
    uint64_t F = (M >> 29) + ((low29 > half29 || (low29 == half29 && lsb)) ? 1 : 0);
    int32_t e32 = E - 1023 + 127;
    if (F >> 24) {
        F >>= 1;
        e32 += 1;
    }
    if (e32 <= 0 || e32 >= 0xff) { ok = false; return 0; }
    return (static_cast<uint32_t>(e32) << 23) | static_cast<uint32_t>(F & 0x7fffff);
}

// The same result from about twenty float instructions for nearly every x;
// `ok` is false when they do not decide it (add_round_bits then does).
//
// With hi = fl32(B) and lo = fl32(B - hi), s + e = hi + x exactly (Knuth's
// two-sum), t = fl32(e + lo) and r + d = s + t exactly (Dekker's fast
// two-sum), r = fl32(s + t).  What t and lo dropped is below 2^-23 ulp(s)
// each (|e| and |lo| are at most half an ulp of s), and the double addition
// that the reference rounds by moves the sum by less than 2^-28 ulp(s): so
// while |d| stays 2^-19 of half an ulp of r away from the rounding boundary,
// and r is no power of two, where the boundary below is nearer, rounding B + x
// once or twice gives r.  Needs hi >= 2^-90 (split_base).
BWC_HD float f32_add(float a, float b)
{
#if defined(__CUDA_ARCH__)
    return __fadd_rn(a, b);
#else
    return a + b;
#endif
}
BWC_HD uint32_t f32_bits(float f)
{
#if defined(__CUDA_ARCH__)
    return __float_as_uint(f);
#else
    uint32_t b;
    memcpy(&b, &f, sizeof b);
    return b;
#endif
}
BWC_HD float f32_of(uint32_t b)
{
#if defined(__CUDA_ARCH__)
    return __uint_as_float(b);
#else
    float f;
    memcpy(&f, &b, sizeof f);
    return f;
#endif
}
struct Base {
    float hi, lo;
};
// hi = 0 (never decided) for a base that is not positive or too small.
BWC_HD Base split_base(double base)
{
    if (!(base >= 0x1p-90 && base <= 0x1p60)) return Base{0.0f, 0.0f};
    const float hi = static_cast<float>(base);
    return Base{hi, static_cast<float>(base - static_cast<double>(hi))};
}
BWC_HD float add_round_split(Base b, float x, bool &ok)
{
    const float s = f32_add(b.hi, x), xs = f32_add(s, -b.hi);
    const float e = f32_add(f32_add(b.hi, -f32_add(s, -xs)), f32_add(x, -xs));
    const float t = f32_add(e, b.lo), r = f32_add(s, t);
    const float d = f32_add(t, -f32_add(r, -s));
    const uint32_t rb = f32_bits(r);
    // half an ulp of r less 2^-19 of it: (1 - 2^-19) 2^(k - 24)
    const float limit = f32_of((rb & 0x7f800000u) - (24u << 23) - 32u);
    ok = b.hi > 0.0f && x >= 0.0f && r < 0x1p100f && (d < 0.0f ? -d : d) < limit && (rb & 0x7fffffu) != 0u;
    return r;
}

}  // namespace bwcons
