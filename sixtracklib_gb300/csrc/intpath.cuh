// intpath.cuh -- parts of the element maps on the integer pipes, with the
// FP64 arithmetic's bits.
//
// A GB300 scheduler issues one FP64 warp instruction every 64 to 76 cycles
// (measured: 64 alone on its SM, 76 with all four schedulers at it) and an
// integer or FP32 one every cycle or two, so the time of the tracking
// kernel is its FP64 instruction count.  The functions here compute a
// result that a few rounded FP64 operations define -- in fixed point, to
// more bits than the result has -- and check that the rounding cannot go
// the other way: every rounding error of the FP64 sequence and every
// truncation here is bounded, and a value closer to a rounding boundary
// than that bound reports failure, on which the caller runs the FP64
// sequence itself.  What they return is bit-identical to that sequence.
//
// Host-compilable: the bounds are checked on the CPU as well.
#pragma once

#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#define STG_HD __host__ __device__ __forceinline__
#else
#define STG_HD inline
#endif

namespace stg {

STG_HD uint64_t bits_of(double v)
{
#if defined(__CUDA_ARCH__)
    return (uint64_t)__double_as_longlong(v);
#else
    uint64_t w;
    std::memcpy(&w, &v, 8);
    return w;
#endif
}

STG_HD double from_bits(uint64_t w)
{
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)w);
#else
    double v;
    std::memcpy(&v, &w, 8);
    return v;
#endif
}

STG_HD double from_words(uint32_t hi, uint32_t lo) { return from_bits(((uint64_t)hi << 32) | lo); }

// Low word of (hi : lo) << n, 0 < n < 32, upper half.
STG_HD uint32_t shl_hi(uint32_t hi, uint32_t lo, int n)
{
#if defined(__CUDA_ARCH__)
    return __funnelshift_l(lo, hi, n);
#else
    return (hi << n) | (lo >> (32 - n));
#endif
}

// (hi : lo) >> min(n, 32), lower word.
STG_HD uint32_t shr_lo_clamp(uint32_t hi, uint32_t lo, uint32_t n)
{
#if defined(__CUDA_ARCH__)
    return __funnelshift_rc(lo, hi, n);
#else
    return n >= 32 ? hi : (uint32_t)((((uint64_t)hi << 32) | lo) >> n);
#endif
}

// v >> n, 0 for n >= 32.
STG_HD uint32_t shr_clamp(uint32_t v, uint32_t n)
{
#if defined(__CUDA_ARCH__)
    uint32_t r;
    asm("shr.u32 %0, %1, %2;" : "=r"(r) : "r"(v), "r"(n));
    return r;
#else
    return n >= 32 ? 0u : v >> n;
#endif
}

STG_HD int count_leading_zeros(uint32_t v)
{
#if defined(__CUDA_ARCH__)
    return __clz((int)v);
#else
    return v ? __builtin_clz(v) : 32;
#endif
}

// v 2^-53 as a double (exact), |v| < 2^32: normalised on the integer pipe.
STG_HD double scaled_53(int64_t v)
{
    int64_t const s = v >> 63;
    uint32_t const m = (uint32_t)((v ^ s) - s);
    int const n = count_leading_zeros(m);
    uint32_t const t = m << (n & 31);  // m = 0 stays 0
    // t 2^-31 2^(-22 - n): biased exponent 1001 - n, less the implicit bit
    // that t >> 11 adds to it
    uint32_t const hi = ((uint32_t)(1000 - n) << 20) + (t >> 11);
    return from_words((m ? hi : 0u) | ((uint32_t)(s >> 32) & 0x80000000u), t << 21);
}

STG_HD bool below_2_32(int64_t v)
{
    uint32_t const h = (uint32_t)((uint64_t)v >> 32);
    return h == 0u || (h == 0xFFFFFFFFu && (uint32_t)v != 0u);
}

// The same for |v| < 2^51: 0.75 + v 2^-53 formed in the significand, one
// FP64 subtraction (exact).
STG_HD double scaled_53_large(int64_t v)
{
    return from_bits(0x3FE8000000000000ull + (uint64_t)v) - 0.75;
}

// (rvv - 1) 2^53 of an rvv within 2^-10 of 1 (exact), and the limit on
// 2 |high word| of xp and yp for drift_slip: 2^-7, or nothing for another
// rvv.
STG_HD int64_t slip_rvv(double rvv)
{
    int64_t const w = (int64_t)(bits_of(rvv) - 0x3FF0000000000000ull);
    return w < 0 ? w : 2 * w;
}

STG_HD uint32_t slip_limit(double rvv)
{
    // [1 - 2^-10, 1 + 2^-10]: NaN, inf, negative and far values fail
    uint64_t const w = bits_of(rvv) - 0x3FEFF80000000000ull;
    return w <= 0x3FF0040000000000ull - 0x3FEFF80000000000ull ? 0x7F000000u : 0u;
}

// The drift's path-length slip rvv - (1 + (xp^2 + yp^2) / 2) with every
// operation rounded (with or without the sum's fma): u = RN(1 + t / 2) is
// 1 + k 2^-52 with k = RN(T), T = t 2^51, and rvv - u is exact.  T is formed
// in fixed point with 25 fraction bits from |xp|, |yp| in units of 2^-70:
// truncations lose less than 6 units of 2^-25, and the FP64 sequence's own
// roundings of t move it by at most 2^-52 T < 2049 units (T < 2^38 for
// |xp|, |yp| < 2^-7).  A T within 2064 units of a half is reported as
// undecided: once in 8,000.  Six of the drift's 14 (exact) and four of its 9
// (fast) FP64 instructions in about 45 integer ones: one turn of 1M polar-grid
// protons on the 20,000-element ring 263.4 -> 221.3 ms (fast), of 131,072
// Gaussian ones 137.3 -> 123.5 ms (exact); 10,000 protons x 100 turns of the
// 258-element FODO ring 17.6 -> 15.5 ms (exact).
STG_HD bool drift_slip(double xp, double yp, int64_t rvv53, uint32_t limit, int64_t *slip53)
{
    uint64_t const wx = bits_of(xp), wy = bits_of(yp);
    uint32_t const hx = (uint32_t)(wx >> 32), lx = (uint32_t)wx;
    uint32_t const hy = (uint32_t)(wy >> 32), ly = (uint32_t)wy;
    uint32_t const ax = hx << 1, ay = hy << 1;
    // |xp| 2^70: the significand with its leading bit at bit 63, shifted by
    // 1016 - exponent (zeros and subnormals shift out to < 2^32)
    uint32_t const sx = 1016u - (ax >> 21), sy = 1016u - (ay >> 21);
    uint32_t const mx = shl_hi(hx, lx, 11) | 0x80000000u, my = shl_hi(hy, ly, 11) | 0x80000000u;
    uint32_t const xh = shr_clamp(mx, sx), yh = shr_clamp(my, sy);
    uint32_t const xl = shr_lo_clamp(mx, lx << 11, sx), yl = shr_lo_clamp(my, ly << 11, sy);
    uint64_t const a = (uint64_t)xh * xh + (uint64_t)yh * yh;
    uint64_t const b = (uint64_t)xh * xl + (uint64_t)yh * yl;
    uint64_t const r = a + (b >> 31) + (1ull << 24);
    *slip53 = rvv53 - (int64_t)((r >> 24) & ~1ull);
    uint32_t const f = (uint32_t)r & 0x1FFFFFFu;
    return (f - 2064u) < (0x2000000u - 2u * 2064u) && ax < limit && ay < limit;
}

// RN(a b) on the integer pipes (34 instructions, about 55 issue cycles against
// the 76 of an FP64 multiplication that fills its pipe): a's significand with
// its leading bit at bit 63 times b's 53 bits, four 32 x 32 products; the
// product's upper 64 bits hold the result's significand with the rounding
// bit below.  False -- use the FP64 instruction -- for operands or results
// far out or not finite, and on an exact half in the next 32 bits.
STG_HD bool mul_rn(double a, double b, double *out)
{
    uint64_t const wa = bits_of(a), wb = bits_of(b);
    uint32_t const ha = (uint32_t)(wa >> 32), la = (uint32_t)wa;
    uint32_t const hb = (uint32_t)(wb >> 32), lb = (uint32_t)wb;
    uint32_t const ea = (ha << 1) >> 21, eb = (hb << 1) >> 21;
    uint32_t const ah = shl_hi(ha, la, 11) | 0x80000000u, al = la << 11;
    uint32_t const bh = (hb & 0xFFFFFu) | 0x100000u;
    uint64_t const ll = (uint64_t)al * lb;
    uint64_t const t = (uint64_t)al * bh + (ll >> 32);
    uint64_t const u = (uint64_t)ah * lb + (uint32_t)t;
    uint64_t const h = (uint64_t)ah * bh + (t >> 32) + (u >> 32);  // [2^51, 2^53)
    uint32_t const f1 = (uint32_t)u, f0 = (uint32_t)ll;            // the 64 bits below
    uint32_t const hh = (uint32_t)(h >> 32), hl = (uint32_t)h;
    bool const lower = (hh >> 20) == 0u;  // 52 bits: one more from below
    uint32_t const rh = lower ? shl_hi(hh, hl, 1) : hh, rl = lower ? shl_hi(hl, f1, 1) : hl;
    uint32_t const f = lower ? shl_hi(f1, f0, 1) : f1;
    uint64_t const r = (((uint64_t)rh << 32) | rl) + (f >> 31);
    // rh's leading bit adds one to the exponent field
    uint32_t const e = ea + eb - (lower ? 1024u : 1023u);
    uint32_t const sign = (ha ^ hb) & 0x80000000u;
    bool const zero = ((ha << 1) | la) == 0u;
    uint64_t const v = r + ((uint64_t)(e << 20) << 32);
    *out = from_bits(zero ? (uint64_t)sign << 32 : v | ((uint64_t)sign << 32));
    bool const fine = f != 0x80000000u && ea - 64u < 1900u && e - 64u < 1900u;
    return (fine || zero) && eb - 64u < 1900u;
}

}  // namespace stg
