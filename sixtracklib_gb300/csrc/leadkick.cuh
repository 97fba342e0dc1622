// leadkick.cuh -- the kick of a multipole whose quadrupole term leads, with
// the FP64 evaluation's bits and a quarter of its FP64 instructions.
//
// In P(z) = b_1 z + z^2 (b_2 + b_3 z + ...) of a quadrupole with multipole
// errors the bracket is 10^-3 or less of b_1, so of the FP64 sequences that
// define the kick (Horner in the exact policy, Goertzel in the fast one) all
// steps but the last see it only through the last few bits of
// u_1 = RN(b_1 + small) and through small corrections to u_1 x and u_1 y.
// Here the bracket is evaluated in FP32 -- pairs of floats (48 bits) for the
// terms that matter, single floats for the rest -- and u_1 is formed by an
// integer addition to b_1's significand.  Every step carries a bound on its
// own error and on the rounding errors of the FP64 sequence it replaces
// (computed per element by the lattice compiler, lead_block); where the
// bound leaves a rounding open, the caller runs the FP64 sequence.
//
// FP64 instructions per kick of order n: fast 5 instead of 2n + 5, exact 4
// instead of 7n - 3 (the corrections added on the significands of u_1 x and
// u_1 y); about 130 FP32 and integer ones issue in their shadow.
// Measured on the 20,000-element ring (orders 1 to 10): 1M polar-grid
// protons, one turn, fast 222.9 -> 130.4 ms; 131,072 Gaussian ones, exact
// 99.6 -> 34.5 ms.  For particles at 1 mm 0.02 % of the kicks are left to
// the FP64 sequence.
#pragma once

#include "intpath.cuh"

#include <cmath>

namespace stg {

// ------------------------------------------------- FP32, never contracted
STG_HD float f_of(uint32_t w)
{
#if defined(__CUDA_ARCH__)
    return __uint_as_float(w);
#else
    float v;
    std::memcpy(&v, &w, 4);
    return v;
#endif
}

STG_HD uint32_t w_of(float v)
{
#if defined(__CUDA_ARCH__)
    return __float_as_uint(v);
#else
    uint32_t w;
    std::memcpy(&w, &v, 4);
    return w;
#endif
}

#if defined(__CUDA_ARCH__)
STG_HD float fadd(float a, float b) { return __fadd_rn(a, b); }
STG_HD float fsub(float a, float b) { return __fsub_rn(a, b); }
STG_HD float fmul(float a, float b) { return __fmul_rn(a, b); }
STG_HD float ffma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
STG_HD int32_t frint(float a) { return __float2int_rn(a); }
STG_HD float fofu(uint32_t a) { return __uint2float_rn(a); }
STG_HD float fmaxabs(float a, float b) { return fmaxf(fabsf(a), fabsf(b)); }
STG_HD float fabs_(float a) { return fabsf(a); }
#else
STG_HD float fadd(float a, float b) { return a + b; }
STG_HD float fsub(float a, float b) { return a - b; }
STG_HD float fmul(float a, float b) { return a * b; }
STG_HD float ffma(float a, float b, float c) { return std::fmaf(a, b, c); }
STG_HD int32_t frint(float a) { return (int32_t)std::lrintf(a); }
STG_HD float fofu(uint32_t a) { return (float)a; }
STG_HD float fmaxabs(float a, float b) { return std::fmax(std::fabs(a), std::fabs(b)); }
STG_HD float fabs_(float a) { return std::fabs(a); }
#endif

// h + l, |l| at most a few 2^-23 |h|
struct FPair {
    float h, l;
};

// A double of magnitude below 1 as a pair: h its first 24 bits, l the other
// 29 rounded to 24 (2^-48 relative).  Below 2^-66 l is 0, below 2^-90
// (zeros, subnormals) h as well.
STG_HD FPair split(double v)
{
    uint64_t const w = bits_of(v);
    uint32_t const hi = (uint32_t)(w >> 32), lo = (uint32_t)w;
    uint32_t const sign = hi & 0x80000000u;
    // exponent re-biased in place: 896 = 1023 - 127, of which the low nine
    // exponent bits keep 384
    uint32_t const m = shl_hi(hi, lo, 3) - (384u << 23);
    uint32_t const h = (hi << 1) < (933u << 21) ? 0u : ((m & 0x7FFFFFFFu) | sign);
    // l = (low 29 bits) 2^(e - 52)
    uint32_t const scale =
        (hi << 1) < (957u << 21) ? 0u : (((m & 0x7F800000u) - (52u << 23)) | sign);
    return FPair{f_of(h), fmul(fofu(lo & 0x1FFFFFFFu), f_of(scale))};
}

// a + b = h + l exactly
STG_HD FPair two_sum(float a, float b)
{
    float const h = fadd(a, b);
    float const t = fsub(h, a);
    return FPair{h, fadd(fsub(a, fsub(h, t)), fsub(b, t))};
}

STG_HD FPair mul(FPair a, FPair b)
{
    float const p = fmul(a.h, b.h);
    float e = ffma(a.h, b.h, -p);
    e = ffma(a.h, b.l, e);
    return FPair{p, ffma(a.l, b.h, e)};
}

// A float as a double, 0 below the normal range.
STG_HD double as_double(float v)
{
    uint32_t const w = w_of(v), a = w & 0x7FFFFFFFu;
    return a < 0x00800000u ? 0.0 : from_words(((a >> 3) + 0x38000000u) | (w & 0x80000000u), w << 29);
}

// Doubles at or outside both ends of [h + l - d, h + l + d].  l is up to 2^28
// units of the last of h's 53 bits and l -+ d is rounded to 24 bits, so d has to
// hold 8 such units (2^-49 of h) more than the error it bounds: the 5 % that
// lead_block adds to bounds of 2^-43 and more do, as does what sc_pair_kick's
// bound leaves over.
STG_HD void double_bounds(FPair v, float d, double *lo_v, double *hi_v)
{
    float const h = fadd(v.h, v.l), l = fsub(v.l, fsub(h, v.h));
    uint32_t const w = w_of(h);
    uint32_t const sign = w & 0x80000000u, e = w & 0x7F800000u;
    // +-2^(52 - exponent): l in units of the last of 53 bits
    float const s = f_of((0x99000000u - e) | sign);
    if (e >= (52u << 23) && fabs_(fmul(d, s)) < 0x1p29f && (w & 0x7FFFFFu) != 0u) {
        int32_t const a = frint(fmul(fsub(l, d), s)), b = frint(fmul(fadd(l, d), s));
        uint64_t const m =
            ((uint64_t)(((w & 0x7FFFFFFFu) >> 3) + 0x38000000u) << 32) | (w << 29);
        uint64_t const sg = (uint64_t)sign << 32;
        *lo_v = from_bits((m + (uint64_t)(int64_t)a) | sg);
        *hi_v = from_bits((m + (uint64_t)(int64_t)b) | sg);
        return;
    }
    // a bound that is not small against h, a value below 2^-75, or a power of
    // two (whose l may lie in a binade of finer units): to single precision
    float const wide = (w << 1) == 0u && d == 0.0f
                           ? 0.0f
                           : fadd(fadd(fmul(d, 1.0078125f), fmul(fabs_(h), 0x1p-22f)), 0x1p-100f);
    *lo_v = as_double(fsub(h, wide));
    *hi_v = as_double(fadd(h, wide));
}

// Nearest integer of (h + l) with |h| < 2^42, and whether h + l stays more
// than d away from every half.
STG_HD bool nearest(FPair v, float d, int64_t *out)
{
    constexpr float kMagic = 12582912.0f;  // 1.5 2^23
    float const m1 = ffma(v.h, 0x1p-20f, kMagic);
    float const f1 = fsub(m1, kMagic);
    float const r1 = ffma(f1, -0x1p20f, v.h);  // |r1| <= 2^19, exact
    float const m2 = fadd(r1, kMagic);
    float const r2 = fsub(r1, fsub(m2, kMagic));  // |r2| <= 1/2, exact
    float const m3 = fadd(fadd(r2, v.l), kMagic);
    float const frac = fadd(fsub(v.l, fsub(m3, kMagic)), r2);
    int32_t const i1 = (int32_t)(w_of(m1) - 0x4B400000u);
    int32_t const i2 = (int32_t)(w_of(m2) + w_of(m3) - 2u * 0x4B400000u);
    *out = (int64_t)i1 * (1 << 20) + i2;
    return fadd(fabs_(frac), d) < 0.49999f;
}

// ---------------------------------------------------------------- the record
// Words of the lead block that follows the coefficients bal[0..2n+1]:
//   0: {1 / ulp(b_1) with b_1's sign, limit on the high words of |x|, |y|}
//   1: {k, k'}: z times the bracket is known to |z| (k + k' s) ulp(b_1)
//   2: {c, c'}: the bracket is known to c + c' s
//   3: {b_2 as a pair}   4: {b_3 as a pair}   5...: {b_4, b_5}, {b_6, b_7} ...
// (first of each pair in the low half; |z| = |x| + |y|, s = x^2 + y^2)
STG_HD int lead_words(int order) { return 5 + (order >= 4 ? (order - 2) / 2 : 0); }

struct LeadTerms {
    FPair x, y, s, g2, g3;
};

STG_HD float low_f(uint64_t w) { return f_of((uint32_t)w); }
STG_HD float high_f(uint64_t w) { return f_of((uint32_t)(w >> 32)); }

// The bracket's Goertzel values g_2 = b_2 + 2x g_3 - s g_4 and g_3, with
// s = x^2 + y^2: z (b_2 + b_3 z + ...) = z g_2 - s g_3.
STG_HD LeadTerms lead_terms(double x, double y, const uint64_t *blk, int order)
{
    LeadTerms t;
    t.x = split(x);
    t.y = split(y);
    float const px = fmul(t.x.h, t.x.h), py = fmul(t.y.h, t.y.h);
    float const ex = ffma(fadd(t.x.h, t.x.h), t.x.l, ffma(t.x.h, t.x.h, -px));
    float const ey = ffma(fadd(t.y.h, t.y.h), t.y.l, ffma(t.y.h, t.y.h, -py));
    t.s = two_sum(px, py);
    t.s.l = fadd(t.s.l, fadd(ex, ey));
    float const r1 = fadd(t.x.h, t.x.l), r = fadd(r1, r1), s = fadd(t.s.h, t.s.l);
    float g4 = 0.0f, g5 = 0.0f;  // g_k, g_(k+1) from the top
    for (int k = order; k >= 4; --k) {
        uint64_t const w = blk[5 + (k - 4) / 2];
        float const b = (k & 1) ? high_f(w) : low_f(w);
        float const g = ffma(r, g4, ffma(-s, g5, b));
        g5 = g4;
        g4 = g;
    }
    t.g3 = two_sum(low_f(blk[4]), ffma(r, g4, -fmul(s, g5)));
    t.g3.l = fadd(t.g3.l, high_f(blk[4]));
    FPair const rg = mul(FPair{fadd(t.x.h, t.x.h), fadd(t.x.l, t.x.l)}, t.g3);
    FPair const sum = two_sum(low_f(blk[3]), rg.h);
    float const l = ffma(-s, g4, fadd(fadd(sum.l, rg.l), high_f(blk[3])));
    t.g2.h = fadd(sum.h, l);  // |l| < |sum.h| but for a cancelling bracket,
    t.g2.l = fsub(l, fsub(t.g2.h, sum.h));  // whose bound is that of its terms
    return t;
}

STG_HD bool lead_in_range(double x, double y, const uint64_t *blk)
{
    uint32_t const ax = (uint32_t)(bits_of(x) >> 32) & 0x7FFFFFFFu;
    uint32_t const ay = (uint32_t)(bits_of(y) >> 32) & 0x7FFFFFFFu;
    uint32_t const lim = (uint32_t)(blk[0] >> 32);
    // the larger one at least 2^-40 (the floor of the bounds)
    return ax < lim && ay < lim && (ax >= 0x3D700000u || ay >= 0x3D700000u);
}

// Whether y is zero or split() keeps all of its bits (2^-66 and above).  The
// corrections of the exact policy are proportional to y, and with momenta of
// y's size their last bits count: below, the pair's truncation (2^-24 of y, from
// 2^-90 down all of it) is outside the bound on them.
STG_HD bool lead_y_whole(double y)
{
    uint64_t const a = bits_of(y) << 1;
    return a == 0u || a >= 957ull << 53;
}

STG_HD float lead_error(const LeadTerms &t, uint64_t k)
{
    return fmul(fadd(fabs_(t.x.h), fabs_(t.y.h)), ffma(high_f(k), t.s.h, low_f(k)));
}

// u_1 = RN(b_1 + Re(z bracket)) of the exact policy, the corrections v_1 y
// and v_1 x, v_1 = Im(z bracket), and the bounds on these: 0 only where y is,
// so that a correction lost below the floats' range is not taken for a known
// zero.  Returns whether u_1 is decided and the bounds hold.
STG_HD bool lead_exact(double x, double y, const uint64_t *bal, int order, double *u1,
                       FPair *e1, FPair *e2, float *bound)
{
    const uint64_t *const blk = bal + 2 * order + 2;
    LeadTerms const t = lead_terms(x, y, blk, order);
    FPair const a = mul(t.x, t.g2), b = mul(t.s, t.g3), v = mul(t.y, t.g2);
    FPair re = two_sum(a.h, -b.h);
    re.l = fadd(re.l, fsub(a.l, b.l));
    float const scale = low_f(blk[0]);
    int64_t i;
    bool const ok =
        nearest(FPair{fmul(re.h, scale), fmul(re.l, scale)}, lead_error(t, blk[1]), &i);
    *u1 = from_bits(bal[2] + (uint64_t)i);
    *e1 = mul(v, t.y);
    *e2 = mul(v, t.x);
    float const d = fmul(fabs_(t.y.h), ffma(high_f(blk[2]), t.s.h, low_f(blk[2])));
    float const least = t.y.h == 0.0f ? 0.0f : 0x1p-149f;
    bound[0] = ffma(fabs_(t.y.h), d, least);
    bound[1] = ffma(fabs_(t.x.h), d, least);
    return ok && lead_y_whole(y);
}

// RN(k + e), e known to +-d, formed on k's significand; false where the
// rounding is open or the sum leaves k's binade.
STG_HD bool nearest_sum(double k, FPair e, float d, double *sum)
{
    uint64_t const w = bits_of(k);
    uint32_t const hi = (uint32_t)(w >> 32);
    // e in units of k's last place, with k's sign: times +-2^(1075 - exponent)
    uint32_t const ex = (hi >> 20) & 0x7FFu;
    uint32_t const sb = ((1202u - ex) << 23) | (hi & 0x80000000u);
    float const s = f_of(sb);
    int64_t i;
    // k between 2^-74 and 2^49, |e| below 2^41 of its last places
    bool const fine = ex - 949u < 123u && fabs_(fmul(e.h, s)) < 0x1p41f;
    bool const ok = nearest(FPair{fmul(e.h, s), fmul(e.l, s)}, fabs_(fmul(d, s)), &i);
    uint64_t const r = w + (uint64_t)i;
    *sum = from_bits(r);
    return fine && ok && ((r ^ w) >> 52) == 0;
}

// c_1 = RN(RN(b_1 - s g_3) + 2x g_2) of the fast policy's Goertzel form, and
// bounds on s g_2.
STG_HD bool lead_fast(double x, double y, const uint64_t *bal, int order, double *c1, double *w)
{
    const uint64_t *const blk = bal + 2 * order + 2;
    LeadTerms const t = lead_terms(x, y, blk, order);
    FPair const a = mul(t.x, t.g2), b = mul(t.s, t.g3);
    float const scale = low_f(blk[0]);
    float const d = lead_error(t, blk[1]);
    float const scale2 = fadd(scale, scale);
    int64_t ia, ib;
    bool const oka = nearest(FPair{fmul(a.h, scale2), fmul(a.l, scale2)}, d, &ia);
    bool const okb = nearest(FPair{fmul(b.h, scale), fmul(b.l, scale)}, d, &ib);
    *c1 = from_bits(bal[2] + (uint64_t)(ia - ib));
    // (the bound never 0, as above)
    double_bounds(mul(t.s, t.g2),
                  ffma(t.s.h, ffma(high_f(blk[2]), t.s.h, low_f(blk[2])), 0x1p-149f), &w[0],
                  &w[1]);
    return oka && okb;
}

// ------------------------------------------------------------ host: the block
// Build the lead block of a straight multipole of order n >= 2 with
// coefficients bal[0..2n+1], none of them skew and no dipole term; false
// where the quadrupole term does not lead.  The bounds: g+_k, the Goertzel
// recurrence on absolute values at |x|, |y| <= R, bounds every value formed;
// the errors follow from the same recurrence with each step's roundings as
// its source terms: P those of the pairs and of the FP64 sequence, S those
// of the single-float tail, which enter with at least two powers of the
// coordinates (so that S / R^2 times x^2 + y^2 bounds them inside R).  R is
// the largest power of two from 2^-5 m down to 2^-9 m at which u_1 is
// undecided at the edge of the range at most every fourth time.
inline bool lead_block(const uint64_t *bal, int order, uint64_t *blk)
{
    auto coef = [&](int k) { return from_bits(bal[2 * k]); };
    auto words = [](double lo, double hi) {
        return (uint64_t)w_of((float)lo) | ((uint64_t)w_of((float)hi) << 32);
    };
    if (order < 2 || order > 64) return false;
    for (int k = 0; k <= order; ++k)
        if (bal[2 * k + 1] != 0 || !(std::fabs(coef(k)) < 0x1p20)) return false;
    double const b1 = std::fabs(coef(1));
    if (bal[0] != 0 || !(b1 > 0x1p-40 && b1 < 0x1p10)) return false;
    int ex;
    (void)std::frexp(b1, &ex);  // 2^(ex - 1) <= b1 < 2^ex
    double const inv_ulp = std::ldexp(1.0, 53 - ex);
    constexpr double u = 0x1p-24, u64 = 0x1p-53, tiny = 0x1p-120;
    for (int re = -5; re >= -9; --re) {
        double const R = std::ldexp(1.0, re), r = 2 * R, s = 2 * R * R;
        double G[2] = {0, 0}, P[2] = {0, 0}, S[2] = {0, 0};  // k + 1, k + 2
        for (int k = order; k >= 2; --k) {
            double const tail = r * G[0] + s * G[1];
            double const g = std::fabs(coef(k)) + tail;
            double p = r * P[0] + s * P[1] + 8 * u64 * g + tiny, q = r * S[0] + s * S[1];
            // r and s rounded, the coefficient rounded, two fma
            if (k >= 4) q += 3.2 * u * g;
            // the tail's product and fma; the sum with the pair b_3 exact
            if (k == 3) q += 3.2 * u * tail, p += 0x1p-46 * g;
            // 2x g_3 in pairs; s g_4 in single floats
            if (k == 2) q += 3.2 * u * s * G[1], p += 0x1p-45 * r * G[0] + 0x1p-46 * g;
            G[1] = G[0], G[0] = g;
            P[1] = P[0], P[0] = p;
            S[1] = S[0], S[0] = q;
        }
        if (!(G[0] > 0x1p-60)) return false;
        // 2x g_2 and s g_3 <= |z| 1.5 R g_3, each per |z|
        double const cp = P[0] + 0x1p-43 * G[0], cs = S[0] / (R * R);
        double const kp = (2 * cp + 1.5 * R * (P[1] + 0x1p-44 * G[1])) * inv_ulp;
        double const ks = (2 * S[0] + 1.5 * R * S[1]) * inv_ulp / (R * R);
        double const tmax = 1.01 * (r * G[0] + s * G[1]);
        if (!(2 * R * (kp + ks * s) < 0x1p-3) || !(tmax * inv_ulp < 0x1p41)) continue;
        if (!(b1 - tmax > std::ldexp(0.5, ex)) || !(b1 + tmax < std::ldexp(1.0, ex))) continue;
        blk[0] = (uint64_t)w_of((float)(coef(1) > 0 ? inv_ulp : -inv_ulp)) |
                 (bits_of(R) & 0xFFFFFFFF00000000ull);
        blk[1] = words(1.05 * kp, 1.05 * ks);
        blk[2] = words(1.05 * cp, 1.05 * cs);
        for (int k = 2; k <= 3; ++k) {
            double const b = k <= order ? coef(k) : 0.0;
            blk[k + 1] = words(b, b - (double)(float)b);
        }
        for (int j = 0; j < lead_words(order) - 5; ++j) {
            int const k = 4 + 2 * j;
            blk[5 + j] = words(coef(k), k + 1 <= order ? coef(k + 1) : 0.0);
        }
        return true;
    }
    return false;
}

}  // namespace stg
