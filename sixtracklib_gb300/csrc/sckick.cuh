// sckick.cuh -- the q-Gaussian space-charge kick in FP32 pairs, where it is
// far below the momenta it is added to.
//
// At collision energy the space-charge kick of one element is 10^-11 of a
// momentum: RN(px + k) needs k to 2^-20 or so, and the FP64 evaluation of k
// (about 40 FP64 instructions of 64-76 cycles for a round beam, 500 with the
// two Faddeeva functions of an elliptic one) settles nothing that pairs of
// floats do not.  The kick is evaluated here in pairs, with a bound on its
// error against the FP64 evaluation; both ends of the bound are added to the
// momentum and where the sums agree they are the FP64 evaluation's, else it
// is run.  Gaussian profiles (q = 1) only.  One turn of the FODO ring with 200
// such kicks and 4 + 4 beam-beam elements, fast: round beams, 65,536
// protons, 2 turns 5.05 -> 3.24 ms; elliptic, 33,333 protons 13.3 -> 8.6 ms
// (100,000: 41.6 -> 19.7 ms).
//
// The Faddeeva function follows faddeeva_cern.h:45-120 in the form of
// cerrf() (maps.cuh): the three-term recurrence Q(n) = w0 Q(n+1) +
// (n/2) Q(n+2) from n = nu down, of which a relative error at step n reaches
// the result with 2^-n of its size or less (measured on 200,000 points of
// the region: single precision for n > n0 costs 2^-(22 + n0)).  So the steps
// above 20 run in single floats, the others in pairs.
#pragma once

#include "leadkick.cuh"

namespace stg {

// 2^(j / 32) as pairs of floats: h the nearest float, l the nearest float of
// the rest (from 60 decimal digits).  An entry is read in one load of 8 bytes,
// which an array of floats is not aligned for.
struct alignas(8) ExpPair {
    float h, l;
};
#define STG_EXP32                                                           \
    {0x1p+0f, 0.0f}, {0x1.059b0ep+0f, -0x1.9d4f52p-25f},                    \
    {0x1.0b5586p+0f, 0x1.9f3122p-25f}, {0x1.11301ep+0f, -0x1.fdb496p-25f},  \
    {0x1.172b84p+0f, -0x1.c15742p-27f}, {0x1.1d4874p+0f, -0x1.d2e8cap-25f}, \
    {0x1.2387a6p+0f, 0x1.ceac48p-25f}, {0x1.29e9ep+0f, -0x1.5c0424p-25f},   \
    {0x1.306fep+0f, 0x1.4636e2p-25f}, {0x1.371a74p+0f, -0x1.18aac6p-25f},   \
    {0x1.3dea64p+0f, 0x1.824684p-25f}, {0x1.44e086p+0f, 0x1.8624b4p-30f},   \
    {0x1.4bfdaep+0f, -0x1.593abcp-25f}, {0x1.5342b6p+0f, -0x1.2c561p-25f},  \
    {0x1.5ab07ep+0f, -0x1.5bd5ecp-27f}, {0x1.6247ecp+0f, -0x1.f8b55p-25f},  \
    {0x1.6a09e6p+0f, 0x1.9fcef4p-26f}, {0x1.71f75ep+0f, 0x1.1d8beep-25f},   \
    {0x1.7a1148p+0f, -0x1.829fdp-25f}, {0x1.82589ap+0f, -0x1.accc7cp-26f},  \
    {0x1.8ace54p+0f, 0x1.15506ep-27f}, {0x1.93737cp+0f, -0x1.e64744p-25f},  \
    {0x1.9c4918p+0f, 0x1.51f848p-27f}, {0x1.a5503cp+0f, -0x1.b83b54p-25f},  \
    {0x1.ae89fap+0f, -0x1.a94b14p-26f}, {0x1.b7f77p+0f, -0x1.a09438p-25f},  \
    {0x1.c199bep+0f, -0x1.3d56b2p-27f}, {0x1.cb720ep+0f, -0x1.8837ccp-27f}, \
    {0x1.d5818ep+0f, -0x1.822dbcp-27f}, {0x1.dfc974p+0f, -0x1.908c94p-25f}, \
    {0x1.ea4afap+0f, 0x1.52486cp-27f}, {0x1.f50766p+0f, -0x1.246ebp-26f}

#if defined(__CUDACC__)
static __device__ const ExpPair kExp32Dev[32] = {STG_EXP32};
#endif
static const ExpPair kExp32[32] = {STG_EXP32};
#undef STG_EXP32

STG_HD FPair exp32(int j)
{
#if defined(__CUDA_ARCH__)
    float2 const v = __ldg(reinterpret_cast<const float2 *>(&kExp32Dev[j]));
    return FPair{v.x, v.y};
#else
    return FPair{kExp32[j].h, kExp32[j].l};
#endif
}

#if defined(__CUDA_ARCH__)
STG_HD float frcp(float a) { return __frcp_rn(a); }
STG_HD float fsqrt_(float a) { return __fsqrt_rn(a); }
#else
STG_HD float frcp(float a) { return 1.0f / a; }
STG_HD float fsqrt_(float a) { return std::sqrt(a); }
#endif

STG_HD FPair renorm(float h, float l)
{
    float const s = fadd(h, l);
    return FPair{s, fsub(l, fsub(s, h))};
}

STG_HD FPair neg(FPair a) { return FPair{-a.h, -a.l}; }

STG_HD FPair add(FPair a, FPair b)
{
    FPair const s = two_sum(a.h, b.h);
    return renorm(s.h, fadd(s.l, fadd(a.l, b.l)));
}

// a b + c d
STG_HD FPair mul_add_mul(FPair a, FPair b, FPair c, FPair d)
{
    FPair const p = mul(a, b), q = mul(c, d), s = two_sum(p.h, q.h);
    return renorm(s.h, fadd(s.l, fadd(p.l, q.l)));
}

STG_HD FPair div(FPair a, FPair b)
{
    float const r = frcp(b.h), q = fmul(a.h, r);
    float const rem = fadd(ffma(-q, b.h, a.h), ffma(-q, b.l, a.l));
    return renorm(q, fmul(rem, r));
}

// e^x for a pair -80 <= x <= 0 by P. T. P. Tang's table-driven method (ACM
// TOMS 15 (1989) 144): x = n ln2 / 32 + r.  With u = 2^-24, to 24 u^2 relative
// and 5 u |x.l| for the sums that the low part passes through; below x = -60
// the result's low part leaves the normal range.
STG_HD FPair exp_pair(FPair x)
{
    constexpr float kMagic = 12582912.0f;  // 1.5 2^23
    float const m = ffma(x.h, 0x1.715476p+5f, kMagic);
    float const n = fsub(m, kMagic);
    int32_t const k = (int32_t)(w_of(m) - 0x4B400000u);
    float const r1 = ffma(-n, 0x1.62ep-6f, x.h);  // exact
    float const p = fmul(-n, 0x1.0bfbe8p-20f);
    float const e = ffma(-n, 0x1.0bfbe8p-20f, -p);
    FPair const s = two_sum(r1, p);
    float const rl = fadd(s.l, fadd(fadd(e, x.l), fmul(-n, 0x1.cf79acp-45f)));
    FPair const r = renorm(s.h, rl);
    FPair const r2 = mul(r, r);
    float const c = fmul(fmul(r.h, r2.h), ffma(r.h, ffma(r.h, 0x1.111112p-7f, 0x1.555556p-5f),
                                              0x1.555556p-3f));
    FPair const q = two_sum(r.h, fmul(0.5f, r2.h));
    FPair const em1 = renorm(q.h, fadd(fadd(q.l, ffma(0.5f, r2.l, r.l)), c));
    FPair const t = exp32(k & 31), tq = mul(t, em1), v = two_sum(t.h, tq.h);
    float const scale = f_of((uint32_t)(127 + (k >> 5)) << 23);
    FPair const y = renorm(v.h, fadd(v.l, fadd(t.l, tq.l)));
    return FPair{fmul(y.h, scale), fmul(y.l, scale)};
}

// One Faddeeva evaluation on its way down the recurrence.
struct WPair {
    FPair x, w0r, q1r, q1i, q2r, q2i, ar, ai;
    float i2h;
    int nc, nu;
};

// Region and truncation of w(x + iy), x, y > 0: inside the algorithm's
// rectangle h, nc and nu from the region parameter q (h = 1 / (3.2 q) enters
// only through the truncation, 1e-10 of w, so its single-float value
// serves), outside it nine steps and Q(2) / Q(1), which is A(1) / Q(1) with
// nc = 1 and h = infinity.  False where the region, nc or nu is too close to
// call.
STG_HD bool w_start(FPair x, FPair y, WPair *s)
{
    float const dx = fadd(fsub(x.h, 0x1.551eb80000000p+2f), fsub(x.l, 0x1.47ae140000000p-24f));
    float const dy = fadd(fsub(y.h, 0x1.128f5c0000000p+2f), fsub(y.l, 0x1.47ae140000000p-25f));
    bool const inner = dx < 0.0f && dy < 0.0f;
    bool const edge = (fabs_(dx) < 1e-9f && dy < 1e-9f) || (fabs_(dy) < 1e-9f && dx < 1e-9f);
    s->x = x;
    s->q1r = FPair{1.0f, 0.0f};
    s->q1i = s->q2r = s->q2i = s->ar = s->ai = FPair{0.0f, 0.0f};
    s->i2h = 0.0f;
    s->nc = 1;
    s->nu = 9;
    s->w0r = y;
    if (!inner) return !edge;
    // q = (1 - y / 4.29) sqrt(1 - (x / 5.33)^2)
    FPair const xr = mul(x, FPair{0x1.803d7ap-3f, 0x1.e7fc28p-29f});
    FPair const xx = mul(xr, xr), yr = mul(y, FPair{0x1.dd63a8p-3f, -0x1.449fecp-29f});
    FPair const one{1.0f, 0.0f}, b = add(one, neg(xx));
    float const r = fsqrt_(b.h);
    float const rl = fmul(fadd(ffma(-r, r, b.h), b.l), fmul(0.5f, frcp(r)));
    FPair const q = mul(add(one, neg(yr)), FPair{r, rl});
    // floors of 23 q and 21 q: a product rounded up to an integer (their
    // last place is 2^-19) leaves a negative rest
    auto floor_of = [&](float k, int *i) {
        int const j = (int)fmul(k, q.h);
        float const rest = fadd(ffma(k, q.h, -(float)j), fmul(k, q.l));
        *i = rest < 0.0f ? j - 1 : j;
        return fabs_(rest) > 0x1p-30f;
    };
    int ic, iu;
    bool const clear = floor_of(23.0f, &ic) && floor_of(21.0f, &iu);
    if (!clear) return false;
    s->nc = 7 + ic;
    s->nu = 10 + iu;
    s->i2h = fmul(1.6f, q.h);
    s->w0r = add(y, FPair{s->i2h, 0.0f});
    return !edge;
}

// Step n in single floats (the low parts stay zero).
STG_HD void w_single(WPair &s, int n)
{
    float const hn = fmul(0.5f, (float)n);
    if (n <= s.nc) {
        s.ar.h = ffma(s.ar.h, s.i2h, s.q1r.h);
        s.ai.h = ffma(s.ai.h, s.i2h, s.q1i.h);
    }
    float const qr = ffma(s.w0r.h, s.q1r.h, ffma(-s.x.h, s.q1i.h, fmul(hn, s.q2r.h)));
    float const qi = ffma(s.w0r.h, s.q1i.h, ffma(s.x.h, s.q1r.h, fmul(hn, s.q2i.h)));
    s.q2r.h = s.q1r.h;
    s.q2i.h = s.q1i.h;
    s.q1r.h = qr;
    s.q1i.h = qi;
}

// To order one by a power of two, so that no square overflows below.
STG_HD void w_scale(WPair &s)
{
    float const down = f_of(0x7F000000u - (w_of(fmaxabs(s.q1r.h, s.q1i.h)) & 0x7F800000u));
    s.q1r.h = fmul(s.q1r.h, down);
    s.q1i.h = fmul(s.q1i.h, down);
    s.q2r.h = fmul(s.q2r.h, down);
    s.q2i.h = fmul(s.q2i.h, down);
    s.ar.h = fmul(s.ar.h, down);
    s.ai.h = fmul(s.ai.h, down);
}

// a b - c d + e f (f's low part zero) with one sum of the low parts: 30 operations.
STG_HD FPair w_row(FPair a, FPair b, FPair c, FPair d, FPair e, float f)
{
    float const p1 = fmul(a.h, b.h), p2 = fmul(c.h, d.h), p3 = fmul(e.h, f);
    float const e1 = ffma(a.h, b.h, -p1), e2 = ffma(c.h, d.h, -p2), e3 = ffma(e.h, f, -p3);
    FPair const s1 = two_sum(p1, -p2), s2 = two_sum(s1.h, p3);
    float l = fadd(fadd(s1.l, s2.l), fadd(fsub(e1, e2), e3));
    l = ffma(a.h, b.l, l);
    l = ffma(a.l, b.h, l);
    l = ffma(-c.h, d.l, l);
    l = ffma(-c.l, d.h, l);
    return renorm(s2.h, ffma(e.l, f, l));
}

// a g + q
STG_HD FPair w_sum(FPair a, float g, FPair q)
{
    float const p = fmul(a.h, g), e = ffma(a.h, g, -p);
    FPair const s = two_sum(p, q.h);
    return FPair{s.h, fadd(fadd(s.l, e), ffma(a.l, g, q.l))};
}

// Step n in pairs.
STG_HD void w_double(WPair &s, int n, bool series)
{
    float const hn = fmul(0.5f, (float)n);
    if (series) {
        s.ar = w_sum(s.ar, s.i2h, s.q1r);
        s.ai = w_sum(s.ai, s.i2h, s.q1i);
    }
    FPair const qr = w_row(s.w0r, s.q1r, s.x, s.q1i, s.q2r, hn);
    FPair const qi = w_row(s.w0r, s.q1i, neg(s.x), s.q1r, s.q2i, hn);
    s.q2r = s.q1r;
    s.q2i = s.q1i;
    s.q1r = qr;
    s.q1i = qi;
}

// w = (2 / sqrt(pi)) conj(A / (2 Q))
STG_HD void w_finish(const WPair &s, FPair *re, FPair *im)
{
    FPair const den = mul_add_mul(s.q1r, s.q1r, s.q1i, s.q1i);
    FPair const c{0x1.20dd76p-1f, -0x1.f7ac94p-26f};  // 1 / sqrt(pi) of the algorithm
    *re = mul(div(mul_add_mul(s.ar, s.q1r, s.ai, s.q1i), den), c);
    *im = mul(div(mul_add_mul(s.ar, s.q1i, neg(s.ai), s.q1r), den), c);
}

// w at two points, to about 2^-43 of |w|; the two recurrences run together
// (each is one chain of dependent operations).
STG_HD bool w_two(FPair x1, FPair y1, FPair x2, FPair y2, FPair *w1r, FPair *w1i, FPair *w2r,
                  FPair *w2i)
{
    WPair a, b;
    bool const fine = w_start(x1, y1, &a) && w_start(x2, y2, &b);
    if (!fine) return false;
    int n = a.nu > b.nu ? a.nu : b.nu;
    for (; n > 20; --n) {
        if (n <= a.nu) w_single(a, n);
        if (n <= b.nu) w_single(b, n);
    }
    w_scale(a);
    w_scale(b);
    // from m on both take every step: no branch between the four chains
    int m = a.nc < b.nc ? a.nc : b.nc;
    m = m < a.nu ? m : a.nu;
    m = m < b.nu ? m : b.nu;
    for (; n > m; --n) {
        if (n <= a.nu) w_double(a, n, n <= a.nc);
        if (n <= b.nu) w_double(b, n, n <= b.nc);
    }
    for (; n > 0; --n) {
        w_double(a, n, true);
        w_double(b, n, true);
    }
    w_finish(a, w1r, w1i);
    w_finish(b, w2r, w2i);
    return true;
}

// Words of the block that follows the kick's FP64 parameters (aux SC_PAIR),
// pairs of floats, the kick's element factor times 2^-90:
//   0: length N sqrt_beta / cq times 1 / (2 pi eps0) (round) or
//      1 / (2 eps0 sqrt(pi) S) (elliptic)
//   1: {bound on the field over that factor, 0}
//   2: sqrt_beta^2
//   round: 3: 0.5 / sigma^2
//   elliptic, u along the wider axis: 3: 1 / S   4: (sigma_v / sigma_u) / S
//      5: (sigma_u / sigma_v) / S   6: 0.5 / sigma_u^2   7: 0.5 / sigma_v^2
constexpr int kScPairWords = 8;

STG_HD FPair pair_of(uint64_t w)
{
    return FPair{f_of((uint32_t)w), f_of((uint32_t)(w >> 32))};
}

// The particle's factor times 2^90 (zero, negative or huge factors: h = 0).
STG_HD FPair sc_factor(double sc_k)
{
    uint64_t const w = bits_of(sc_k);
    uint32_t const hi = (uint32_t)(w >> 32);
    // 2^-150 .. 2^-90
    bool const fine = hi - ((1023u - 150u) << 20) < (60u << 20);
    FPair const p = split(from_words(hi + (90u << 20), (uint32_t)w));
    return fine ? p : FPair{0.0f, 0.0f};
}

// Whether the kick is small enough for its bound to decide RN(p + k): the
// largest field times the factors is below 2^-14 of both momenta.
STG_HD bool sc_small(FPair k, double px, double py, const uint64_t *blk)
{
    float const top = fmul(fmul(k.h, f_of((uint32_t)blk[0])), f_of((uint32_t)blk[1]));
    uint32_t const ax = (uint32_t)(bits_of(px) >> 32) & 0x7FFFFFFFu;
    uint32_t const ay = (uint32_t)(bits_of(py) >> 32) & 0x7FFFFFFFu;
    // top as the high word of a double, rounded up
    uint32_t const t = (w_of(top) >> 3) + 0x38000001u + (14u << 20);
    return top > 0x1p-110f && ax >= t && ay >= t && ax < 0x7FF00000u && ay < 0x7FF00000u;
}

// Bounds on the kick; x, y relative to the beam, z = zeta / rvv.  False where
// the pairs do not serve (on an axis, on the edge of the Faddeeva function's
// regions, far tails).
STG_HD bool sc_pair_kick(double x, double y, FPair k, double zeta, double inv_rvv,
                         const uint64_t *blk, bool round, bool wide_x, double *kx, double *ky)
{
    uint32_t const hx = (uint32_t)(bits_of(x) >> 32) & 0x7FFFFFFFu;
    uint32_t const hy = (uint32_t)(bits_of(y) >> 32) & 0x7FFFFFFFu;
    uint32_t const hz = (uint32_t)(bits_of(zeta) >> 32) & 0x7FFFFFFFu;
    uint32_t const hr = (uint32_t)(bits_of(inv_rvv) >> 32);
    // |x|, |y| in [2^-40, 0.5), |zeta| < 1, 0.5 <= 1 / rvv < 2
    bool fine = hx - 0x3D700000u < 0x02700000u && hy - 0x3D700000u < 0x02700000u &&
                hz < 0x3FF00000u && hr - 0x3FE00000u < 0x00200000u;
    if (!fine) return false;
    FPair const X = split(x), Y = split(y), z = mul(split(zeta), split(inv_rvv));
    FPair const az = neg(mul(mul(z, z), pair_of(blk[2])));
    if (az.h < -60.0f) return false;
    FPair const K = mul(mul(k, pair_of(blk[0])), exp_pair(az));
    // The bound.  With u = 2^-24 the low part of a split number is at most 2 u
    // of it and mul() of pairs with low parts a and b (in units of u) errs by
    // ab + 3 + 3a + 2b or so (u^2): zeta / rvv by 14 u^2, az by 97 u^2 with a
    // low part of 13 u, whose sums in exp_pair add 65 u^2 |az| to its own 24 u^2.
    // K is known to (162 |az| + 46) u^2; the round field adds 38 (its exponent),
    // 26 (difference and quotient) and 10 (times X), the elliptic one 67 of
    // |w| or less: below (162 |az| + 120) u^2, of which the FP64 evaluation's
    // own roundings and those of double_bounds take less than one.  Far out K or
    // the kick may leave the floats' range: never a bound of 0, which would
    // stand for a known kick of 0 (below 2^-75 double_bounds allows 2^-100).
    constexpr float kLeast = 0x1p-149f;
    float const rel = ffma(-az.h, 0x1.6p-41f, 0x1.2p-41f);  // (176 |az| + 144) u^2
    if (round) {
        FPair const r2 = mul_add_mul(X, X, Y, Y);
        // within 1e-10 m of the axis the field is another, sqrt(r2) / sigma
        if (r2.h < 1.0001e-20f) return false;
        FPair u = neg(mul(r2, pair_of(blk[3])));
        if (u.h < -80.0f) u = FPair{-80.0f, 0.0f};
        FPair const e = exp_pair(u), one = two_sum(1.0f, -e.h);
        FPair const g = mul(K, div(renorm(one.h, fsub(one.l, e.l)), r2));
        float const d = fmul(fmul(K.h, frcp(r2.h)), rel);
        double_bounds(mul(X, g), ffma(fabs_(X.h), d, kLeast), &kx[0], &kx[1]);
        double_bounds(mul(Y, g), ffma(fabs_(Y.h), d, kLeast), &ky[0], &ky[1]);
        return true;
    }
    FPair const ax{fabs_(X.h), X.h < 0.0f ? -X.l : X.l}, ay{fabs_(Y.h), Y.h < 0.0f ? -Y.l : Y.l};
    FPair const u = wide_x ? ax : ay, v = wide_x ? ay : ax;
    FPair const is = pair_of(blk[3]);
    FPair const zr = mul(u, is), zi = mul(v, is), er = mul(u, pair_of(blk[4])),
                ei = mul(v, pair_of(blk[5]));
    // |z| below 2^6, so that the squares of nine steps stay in range
    if (!(zr.h < 64.0f && zi.h < 64.0f && er.h < 64.0f && ei.h < 64.0f)) return false;
    FPair w1r, w1i, w2r, w2i;
    if (!w_two(zr, zi, er, ei, &w1r, &w1i, &w2r, &w2i)) return false;
    FPair arg = neg(mul_add_mul(mul(u, u), pair_of(blk[6]), mul(v, v), pair_of(blk[7])));
    if (arg.h < -80.0f) arg = FPair{-80.0f, 0.0f};
    FPair const e = exp_pair(arg);
    FPair const fu = mul(K, add(w1i, neg(mul(w2i, e)))), fv = mul(K, add(w1r, neg(mul(w2r, e))));
    float const d = ffma(fmul(K.h, fadd(fadd(w1r.h, w1i.h), fmul(e.h, fadd(w2r.h, w2i.h)))),
                         rel, kLeast);
    FPair fx = wide_x ? fu : fv, fy = wide_x ? fv : fu;
    if (X.h < 0.0f) fx = neg(fx);
    if (Y.h < 0.0f) fy = neg(fy);
    double_bounds(fx, d, &kx[0], &kx[1]);
    double_bounds(fy, d, &ky[0], &ky[1]);
    return true;
}

// ------------------------------------------------------------ host: the block
// `line`: length N sqrt_beta / cq.  False where a constant leaves the range
// of floats.
inline bool sc_pair_block(double line, double sqrt_beta, bool round, double sigma, double sx,
                          double sy, uint64_t *blk)
{
    constexpr double pi = 3.14159265358979323846, eps0 = 8.854187817620e-12;
    constexpr double sqrt_pi = 1.77245385090551602730;
    // a round field of 2^30 K, so that K keeps its low part for kicks of 2^-75
    if (round && !(sigma > 0x1p-30)) return false;
    double const su = sx > sy ? sx : sy, sv = sx > sy ? sy : sx;
    double const S = std::sqrt(2.0 * (su * su - sv * sv));
    double const factor = std::ldexp(
        line * (round ? 1.0 / (2.0 * pi * eps0) : 1.0 / (2.0 * eps0 * sqrt_pi * S)), -90);
    // the round field is at most 0.4513 / sigma; Re and Im of w, at most 1 and
    // 0.61, bound the elliptic one
    double const words[kScPairWords] = {
        factor, round ? 0.46 / sigma : 1.0, sqrt_beta * sqrt_beta,
        round ? 0.5 / (sigma * sigma) : 1.0 / S, round ? 0.0 : sv / su / S,
        round ? 0.0 : su / sv / S, round ? 0.0 : 0.5 / (su * su), round ? 0.0 : 0.5 / (sv * sv)};
    for (int k = 0; k < kScPairWords; ++k) {
        double const v = words[k];
        if (!(v == 0.0 && round && k >= 4) && !(v > 0x1p-60 && v < 0x1p60)) return false;
        float const h = (float)v;
        blk[k] = (uint64_t)w_of(h) | ((uint64_t)w_of((float)(v - (double)h)) << 32);
    }
    return true;
}

}  // namespace stg
