// Checks the kicks of leadkick.cuh and sckick.cuh on the CPU over the whole range of
// coordinates and momenta that they accept.  argv: what, samples, seed.
// Prints "<samples> <undecided> <different>".
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "sckick.cuh"

using namespace stg;

static std::mt19937_64 gen;

static double uniform() { return (double)(gen() >> 11) * 0x1p-53; }
static double between(double a, double b) { return a + (b - a) * uniform(); }
static double sign() { return gen() & 1 ? 1.0 : -1.0; }
static double normal()
{
    return std::sqrt(-2.0 * std::log(uniform() + 0x1p-60)) * std::cos(6.283185307179586 * uniform());
}
// of either sign, its logarithm to base 10 uniform
static double decades(double lo, double hi) { return sign() * std::pow(10.0, between(lo, hi)); }
static double plus(double v) { return v == 0.0 ? 0.0 : v; }

// One coordinate or both within [1e-12, 8e-3] m, the other down to 1e-40 m or
// zero; a momentum of the kick's own size, of a beam's, or zero.  Quadrupoles
// and errors of any strength that gives a lead block.
static void lead(bool fast, long n, long *undecided, long *different)
{
    for (long el = 0; el < n / 100;) {
        int const order = (fast ? 3 : 2) + (int)(gen() % 9);
        uint64_t bal[64] = {};
        double const b1 = decades(-12, 2.9), ratio = std::fabs(decades(-8, 1));
        bal[2] = bits_of(b1);
        double scale = std::fabs(b1) * ratio;
        for (int k = 2; k <= order; ++k) bal[2 * k] = bits_of(normal() * scale), scale *= 0.3;
        if (!lead_block(bal, order, bal + 2 * order + 2)) continue;
        ++el;
        for (int l = 0; l < 100; ++l) {
            double x = decades(-12, -2.1), y = decades(l & 1 ? -40 : -12, -2.1);
            if (l % 25 == 0) y = l % 50 ? 0.0 : -0.0;
            if (l % 4 == 2) std::swap(x, y);
            double rx, ry;  // the kick: px -= rx, py += ry
            if (fast) {
                double const r = x + x, s = std::fma(x, x, y * y);
                double c1 = from_bits(bal[2 * order]);
                double c0 = std::fma(r, c1, from_bits(bal[2 * order - 2]));
                for (int j = order - 2; j >= 1; --j) {
                    double const cj = std::fma(r, c0, std::fma(-s, c1, from_bits(bal[2 * j])));
                    c1 = c0;
                    c0 = cj;
                }
                rx = std::fma(x, c0, std::fma(-s, c1, from_bits(bal[0])));
                ry = y * c0;
            } else {
                double u = from_bits(bal[2 * order]), v = 0.0;
                for (int k = order - 1; k >= 0; --k) {
                    double const zr = u * x - v * y, zi = u * y + v * x;
                    u = from_bits(bal[2 * k]) + zr;
                    v = from_bits(bal[2 * k + 1]) + zi;
                }
                rx = u;
                ry = v;
            }
            int const m = (int)(gen() % 4);
            double const px = m == 0 ? 1e-5 * normal() : m == 1 ? 0.0 : rx * decades(-3, 3);
            double const py = m == 0 ? 1e-5 * normal() : m == 1 ? 0.0 : ry * decades(-3, 3);
            double a, b, c, d;
            bool ok = lead_in_range(x, y, bal + 2 * order + 2);
            if (fast) {
                double u1, w[2];
                ok = ok && lead_fast(x, y, bal, order, &u1, w);
                a = px - std::fma(x, u1, -w[0]), b = px - std::fma(x, u1, -w[1]);
                c = d = py + y * u1;
            } else {
                double u1, s1, s2, b1[2], b2[2];
                FPair e1, e2;
                float dd[2];
                ok = ok && lead_exact(x, y, bal, order, &u1, &e1, &e2, dd);
                double const kx = u1 * x, ky = u1 * y;
                FPair const m1{-e1.h, -e1.l};
                double_bounds(m1, dd[0], &b1[0], &b1[1]);
                double_bounds(e2, dd[1], &b2[0], &b2[1]);
                a = px - plus(kx + b1[0]), b = px - plus(kx + b1[1]);
                c = py + plus(ky + b2[0]), d = py + plus(ky + b2[1]);
                if (nearest_sum(kx, m1, dd[0], &s1)) a = b = px - s1;
                if (nearest_sum(ky, e2, dd[1], &s2)) c = d = py + s2;
            }
            if (!ok || bits_of(a) != bits_of(b) || bits_of(c) != bits_of(d))
                ++*undecided;
            else if (bits_of(a) != bits_of(px - rx) || bits_of(c) != bits_of(py + ry))
                ++*different;
        }
    }
}

// The Faddeeva function of the CERN algorithm in long double (x, y > 0).
static void cerrf(double x, double y, long double *wr, long double *wi)
{
    bool const inner = x < 5.33 && y < 4.29;
    double const q = inner ? (1.0 - y / 4.29) * std::sqrt(1.0 - (x / 5.33) * (x / 5.33)) : 0.0;
    int const nc = inner ? 7 + (int)(23.0 * q) : 1, nu = inner ? 10 + (int)(21.0 * q) : 9;
    long double const g = 1.6 * q, u = y + g, v = x;
    long double q1r = 1, q1i = 0, q2r = 0, q2i = 0, ar = 0, ai = 0;
    for (int n = nu; n > 0; --n) {
        if (n <= nc) ar = ar * g + q1r, ai = ai * g + q1i;
        long double const qr = u * q1r - v * q1i + 0.5L * n * q2r;
        long double const qi = u * q1i + v * q1r + 0.5L * n * q2i;
        q2r = q1r, q2i = q1i, q1r = qr, q1i = qi;
    }
    long double const c = 0.5L * 1.12837916709551L / (q1r * q1r + q1i * q1i);
    *wr = (ar * q1r + ai * q1i) * c;
    *wi = (ar * q1i - ai * q1r) * c;
}

// Space charge of a Gaussian beam; of the round field both forms, the one
// within 1e-10 m of the axis included.  A kick outside its bounds counts as
// different whether its momenta are decided or not.
struct Beam {
    double sx, sy, sb, line;
    uint64_t blk[kScPairWords];
    long double factor;

    bool make(double x, double y, double bunch)
    {
        constexpr long double pi = 3.14159265358979323846L, eps0 = 8.854187817620e-12L;
        sx = x;
        sy = y;
        sb = 1.0 / (std::sqrt(2.0) * bunch);
        line = 0.1 * 1e11 * sb / std::sqrt(3.14159265358979323846);
        double const su = std::fmax(sx, sy), sv = std::fmin(sx, sy);
        factor = line / (sx == sy ? 2 * pi * eps0
                                  : 2 * eps0 * sqrtl(pi * 2.0L * (su * su - sv * sv)));
        return sc_pair_block(line, sb, sx == sy, 0.5 * (sx + sy), sx, sy, blk);
    }

    void field(double x, double y, long double *ex, long double *ey) const
    {
        if (sx == sy) {
            long double const r2 = (long double)x * x + (long double)y * y, s = sx;
            long double const t = r2 < 1e-20L ? sqrtl(r2) / s : -expm1l(-0.5L * r2 / (s * s)) / r2;
            *ex = t * x, *ey = t * y;
            return;
        }
        bool const wide = sx > sy;
        double const su = std::fmax(sx, sy), sv = std::fmin(sx, sy);
        double const S = std::sqrt(2.0 * (su * su - sv * sv));
        double const u = std::fabs(wide ? x : y), v = std::fabs(wide ? y : x);
        long double a, b, c, d;
        cerrf(u / S, v / S, &a, &b);
        cerrf(sv / su * u / S, su / sv * v / S, &c, &d);
        long double const e = expl(-0.5L * ((long double)u * u / ((long double)su * su) +
                                            (long double)v * v / ((long double)sv * sv)));
        long double const fu = b - d * e, fv = a - c * e;
        *ex = std::copysign(1.0, x) * (wide ? fu : fv);
        *ey = std::copysign(1.0, y) * (wide ? fv : fu);
    }

    void one(double x, double y, double zeta, double irv, double k0, double room, long *undecided,
             long *different) const
    {
        long double const z = (long double)zeta * irv;
        long double const K = k0 * factor * expl(-(long double)sb * sb * z * z);
        long double ex, ey;
        field(x, y, &ex, &ey);
        ex *= K, ey *= K;
        // momenta from the smallest that may be decided up
        double const top = (double)(k0 * factor) * (sx == sy ? 0.46 / sx : 1.0) * 16500.0;
        double const px = sign() * top * room, py = sign() * top * room * between(1, 2);
        FPair const k = sc_factor(k0);
        double kx[2], ky[2];
        if (!sc_small(k, px, py, blk) ||
            !sc_pair_kick(x, y, k, zeta, irv, blk, sx == sy, sx > sy, kx, ky)) {
            ++*undecided;
            return;
        }
        bool const in = std::fmin(kx[0], kx[1]) <= ex && ex <= std::fmax(kx[0], kx[1]) &&
                        std::fmin(ky[0], ky[1]) <= ey && ey <= std::fmax(ky[0], ky[1]);
        bool const same = px + kx[0] == px + kx[1] && py + ky[0] == py + ky[1];
        if (!in || (same && (px + kx[0] != px + (double)ex || py + ky[0] != py + (double)ey)))
            ++*different;
        else if (!same)
            ++*undecided;
    }
};

static void near_axis(long n, long *undecided, long *different)
{
    for (long i = 0; i < n;) {
        double const sigma = std::fabs(decades(-6, -3));
        Beam b;
        if (!b.make(sigma, sigma, 0.1)) continue;
        for (int l = 0; l < 100; ++l, ++i) {
            double const x = decades(-13, -8), y = decades(-13, -8);
            b.one(x, y, 0.05 * normal(), 1.0 + 1e-6 * normal(), 3.9e-40 * between(1, 2),
                  std::fabs(decades(0, 4)), undecided, different);
        }
    }
}

// The longitudinal exponent over its whole range, particles within four sigma.
static void tails(bool round, long n, long *undecided, long *different)
{
    for (long i = 0; i < n;) {
        double const sx = std::fabs(decades(-8, -2));
        Beam b;
        if (!b.make(sx, round ? sx : sx * std::fabs(decades(-1.5, 1.5)),
                    std::fabs(decades(-3, -0.5))))
            continue;
        for (int l = 0; l < 100; ++l, ++i) {
            double const x = 4 * b.sx * between(-1, 1), y = 4 * b.sy * between(-1, 1);
            b.one(x, y, sign() * std::sqrt(61.0 * uniform()) / b.sb, 1.0 + 1e-6 * normal(),
                  3.9e-40 * std::fabs(decades(-3, 3)), std::fabs(decades(0, 4)), undecided,
                  different);
        }
    }
}

// The table of exp_pair: entries and their alignment for one load each.
static void table(long *different)
{
    for (int j = 0; j < 32; ++j) {
        long double const v = exp2l(j / 32.0L);
        float const h = (float)v, l = (float)(v - h);
        FPair const t = exp32(j);
        if (t.h != h || t.l != l || alignof(decltype(kExp32[0])) < 8 || (uintptr_t)&kExp32[j] % 8)
            ++*different;
    }
}

int main(int argc, char **argv)
{
    if (argc < 4) return 2;
    long const n = atol(argv[2]);
    gen.seed((uint64_t)atol(argv[3]));
    long undecided = 0, different = 0;
    if (!strcmp(argv[1], "table"))
        table(&different);
    else if (!strcmp(argv[1], "near axis"))
        near_axis(n, &undecided, &different);
    else if (!strncmp(argv[1], "tails", 5))
        tails(!strcmp(argv[1], "tails round"), n, &undecided, &different);
    else
        lead(!strcmp(argv[1], "lead fast"), n, &undecided, &different);
    printf("%ld %ld %ld\n", n, undecided, different);
    return 0;
}
