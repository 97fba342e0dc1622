// Checks intpath.cuh, leadkick.cuh and sckick.cuh on the CPU: every value they
// decide has the bits of the FP64 sequence it stands for.  argv: what, samples, seed.  Prints
// "<samples> <undecided> <different>".
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "sckick.cuh"

using namespace stg;

static std::mt19937_64 gen;

static double real(int emin, int emax)
{
    int const e = emin + (int)(gen() % (uint64_t)(emax - emin + 1));
    double const m = std::ldexp(1.0 + (double)(gen() >> 12) * 0x1p-52, e);
    return gen() & 1 ? m : -m;
}

static const double kSpecial[] = {0.0, -0.0, INFINITY, -INFINITY, NAN, 1.0, 0x1p-7, -0x1p-7,
                                  0x1.fffffffffffffp-8, 5e-324, -1e-310, 0x1p-30, 0x1p-26};

static double momentum(const char *what)
{
    if (!strcmp(what, "ordinary")) return real(-30, -8);
    if (!strcmp(what, "wide")) return real(-1074, 1);
    // sums of few bits: t / 2 falls on and beside the halves of 2^-52
    if (!strcmp(what, "ties")) return std::ldexp((double)(gen() % 128) - 64, -32 + (int)(gen() % 6));
    return kSpecial[gen() % (sizeof(kSpecial) / sizeof(double))];
}

static double uniform() { return (double)(gen() >> 11) * 0x1p-53; }
static double normal()
{
    return std::sqrt(-2.0 * std::log(uniform() + 0x1p-60)) * std::cos(6.283185307179586 * uniform());
}
static double plus(double v) { return v == 0.0 ? 0.0 : v; }

// Multipoles with lead blocks at coordinates of the given rms, some of them
// zero, subnormal or near an axis.
static void lead(bool fast, double rms, double errors, long n, long *undecided, long *different)
{
    for (long el = 0; el < n / 100; ++el) {
        int const order = (fast ? 3 : 2) + (int)(gen() % 9);
        uint64_t bal[64] = {};
        bal[2] = bits_of((gen() & 1 ? 1.0 : -1.0) * (0.005 + 0.05 * uniform()));
        double scale = errors;
        for (int k = 2; k <= order; ++k) bal[2 * k] = bits_of(normal() * (scale *= 0.1));
        if (!lead_block(bal, order, bal + 2 * order + 2)) {
            *undecided += 100;
            continue;
        }
        for (int l = 0; l < 100; ++l) {
            double x = rms * normal(), y = rms * normal();
            int const q = (int)(gen() % 24);
            if (q == 0) x = 0.0;
            if (q == 1) y = -0.0;
            if (q == 2) x *= 1e-3;
            if (q == 3) y *= std::pow(10.0, -30.0 * uniform());
            if (q == 4) x *= 1e-320;
            double const px = 1e-5 * normal() + (gen() & 1) * x / 30, py = 1e-5 * normal() + y / 40;
            double rx, ry, a, b, c, d;
            bool ok = lead_in_range(x, y, bal + 2 * order + 2);
            if (fast) {
                double const r = x + x, s = std::fma(x, x, y * y);
                double c1 = from_bits(bal[2 * order]);
                double c0 = std::fma(r, c1, from_bits(bal[2 * order - 2]));
                for (int j = order - 2; j >= 1; --j) {
                    double const cj = std::fma(r, c0, std::fma(-s, c1, from_bits(bal[2 * j])));
                    c1 = c0;
                    c0 = cj;
                }
                rx = px - std::fma(x, c0, std::fma(-s, c1, from_bits(bal[0])));
                ry = py + y * c0;
                double u1, w[2];
                ok = ok && lead_fast(x, y, bal, order, &u1, w);
                a = px - std::fma(x, u1, -w[0]), b = px - std::fma(x, u1, -w[1]);
                c = d = py + y * u1;
            } else {
                double u = from_bits(bal[2 * order]), v = 0.0;
                for (int k = order - 1; k >= 0; --k) {
                    double const zr = u * x - v * y, zi = u * y + v * x;
                    u = from_bits(bal[2 * k]) + zr;
                    v = from_bits(bal[2 * k + 1]) + zi;
                }
                rx = px - u;
                ry = py + v;
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
                // formed on the significands: within the bounds
                if (nearest_sum(kx, m1, dd[0], &s1)) a = b = px - s1;
                if (nearest_sum(ky, e2, dd[1], &s2)) c = d = py + s2;
            }
            if (!ok || bits_of(a) != bits_of(b) || bits_of(c) != bits_of(d))
                ++*undecided;
            else if (bits_of(a) != bits_of(rx) || bits_of(c) != bits_of(ry))
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

// Space-charge kicks of a beam of sx by sy, particles of rms amp: whether
// the bounds hold the kick, and the momenta it leads to.
static void space_charge(double sx, double sy, double amp, long n, long *undecided,
                         long *different)
{
    constexpr double pi = 3.14159265358979323846, eps0 = 8.854187817620e-12;
    bool const round = sx == sy, wide_x = sx > sy;
    double const sb = 1.0 / (std::sqrt(2.0) * 0.1), line = 0.1 * 1e11 * sb / std::sqrt(pi);
    double const su = wide_x ? sx : sy, sv = wide_x ? sy : sx;
    double const S = std::sqrt(2.0 * (su * su - sv * sv));
    double const factor = line / (round ? 2.0 * pi * eps0 : 2.0 * eps0 * std::sqrt(pi) * S);
    uint64_t blk[kScPairWords];
    if (!sc_pair_block(line, sb, round, 0.5 * (sx + sy), sx, sy, blk)) {
        *undecided = n;
        return;
    }
    for (long i = 0; i < n; ++i) {
        double const x = amp * normal(), y = amp * normal(), zeta = 0.05 * normal();
        double const irv = 1.0 + 1e-6 * normal(), k0 = 3.9e-40 * (1.0 + 1e-3 * normal());
        double const px = 1e-5 * normal(), py = 1e-5 * normal();
        long double const z = (long double)zeta * irv;
        long double const K = (long double)k0 * factor * expl(-(long double)sb * sb * z * z);
        long double ex, ey;
        if (round) {
            long double const r2 = (long double)x * x + (long double)y * y;
            long double const t = K * -expm1l(-0.5L * r2 / (sx * sx)) / r2;
            ex = t * x, ey = t * y;
        } else {
            double const u = std::fabs(wide_x ? x : y), v = std::fabs(wide_x ? y : x);
            long double a, b, c, d;
            cerrf(u / S, v / S, &a, &b);
            cerrf(sv / su * u / S, su / sv * v / S, &c, &d);
            long double const e = expl(-0.5L * ((long double)u * u / (su * su) +
                                                (long double)v * v / (sv * sv)));
            long double const fu = K * (b - d * e), fv = K * (a - c * e);
            ex = std::copysign((double)(wide_x ? fu : fv), x);
            ey = std::copysign((double)(wide_x ? fv : fu), y);
        }
        FPair const k = sc_factor(k0);
        double kx[2], ky[2];
        if (!sc_small(k, px, py, blk) ||
            !sc_pair_kick(x, y, k, zeta, irv, blk, round, wide_x, kx, ky) ||
            px + kx[0] != px + kx[1] || py + ky[0] != py + ky[1]) {
            ++*undecided;
            continue;
        }
        bool const in = std::fmin(kx[0], kx[1]) <= ex && ex <= std::fmax(kx[0], kx[1]) &&
                        std::fmin(ky[0], ky[1]) <= ey && ey <= std::fmax(ky[0], ky[1]);
        if (!in || px + kx[0] != px + (double)ex || py + ky[0] != py + (double)ey) ++*different;
    }
}

int main(int argc, char **argv)
{
    if (argc < 4) return 2;
    long const n = atol(argv[2]);
    gen.seed((uint64_t)atol(argv[3]));
    long undecided = 0, different = 0;
    if (!strncmp(argv[1], "lead", 4)) {
        bool const fast = argv[1][5] == 'f', wide = strstr(argv[1], "wide") != nullptr;
        lead(fast, wide ? 5e-3 : 1e-3, wide ? 1e-2 : 1e-4, n, &undecided, &different);
        printf("%ld %ld %ld\n", n, undecided, different);
        return 0;
    }
    if (!strncmp(argv[1], "product", 7)) {
        for (long i = 0; i < n; ++i) {
            double a, b;
            if (strstr(argv[1], "bits")) {  // any bit pattern
                a = from_bits(gen()), b = from_bits(gen());
            } else if (strstr(argv[1], "short")) {  // exact and half-way products
                a = std::ldexp((double)(int64_t)(gen() >> (10 + gen() % 50)), -40);
                b = std::ldexp((double)(int64_t)(gen() >> (10 + gen() % 50)), -60);
            } else if (strstr(argv[1], "special")) {
                a = kSpecial[gen() % 13], b = kSpecial[gen() % 13];
            } else {
                a = real(-40, 2), b = 1.0 + real(-52, -2);
            }
            double r;
            if (!mul_rn(a, b, &r))
                ++undecided;
            else if (bits_of(r) != bits_of(a * b))
                ++different;
        }
        printf("%ld %ld %ld\n", n, undecided, different);
        return 0;
    }
    if (!strncmp(argv[1], "sc", 2)) {
        double const amp = strstr(argv[1], "wide") ? 5e-3 : strstr(argv[1], "core") ? 2e-5 : 1e-3;
        double const sy = strstr(argv[1], "round") ? 1e-3 : strstr(argv[1], "tall") ? 1.2e-3 : 0.3e-3;
        space_charge(1e-3, sy, amp, n, &undecided, &different);
        printf("%ld %ld %ld\n", n, undecided, different);
        return 0;
    }
    for (long i = 0; i < n; ++i) {
        double const xp = momentum(argv[1]), yp = momentum(argv[1]);
        double rvv = 1.0 + real(-52, -9);
        if (!strcmp(argv[1], "special")) rvv = (gen() & 1) ? rvv : kSpecial[gen() % 13];
        int64_t s;
        if (!drift_slip(xp, yp, slip_rvv(rvv), slip_limit(rvv), &s)) {
            ++undecided;
            continue;
        }
        double const got = below_2_32(s) ? scaled_53(s) : scaled_53_large(s);
        double const exact = rvv - (1.0 + (xp * xp + yp * yp) * 0.5);
        double const fast = rvv - std::fma(std::fma(yp, yp, xp * xp), 0.5, 1.0);
        if (bits_of(got) != bits_of(exact) || bits_of(got) != bits_of(fast)) ++different;
    }
    printf("%ld %ld %ld\n", n, undecided, different);
    return 0;
}
