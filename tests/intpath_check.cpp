// Checks intpath.cuh and leadkick.cuh on the CPU: every value they decide has
// the bits of the FP64 sequence it stands for.  argv: what, samples, seed.  Prints
// "<samples> <undecided> <different>".
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "leadkick.cuh"

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
                double u1, e1[2], e2[2];
                ok = ok && lead_exact(x, y, bal, order, &u1, e1, e2);
                a = px - plus(u1 * x - e1[0]), b = px - plus(u1 * x - e1[1]);
                c = py + plus(u1 * y + e2[0]), d = py + plus(u1 * y + e2[1]);
            }
            if (!ok || bits_of(a) != bits_of(b) || bits_of(c) != bits_of(d))
                ++*undecided;
            else if (bits_of(a) != bits_of(rx) || bits_of(c) != bits_of(ry))
                ++*different;
        }
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
