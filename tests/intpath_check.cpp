// Checks intpath.cuh on the CPU: every value it decides has the bits of the
// FP64 sequence it stands for.  argv: what, samples, seed.  Prints
// "<samples> <undecided> <different>".
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "intpath.cuh"

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

int main(int argc, char **argv)
{
    if (argc < 4) return 2;
    long const n = atol(argv[2]);
    gen.seed((uint64_t)atol(argv[3]));
    long undecided = 0, different = 0;
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
