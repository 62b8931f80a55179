// Compares the integer forms of erlbm_gb300/csrc/fp64_int.cuh with the FP64 operations they stand for, on the CPU.
// Prints "cases bad" (build with -ffp-contract=off).
#define __host__
#define __device__
#define __forceinline__ inline
#include "../../erlbm_gb300/csrc/fp64_int.cuh"

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

using namespace erlbm::fp64int;

static std::mt19937_64 rng;

// A value of modulus below `most`: any scale down to underflow, short mantissas (ties), zeros of both signs.
static double draw(double most)
{
    const double x = std::ldexp((double)(int64_t)rng(), -63) * most;
    switch (rng() % 8) {
    case 0: return std::ldexp(x, -(int)(rng() % 70));
    case 1: return std::ldexp(x, -(int)(rng() % 1100));
    case 2: return std::ldexp((double)((int)(rng() % 33) - 16), -8 - (int)(rng() % 6)) * (most / 0.08);
    case 3: return rng() % 4 ? x : 0.0 * x;
    default: return std::ldexp(x, -(int)(rng() % 8));
    }
}

int main(int argc, char **argv)
{
    rng.seed(7);
    const long n = argc > 1 ? atol(argv[1]) : 1000000;
    long cases = 0, bad = 0;
    for (long it = 0; it < n; it++) {
        const double u[3] = {draw(0.08), draw(0.08), draw(0.08)};
        const double cv = it % 4 == 0 ? u[0] : it % 4 == 1 ? u[0] + u[1] : it % 4 == 2 ? u[0] - u[1] : 2.0 * u[0];
        const double C = 1.5 * ((u[0] * u[0] + u[1] * u[1]) + u[2] * u[2]);
        if (!(std::fabs(cv) < EQ_MAX) || !(C < 0.115)) continue;
        const double t3 = cv * 3., B = ((0.5 * cv) * cv * 3.) * 3.;
        const double a = ((1.0 + t3) + B) - C, b = ((1.0 - t3) + B) - C;
        double p, m;
        eq_pair(cv, cv * cv, fixed62(C), p, m);
        cases++;
        bad += bits(p) != bits(a) || bits(m) != bits(b);
    }
    // chains of adds and subtractions of populations in fixed point against the FP64 chain
    for (long it = 0; it < n; it++) {
        double s = 0;
        int64_t S = 0;
        for (int k = 0; k < 6; k++) {
            double f = std::ldexp(0.5 + std::ldexp((double)(rng() >> 12), -53), -(int)(rng() % 7));
            if (rng() % 4 == 0) f = std::ldexp(std::floor(std::ldexp(f, 20)), -20);
            const bool in = fix_range(f) < FIX_SPAN;
            bad += !in || to_double(to_fixed(f)) != f;
            const bool minus = rng() % 2;
            s = k == 0 ? f : minus ? s - f : s + f;
            S = k == 0 ? to_fixed(f) : round53(minus ? S - to_fixed(f) : S + to_fixed(f));
            bad += bits(to_double(S)) != bits(s + 0.0);
            cases++;
        }
    }
    // reciprocals, from first approximations off by up to 2^-20
    for (long it = 0; it < n; it++) {
        uint64_t M = rng() >> 12;
        if (rng() % 3 == 0) M = rng() % 64;
        if (rng() % 3 == 0) M = ~M & 0xfffffffffffffull;
        const double r = from_bits(M | ((rng() % 8 ? 1023 - 3 + rng() % 8 : 513 + rng() % 1000) << 52));
        double y = 0x1p32 / (1.0 + (double)M * 0x1p-52) * (1.0 + ((double)(rng() % 2001) - 1000.0) / 1000.0 * 0x1p-20);
        cases++;
        bad += bits(reciprocal_from(r, y >= 0x1p32 ? 0xffffffffu : (uint32_t)y)) != bits(1.0 / r);
    }
    // quotients by a constant and by 3
    for (long it = 0; it < n; it++) {
        const double y = std::ldexp(1.0 + std::ldexp((double)(rng() >> 12), -52), (int)(rng() % 9) - 6);
        double a = std::ldexp((double)(int64_t)rng(), -(int)(rng() % 600));
        if (rng() % 3 == 0) a = y * (double)(1 + rng() % 64) * (1.0 + std::ldexp((double)(rng() % 5) - 2.0, -52));
        if (!quotient_range(a)) continue;
        cases++;
        bad += bits(quotient(a, y, 1.0 / y)) != bits(a / y) || bits(quotient3(a)) != bits(a / 3.0);
    }
    for (double x : {0.0, -0.0, 0x1p-1022, 0x1p-512, 0x1p512, 0x1p1023, (double)INFINITY, (double)NAN})
        bad += quotient_range(x) || quotient_range(-x);
    bad += !quotient_range(0x1p-511) || !quotient_range(-1.0) || !quotient_range(0x1.8p511);
    const double out[] = {1.0, 1.5, 0x1p-8, 0x1.fffffffffffffp-8, -0.1, 0.0, -0.0, INFINITY, -INFINITY, NAN};
    for (double x : out) bad += fix_range(x) < FIX_SPAN;
    printf("%ld %ld\n", cases, bad);
    return 0;
}
