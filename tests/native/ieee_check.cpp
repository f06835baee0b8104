// Checks csrc/pd_ieee.h against the IEEE operators: random operands,
// quotients and roots next to the middle of two neighbours, significands at
// the ends of a binade, with seeds anywhere within the bounds the header
// states.  Prints "ok" and the share of roots reported as not known exact.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../../peridyn_b200/csrc/pd_ieee.h"

using namespace pd;

static std::mt19937_64 rng(7);
static double unit() { return (double)(rng() >> 11) * 0x1p-53; }
// significand in [1, 2): random, near an end of the binade, or short
static double significand() {
    const uint64_t r = rng();
    switch (r % 5) {
        case 0: return 1.0 + (double)((r >> 8) % 64) * 0x1p-52;
        case 1: return 2.0 - (double)(1 + (r >> 8) % 64) * 0x1p-52;
        case 2: return 1.0 + (double)((r >> 8) % 4096) * 0x1p-12;
        default: return 1.0 + (double)(r >> 12) * 0x1p-52;
    }
}
static double seed(double exact, double bound) {
    const uint64_t r = rng() % 4;
    const double e = r == 0 ? bound : r == 1 ? -bound : (2.0 * unit() - 1.0) * bound;
    return exact * (1.0 + e);
}
static bool same(double a, double b) { return std::memcmp(&a, &b, 8) == 0; }

int main(int argc, char **argv) {
    const long n = argc > 1 ? std::atol(argv[1]) : 1000000;
    long unsure = 0;
    for (long i = 0; i < n; ++i) {
        const double b = std::ldexp(significand(), (int)(rng() % 199) - 100);
        double a = std::ldexp(significand(), (int)(rng() % 1199) - 600);
        if (i % 3 == 0) {  // a quotient next to the middle of two neighbours
            const double q = 1.0 + (double)(rng() >> 12) * 0x1p-52;
            const long double m = (long double)q + 0x1p-53L;
            a = (double)(m * (long double)b);
        }
        if (i % 7 == 0) a = 0.0;
        if (rng() & 1) a = -a;
        if (div_ok(b)) {
            const double r = rcp_refine(b, seed(1.0 / b, 0x1p-19));
            if (!same(r, 1.0 / b)) return std::printf("rcp %a: %a\n", b, r), 1;
            if (magnitude(a) >= kMagLo && !same(div_rn(a, b, r), a / b))
                return std::printf("div %a %a: %a\n", a, b, div_rn(a, b, r)), 1;
        }
        double s = std::ldexp(significand(), (int)(rng() % 397) - 199);
        if (i % 3 == 1) {  // a root next to the middle of two neighbours, or exact
            const double g = significand();
            const long double m = (long double)g + (i & 1 ? 0x1p-53L : 0.0L);
            s = (double)(m * m);
        }
        double root, rcp;
        if (!sqrt_rcp_refine(s, seed(1.0 / std::sqrt(s), 0x1p-19), root, rcp)) {
            ++unsure;
            continue;
        }
        if (!same(root, std::sqrt(s)) || !same(rcp, 1.0 / std::sqrt(s))) return std::printf("sqrt %a\n", s), 1;
    }
    // operands that must be refused
    double root, rcp;
    for (const double v : {0.0, -1.0, (double)INFINITY, (double)NAN, 0x1p-1060, 0x1p-300, 0x1p300})
        if (sqrt_rcp_refine(v, 1.0 / std::sqrt(v), root, rcp)) return std::printf("accepted sqrt %a\n", v), 1;
    for (const double v : {0.0, -2.0, (double)INFINITY, (double)NAN, 0x1p-101, 0x1p100, 2.0 - 0x1p-52})
        if (div_ok(v)) return std::printf("accepted divisor %a\n", v), 1;
    if (magnitude(0x1p-1074) >= kMagLo || magnitude(0x1p-601) >= kMagLo || magnitude(-0x1p-1074) >= kMagLo)
        return std::printf("accepted a small numerator\n"), 1;
    std::printf("ok %.2g\n", (double)unsure / (double)n);
    return 0;
}
