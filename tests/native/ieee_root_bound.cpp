// csrc/pd_ieee.h's square root with seeds anywhere within the bound the
// header states, 2^-18.9 of 1/sqrt(a): where sqrt_rcp_refine reports an exact
// result, root and reciprocal equal the operators'.  Prints "ok" and the
// share reported as not known exact.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../../peridyn_b200/csrc/pd_ieee.h"

using namespace pd;

int main(int argc, char **argv) {
    const long n = argc > 1 ? std::atol(argv[1]) : 1000000;
    const double bound = std::exp2(-18.9);
    std::mt19937_64 rng(11);
    auto unit = [&] { return (double)(rng() >> 11) * 0x1p-53; };
    long unsure = 0;
    for (long i = 0; i < n; ++i) {
        double a = std::ldexp(1.0 + unit(), (int)(rng() % 397) - 199);
        if (i % 3 == 0) {  // next to, or on, the square of a double or of the middle of two
            const long double m = (long double)(1.0 + unit()) + (i & 1 ? 0x1p-53L : 0.0L);
            a = std::ldexp((double)(m * m), 2 * ((int)(rng() % 190) - 95));
        } else if (i % 3 == 1) {  // next to a power of two
            a = std::ldexp(1.0 + ((double)(rng() % 129) - 64.0) * 0x1p-53, (int)(rng() % 390) - 195);
        }
        const uint64_t r = rng() % 4;
        const double e = r == 0 ? bound : r == 1 ? -bound : (2.0 * unit() - 1.0) * bound;
        double root, rcp;
        if (!sqrt_rcp_refine(a, 1.0 / std::sqrt(a) * (1.0 + e), root, rcp)) {
            ++unsure;
            continue;
        }
        if (root != std::sqrt(a) || rcp != 1.0 / std::sqrt(a)) return std::printf("sqrt %a, seed off by %a\n", a, e), 1;
    }
    std::printf("ok %.2g\n", (double)unsure / (double)n);
    return unsure > n / 2;
}
