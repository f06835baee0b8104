// pd_ieee.h -- IEEE-rounded reciprocal, quotient and square root without a
// branch, for the serial-order FP64 kernels (device) and their check (host).
//
// Reciprocal and quotient (Markstein 1990, "Computation of elementary
// functions on the IBM RISC System/6000 processor"; Muller et al., Handbook
// of Floating-Point Arithmetic, the chapter on division with a fused
// multiply-add):
//   * y within one ulp of 1/b, b's significand not all ones:
//     RN(y + y RN(1 - b y)) = RN(1/b);
//   * r = RN(1/b), q within one ulp of a/b, a - b q exact:
//     RN(q + r (a - b q)) = RN(a/b).
// The seed rcp.approx.ftz.f64 is off by at most 2^-19 (every leading
// significand measured: 2^-19.94); one cubic step takes it to 2^-57 before
// rounding, so y is within one ulp.  a r is within two ulps of a/b, so one
// correction makes q faithful and the second rounds it.
//
// Square root: rsqrt.approx.ftz.f64 is off by at most 2^-18.9 (|1 - a y y|,
// about twice that, measured: 2^-19.04); one cubic step takes y to a couple of ulps, and the
// corrected root is sqrt(a) to 2^-100 before its rounding, so it can only be
// misrounded when sqrt(a) lies that close to the middle of two neighbours.
// There the (exact) residual a - root^2 is root ulp(root) in magnitude to
// 2^-50, so a residual whose high word reaches that of root ulp(root), less
// one, is reported as not known to be exact (one operand in 2^19).
//
// For operands div_ok and magnitude accept the results equal the IEEE
// operators'; the kernels evaluate the others with the operators.  Those
// take a slow path for a zero or very small numerator, and an undisturbed
// region of a body has zero stretch in every bond: the PMB force pass of a
// 48^3 cube executed 540 instructions per bond with them, 230 without.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define PD_HD __host__ __device__ __forceinline__
#else
#define PD_HD inline
#endif

namespace pd {

PD_HD int32_t hi_word(double a) {
#ifdef __CUDA_ARCH__
    return __double2hiint(a);
#else
    int64_t b;
    std::memcpy(&b, &a, 8);
    return (int32_t)(b >> 32);
#endif
}
PD_HD int32_t lo_word(double a) {
#ifdef __CUDA_ARCH__
    return __double2loint(a);
#else
    int64_t b;
    std::memcpy(&b, &a, 8);
    return (int32_t)b;
#endif
}
PD_HD double from_words(int32_t hi, int32_t lo) {
#ifdef __CUDA_ARCH__
    return __hiloint2double(hi, lo);
#else
    const int64_t b = ((int64_t)hi << 32) | (uint32_t)lo;
    double a;
    std::memcpy(&a, &b, 8);
    return a;
#endif
}

// RN(1/b) from a seed y.
PD_HD double rcp_refine(double b, double y) {
    double e = fma(-b, y, 1.0);
    y = fma(y, fma(e, e, e), y);
    return fma(y, fma(-b, y, 1.0), y);
}

// RN(a/b) for b > 0 and r = RN(1/b); the sign of a zero quotient is a's.
PD_HD double div_rn(double a, double b, double r) {
    double q = a * r;
    q = fma(fma(-b, q, a), r, q);
    q = fma(fma(-b, q, a), r, q);
    return from_words((hi_word(q) & 0x7fffffff) | (hi_word(a) & (int32_t)0x80000000), lo_word(q));
}

// Operands rcp_refine and div_rn are exact for: divisors positive, in
// [2^-100, 2^100), their significand not all ones (its low word, here);
// numerators zero or of magnitude in [2^-600, 2^600).  Quotients and
// residuals then stay normal.
PD_HD bool div_ok(double b) {
    return (uint32_t)hi_word(b) - ((1023u - 100u) << 20) < (200u << 20) && lo_word(b) != -1;
}
// 2 |high word|, plus one when the low word is not zero, less one: orders
// magnitudes, with zero above everything and a subnormal at the bottom.
PD_HD uint32_t magnitude(double a) {
    return 2u * (uint32_t)hi_word(a) + (lo_word(a) != 0 ? 1u : 0u) - 1u;
}
constexpr uint32_t kMagLo = (1023u - 600u) << 21, kMagHi = (1023u + 400u) << 21;

// root = RN(sqrt(a)) and rcp = RN(1 / root) from a seed y of 1/sqrt(a);
// returns whether both are known to be exact.  Out of range or unordered
// operands give a root outside div_ok's range.
PD_HD bool sqrt_rcp_refine(double a, double y, double &root, double &rcp) {
    const double e = fma(-(a * y), y, 1.0);
    y = fma(y * e, fma(e, 0.375, 0.5), y);
    double g = a * y;
    g = fma(fma(-g, g, a), 0.5 * y, g);
    const double d = fma(-g, g, a);
    const int32_t h = hi_word(g);
    const int32_t half = (int32_t)((uint32_t)h + ((uint32_t)h & 0x7ff00000u) - (1075u << 20));  // of g ulp(g)
    y = fma(y, fma(-g, y, 1.0), y);
    rcp = fma(y, fma(-g, y, 1.0), y);
    root = g;
    return div_ok(g) && (hi_word(d) & 0x7fffffff) < half - 1;
}

#ifdef __CUDACC__
__device__ __forceinline__ double rcp_rn(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    return rcp_refine(b, y);
}
__device__ __forceinline__ bool sqrt_rcp_rn(double a, double &root, double &rcp) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    return sqrt_rcp_refine(a, y, root, rcp);
}
#endif

}  // namespace pd
