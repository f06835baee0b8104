// csrc/pd_ieee.h on the device: the single-instruction seeds against the
// bounds the header states, and rcp_rn, div_rn and sqrt_rcp_rn against the
// IEEE operators, for every leading 21 bits of a significand with several
// tails.  Prints "ok", the seeds' errors (log2) and the share of roots
// reported as not known exact.
#include <cmath>
#include <cstdio>

#include "../../peridyn_b200/csrc/pd_ieee.h"

using namespace pd;

struct Result {
    unsigned long long rcp_err, root_err;  // largest |1 - b y|, |1 - a y y| (bits of a non-negative double)
    unsigned long long wrong, unsure;
};

constexpr uint32_t kLead = 1u << 21;
constexpr int kTails = 6;

__device__ double operand(uint32_t lead, int tail, int exponent) {
    const uint32_t h = lead * 2654435761u ^ (uint32_t)tail * 40503u;
    const uint32_t low = tail == 0 ? 0u : tail == 1 ? 0x7ffffffeu : h & 0x7fffffffu;
    const uint64_t m = ((uint64_t)lead << 31) | low;
    return __longlong_as_double((long long)(((uint64_t)(1023 + exponent) << 52) | m));
}

__global__ void check(Result *r) {
    const uint32_t lead = blockIdx.x * blockDim.x + threadIdx.x;
    if (lead >= kLead) return;
    double rcp_err = 0.0, root_err = 0.0;
    unsigned long long wrong = 0, unsure = 0;
    for (int t = 0; t < kTails; ++t) {
        const int e = t < 2 ? 0 : (int)((lead * 7u + 13u * t) % 180u) - 90;
        const double b = operand(lead, t, e);
        double y;
        asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
        rcp_err = fmax(rcp_err, fabs(fma(-b, y, 1.0)));
        if (div_ok(b)) {
            const double rb = rcp_rn(b), a = operand(lead * 2246822519u % kLead, t, (e * 3) % 100);
            wrong += rb != 1.0 / b;
            wrong += div_rn(a, b, rb) != a / b;
            wrong += div_rn(-a, b, rb) != -a / b;
        }
        for (int odd = 0; odd < 2; ++odd) {
            const double a = operand(lead, t, 2 * (e / 2) + odd);
            asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
            root_err = fmax(root_err, fabs(fma(-(a * y), y, 1.0)));
            double root, rcp;
            if (!sqrt_rcp_rn(a, root, rcp)) ++unsure;
            else wrong += (root != sqrt(a)) + (rcp != 1.0 / sqrt(a));
        }
    }
    atomicMax(&r->rcp_err, (unsigned long long)__double_as_longlong(rcp_err));
    atomicMax(&r->root_err, (unsigned long long)__double_as_longlong(root_err));
    if (wrong) atomicAdd(&r->wrong, wrong);
    if (unsure) atomicAdd(&r->unsure, unsure);
}

static double value(unsigned long long bits) {
    double d;
    std::memcpy(&d, &bits, 8);
    return d;
}

int main() {
    Result *d, h{};
    if (cudaMalloc(&d, sizeof(Result)) != cudaSuccess || cudaMemset(d, 0, sizeof(Result)) != cudaSuccess) return 2;
    check<<<kLead / 256, 256>>>(d);
    const cudaError_t err = cudaMemcpy(&h, d, sizeof(Result), cudaMemcpyDeviceToHost);
    if (err != cudaSuccess) return std::printf("%s\n", cudaGetErrorString(err)), 2;
    const double er = value(h.rcp_err), es = value(h.root_err), n = 2.0 * kLead * kTails;
    // a reciprocal seed within 2^-19; a root seed within e = 2^-18.9, so |1 - a y y| within 2 e + e^2
    const double e = std::exp2(-18.9);
    const bool good = h.wrong == 0 && er > 0.0 && er <= 0x1p-19 && es > 0.0 && es <= 2.0 * e + e * e &&
                      (double)h.unsure < 1e-3 * n;
    std::printf("%s wrong %llu, |1 - b y| 2^%.2f, |1 - a y y| 2^%.2f, not known exact %.3g\n", good ? "ok" : "failed",
                h.wrong, std::log2(er), std::log2(es), (double)h.unsure / n);
    cudaFree(d);
    return good ? 0 : 1;
}
