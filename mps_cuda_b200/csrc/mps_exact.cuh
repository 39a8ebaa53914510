// mps_exact.cuh -- correctly rounded square root and division for operands in a known range.
//
// The step's pair terms need IEEE square roots and quotients (kernel.cu:1062-1064, 1346-1348,
// 1731-1735). sqrt() and `/` pay for the whole range of their type: scaling, special values and
// a branch to a slow path in every pair. A pair's operands lie in a narrow range that is checked
// once (SceneDev::pair_lo), and inside it a hardware estimate, one Newton step and one residual
// step in fused multiply-adds round correctly:
//   root      g = x y, g' = g + (x - g^2) y / 2 with y ~ 1/sqrt(x)
//   quotient  y' = y + y (1 - b y), q = a y', q' = q + (a - b q) y' with y ~ 1/b
// (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor",
// IBM J. Res. Dev. 34, 1990: with y' the correctly rounded reciprocal and no overflow or
// underflow in between, q' is the correctly rounded quotient).
//
// What is shown. Single: the root and the reciprocal by trial of every significand
// (tests/test_gpu_exact.py), so the quotient by the theorem. Double, with 1 <= b < 2: a reciprocal y
// within 0.6 last places of 1/b becomes the nearest double by one more step, which before it rounds
// is short of 1/b by (1 - b y)^2 / b < 1.5 2^-106 / b. A middle m of two doubles has
// b m = 1 + j 2^-106 with an integer j other than 0, so it lies at least 2^-106 / b from 1/b, and
// only j = -1 could make the step round wrongly. The significands of b and m, as integers, then
// multiply to 2^106 - 1, which has one divisor of 53 bits: 2^53 - 1. That divisor b is set apart,
// and the quotient follows by the theorem. The double root's last step errs by less than 2^-51 last
// places, and only operands whose exact root lies nearer than that to a middle could round wrongly;
// tests/test_gpu_exact_hard.py tries all of those, and the quotients nearest to a middle.
#pragma once
#include <cuda_runtime.h>

namespace mps {

__device__ __forceinline__ float rsqrt_est(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp_est(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ double rsqrt_est(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}
__device__ __forceinline__ double rcp_est(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}

// sqrt(x)
__device__ __forceinline__ float sqrt_in(float x) {
    const float y = rsqrt_est(x);
    const float g = x * y, h = 0.5f * y;
    return __fmaf_rn(__fmaf_rn(-g, g, x), h, g);
}
__device__ __forceinline__ double sqrt_in(double x) {
    const double y = rsqrt_est(x);  // about 20 bits: two coupled Newton steps, then the residual
    double g = x * y, h = 0.5 * y;
    double r = __fma_rn(-g, h, 0.5);
    g = __fma_rn(g, r, g);
    h = __fma_rn(h, r, h);
    r = __fma_rn(-g, h, 0.5);
    g = __fma_rn(g, r, g);
    h = __fma_rn(h, r, h);
    return __fma_rn(__fma_rn(-g, g, x), h, g);
}

// 1 / b
__device__ __forceinline__ float rcp_in(float b) {
    const float y = rcp_est(b);
    return __fmaf_rn(y, __fmaf_rn(-b, y, 1.0f), y);
}
__device__ __forceinline__ double rcp_in(double b) {
    double y = rcp_est(b);
    const double e = __fma_rn(-b, y, 1.0);
    y = __fma_rn(y, __fma_rn(e, e, e), y);     // y (1 + e + e^2): the estimate's 20 bits to 0.6 places
    y = __fma_rn(y, __fma_rn(-b, y, 1.0), y);  // to the nearest double
    // 1 / (2 - 2^-52) lies just above the middle of 1/2 and the next double, where the step ties
    const int hi = __double2hiint(b), lo = __double2loint(b);
    const int tie = ((hi | int(0xfff00000u)) & lo) == -1;
    return __hiloint2double(__double2hiint(y), __double2loint(y) | tie);
}

// a / b given y = 1 / b, correctly rounded
__device__ __forceinline__ float div_by(float a, float b, float y) {
    const float q = a * y;
    return __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
}
__device__ __forceinline__ double div_by(double a, double b, double y) {
    const double q = a * y;
    return __fma_rn(__fma_rn(-b, q, a), y, q);
}
template <class R> __device__ __forceinline__ R div_in(R a, R b) { return div_by(a, b, rcp_in(b)); }

}  // namespace mps
