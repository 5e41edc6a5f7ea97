// sifv_fastmath.cuh -- arithmetic building blocks of the fast-FP64 and
// mixed-precision paths (never used by the reference-ordered path): fast
// reciprocal / square root, and both WENO5 face values of a cell from one
// set of smoothness indicators.
#pragma once

#include <cuda_runtime.h>

namespace sifv {

// Fast reciprocal and square root of the fast / mixed paths.  FP64: the
// hardware approximation (rcp.approx.ftz.f64 / rsqrt.approx.ftz.f64, about
// 2^-20 relative error, measured) refined by one third-order step: with
// e = 1 - x y, 1/x = y / (1 - e) = y (1 + e + e^2) + O(e^3); with
// e = 1 - x y^2, 1/sqrt(x) = y (1 - e)^(-1/2) = y (1 + e/2 + 3 e^2 / 8) + O(e^3),
// O(e^3) ~ 2^-60, below half an ulp (one step where two Newton-Raphson steps
// y <- y + y e took four fused operations); sqrt(x) = x * (1 / sqrt(x))
// with one correction s <- s + (x - s^2) y / 2.  Within 1 ulp of the IEEE
// results (checked against them by sifv_fastmath_selftest).  FP32: the
// single-instruction approximations (about 1 ulp).  The reference-ordered
// path never uses these.
__device__ __forceinline__ double frcp(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}
__device__ __forceinline__ float frcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// sqrt of a positive normal argument
__device__ __forceinline__ double fsqrt_pos(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x * y, y, 1.0);
    y = fma(y, e * fma(e, 0.375, 0.5), y);
    double sq = x * y;
    double r = fma(-sq, sq, x);
    return fma(r, 0.5 * y, sq);
}
__device__ __forceinline__ float fsqrt_pos(float x) {
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// 1 / sqrt(x) of a positive normal argument: the hardware approximation
// refined by the third-order step above (FP64; within 1 ulp of IEEE
// 1 / sqrt(x), checked by sifv_fastmath_selftest), the single-instruction
// approximation in FP32.
__device__ __forceinline__ double frsqrt_pos(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x * y, y, 1.0);
    return fma(y, e * fma(e, 0.375, 0.5), y);
}
__device__ __forceinline__ float frsqrt_pos(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Both WENO5 face values of the cell whose 5-cell stencil is v0..v4
// (v2 = the cell): L = value at its right face from the left,
// R = value at its left face from the right.
//
// In terms of the four differences d: the indicators times four are
// 13/3 t^2 + s^2 with t, s one operation each, and since the weights sum to
// one the candidates enter as their offsets from v2 (times six; the 1/6 goes
// into the normalisation).  The linear weights count as 1 : 6 : 3.
// 56 operations and two reciprocals where the form in cell values took 77
// (fused 2D stage at 4096^2: 3.84 -> 3.26 ms per step).
__device__ __forceinline__ void weno5_pair(double v0, double v1, double v2, double v3, double v4, double eps,
                                           double& L, double& R) {
    const double d0 = v1 - v0, d1 = v2 - v1, d2 = v3 - v2, d3 = v4 - v3;
    const double t0 = d1 - d0, t1 = d2 - d1, t2 = d3 - d2;
    const double s0 = fma(3.0, d1, -d0), s1 = d1 + d2, s2 = fma(-3.0, d2, d3);
    const double e = 4.0 * eps;
    double q0 = fma(s0, s0, fma((13.0 / 3.0) * t0, t0, e));
    double q1 = fma(s1, s1, fma((13.0 / 3.0) * t1, t1, e));
    double q2 = fma(s2, s2, fma((13.0 / 3.0) * t2, t2, e));
    q0 *= q0; q1 *= q1; q2 *= q2;
    // a_k = d_k / q_k; multiplying through by q0 q1 q2 leaves one division per side
    const double m01 = q0 * q1, m12 = q1 * q2, c1 = 6.0 * (q0 * q2);
    const double l2 = 3.0 * m01, r0 = 3.0 * m12;   // L: (1, 6, 3) on (q0, q1, q2); R: (3, 6, 1)
    const double nL = fma(l2, fma(4.0, d2, -d3), fma(c1, fma(2.0, d2, d1), m12 * fma(5.0, d1, -2.0 * d0)));
    const double nR = fma(r0, fma(4.0, d1, -d0), fma(c1, fma(2.0, d1, d2), m01 * fma(5.0, d2, -2.0 * d3)));
    L = fma(nL, frcp(6.0 * ((m12 + c1) + l2)), v2);
    R = fma(-nR, frcp(6.0 * ((m01 + c1) + r0)), v2);
}

// FP32 version: the product form would overflow single precision for
// large-valued fields (q ~ (dp^2)^2), so the weights use reciprocals (of
// q^2 / 16, which overflows no earlier than the indicators' own squares).
__device__ __forceinline__ void weno5_pair(float v0, float v1, float v2, float v3, float v4, float eps, float& L,
                                           float& R) {
    const float d0 = v1 - v0, d1 = v2 - v1, d2 = v3 - v2, d3 = v4 - v3;
    const float t0 = d1 - d0, t1 = d2 - d1, t2 = d3 - d2;
    const float s0 = fmaf(3.0f, d1, -d0), s1 = d1 + d2, s2 = fmaf(-3.0f, d2, d3);
    const float e = 4.0f * eps;
    const float q0 = fmaf(s0, s0, fmaf((13.0f / 3.0f) * t0, t0, e));
    const float q1 = fmaf(s1, s1, fmaf((13.0f / 3.0f) * t1, t1, e));
    const float q2 = fmaf(s2, s2, fmaf((13.0f / 3.0f) * t2, t2, e));
    const float a0 = frcp((0.0625f * q0) * q0), a1 = 6.0f * frcp((0.0625f * q1) * q1), a2 = frcp((0.0625f * q2) * q2);
    const float l2 = 3.0f * a2, r0 = 3.0f * a0;
    const float nL = fmaf(l2, fmaf(4.0f, d2, -d3), fmaf(a1, fmaf(2.0f, d2, d1), a0 * fmaf(5.0f, d1, -2.0f * d0)));
    const float nR = fmaf(r0, fmaf(4.0f, d1, -d0), fmaf(a1, fmaf(2.0f, d1, d2), a2 * fmaf(5.0f, d2, -2.0f * d3)));
    L = fmaf(nL, frcp(6.0f * ((a0 + a1) + l2)), v2);
    R = fmaf(-nR, frcp(6.0f * ((a2 + a1) + r0)), v2);
}

template <typename T>
__device__ __forceinline__ T trsqrt(T x) { return frsqrt_pos(x); }

template <typename T>
__device__ __forceinline__ T trcp(T x);
template <>
__device__ __forceinline__ double trcp<double>(double x) { return frcp(x); }
template <>
__device__ __forceinline__ float trcp<float>(float x) { return frcp(x); }


}  // namespace sifv
