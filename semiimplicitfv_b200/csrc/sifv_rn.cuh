// sifv_rn.cuh -- correctly rounded FP64 quotients without the division's
// branches, for the reference-ordered kernels.
//
// An IEEE division is compiled to a fast path, a range test and a branch to a
// slow path; each branch ends a basic block, so the six to eight independent
// divisions of a reconstruction run one dependent chain after the other.
// Here the quotients are fused multiply-adds only, the range test is one per
// reconstruction, and the compiler interleaves them.  The results are the
// IEEE quotients bit for bit.
#pragma once

#include <cuda_runtime.h>

namespace sifv {

// Correctly rounded a / b given y = RN(1 / b).  q0 = a y is within 1.5 ulp of
// a / b; one residual correction q1 = RN(q0 + RN(a - b q0) y) is faithful
// (within 1 ulp); Markstein's theorem (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Dev. 34(1), 1990: for y = RN(1 / b) and a faithful q, r = a - b q is exact
// and RN(q + r y) = RN(a / b)) makes the second correction the correctly
// rounded quotient.  Valid when |y| lies in [2^-450, 2^450] and a is +0 or
// |a| lies in [2^-450, 2^450] (quotient and residual then stay clear of
// overflow and gradual underflow; a = +0 gives +0 or -0 as a / b does).
// Callers check both with rn_fast_operand / rn_fast_recip and take the
// plain division otherwise.
__device__ __forceinline__ double div_markstein(double a, double b, double y) {
    const double q0 = a * y;
    const double q1 = fma(fma(-q0, b, a), y, q0);
    return fma(fma(-q1, b, a), y, q1);
}
// |x| in [2^-450, 2^450] (biased exponent 573..1473)
__device__ __forceinline__ bool rn_fast_recip(double x) {
    return ((unsigned)__double2hiint(x) & 0x7ff00000u) - 0x23d00000u <= 0x38400000u;
}
// the same, or x = +0
__device__ __forceinline__ bool rn_fast_operand(double x) {
    return rn_fast_recip(x) || (((unsigned)__double2hiint(x) | (unsigned)__double2loint(x)) == 0u);
}

// 1 / b of a positive normal b to within (1/2 + 2^-6) ulp: the hardware
// approximation (2^-20) and one third-order step, y (1 + e + e^2).
__device__ __forceinline__ double rcp_near(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    const double e = fma(-b, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// RN(1 / b) from rcp_near's y (Markstein 1990: the residual 1 - b y is exact
// and one correction rounds correctly unless every bit of b's significand is
// set; callers test the low word).
__device__ __forceinline__ double rcp_rn(double b, double y) { return fma(fma(-b, y, 1.0), y, y); }

// RN(a / b) for a = RN(1/10), RN(6/10) or RN(3/10) (the WENO5 linear weights)
// and y = rcp_near(b).  q1 is within (1/2 + 2^-51) ulp of a / b, so its
// residual is exact and q1 + r y is off by at most half an ulp times y's
// relative error before the final rounding.  With integer significands A, B a
// quotient lies t / (2 B) ulp from the nearest midpoint M / 2, where
// t = |2^(s+1) A - M B| is a positive integer (s = 52 or 53): the final
// rounding can only go wrong for t = 1 and B > 0.98 2^53, that is, for a
// divisor B of 2^(s+1) A +- 1 in that range.  These two significands have
// none (tests/test_markstein_quotient.py goes through the factorisations).
__device__ __forceinline__ double div_weight_rn(double a, double b, double y) { return div_markstein(a, b, y); }

}  // namespace sifv
