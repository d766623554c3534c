// FP64 reciprocal, quotient, square root and exponential of the solves, for
// operands the caller has shown to be in range (no zero, infinity, NaN,
// subnormal, overflow or underflow anywhere), without special cases.
//
// The solves are bound by instruction issue: of the 896 instructions the IR
// solve issued per layer and warp, 334 were FP64 arithmetic and most of the
// rest the operand tests, branches and conversions of 13 divisions, 2 square
// roots and 2 exponentials.  These forms have none; the solves test the few
// operands that can leave the range (integer compares on the high words, one
// flag per system) and send such systems through the general code.
//
// Every result is the correctly rounded one, so it equals the operators
// `/` and sqrt() -- and the CPU oracle -- bit for bit.  "Near a midpoint" below
// is a value so close to the middle of two doubles that the error stated could
// change its rounding; u is the distance of the two.
//   rcp_n   Newton-Raphson, y <- y + y (1 - b y), from the hardware approximation
//           (rcp.approx.ftz.f64): two steps leave a relative error of 2^-80
//           before the second one's rounding, upwards, so y is 1/b or up to one
//           u above it.  The third step is P. Markstein's ("Computation of
//           elementary functions on the IBM RISC System/6000 processor", IBM J.
//           Res. Dev. 34(1), 1990): 1 - b y is exact, and y + y (1 - b y) lies
//           b (y - 1/b)^2 below 1/b.  For a b in [1, 2) 1/b is N 2^-106 / b from
//           its midpoint, N a whole number, not 0, so it matters for N = 1 .. 4
//           alone; there y, rounded up, is u/2 = 2^-54 above 1/b, and b^2 / 4 < N.
//           (Rounded to nearest, y would be u/2 below 1/b for the significand of
//           all ones -- 1 - W0 COSB and 1 + ALPHA of a thin layer -- and stay.)
//   quot    q = a y, q' = q + y (a - b q) with y = 1/b rounded (same paper).
//           q' before its rounding is off a/b by |a/b - q| |b y - 1|, at most
//           3 b 2^-108 for a < b in [1, 2), u = 2^-53.  a/b is N 2^-106 / b from
//           its midpoint, so it matters for |N| <= 3 alone; there a y, off by
//           less than u, rounds to one of the two doubles beside a/b, u/2 from
//           it, and b^2 / 4 < |N|.  For a >= b both u and the distance are twice
//           as large, the error of a y is below u/2, and the same holds.  So
//           quotients over one divisor share its reciprocal;
//   sqrt_n  Goldschmidt's coupled iterations for sqrt(x) and 1/(2 sqrt(x)) from
//           rsqrt.approx.ftz.f64, then g' = g + h (x - g g) (P. Markstein,
//           "Software division and square root using Goldschmidt's algorithms",
//           6th Conference on Real Numbers and Computers, 2004).
// tests/test_arithmetic_gpu.py compares them with CUDA's operators, at random
// operands and at those whose exact results lie nearest to midpoints.
// exp_r is mgcm_rt_exp (include/mgcm_rt_math.h), operation for operation:
// rounding to an integer by adding 1.5 2^52, S_j = RN(lead + trail) being
// lead itself, the scaling by 2^m an addition to the exponent.
#pragma once
#include "../../include/mgcm_rt_math.h"

namespace mgcm {

__device__ __forceinline__ unsigned hi32(double x) { return (unsigned)__double2hiint(x); }

// True when |x| is outside [2^-300, 2^300): zero, infinity and NaN included.
__device__ __forceinline__ bool out_of_range(double x) {
    return (hi32(x) & 0x7fffffffu) - 0x2d300000u >= 0x25800000u;
}

// 1 / b, b > 0.
__device__ __forceinline__ double rcp_n(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    y = __fma_rn(y, __fma_rn(-b, y, 1.0), y);
    y = __fma_ru(y, __fma_rn(-b, y, 1.0), y);
    return __fma_rn(__fma_rn(-b, y, 1.0), y, y);
}

// 1 / b for a divisor of either sign (the iterate is rounded up in magnitude).
__device__ __forceinline__ double rcp_s(double b) {
    const double y = rcp_n(fabs(b));
    return __hiloint2double(__double2hiint(y) | (__double2hiint(b) & (int)0x80000000u), __double2loint(y));
}

// a / b, y = 1 / b rounded (rcp_n, rcp_s).
__device__ __forceinline__ double quot(double a, double b, double y) {
    const double q = __dmul_rn(a, y);
    return __fma_rn(__fma_rn(-b, q, a), y, q);
}

__device__ __forceinline__ double sqrt_n(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double g = __dmul_rn(x, y), h = __dmul_rn(0.5, y);
    double r = __fma_rn(-h, g, 0.5);
    g = __fma_rn(g, r, g);
    h = __fma_rn(h, r, h);
    r = __fma_rn(-h, g, 0.5);
    g = __fma_rn(g, r, g);
    h = __fma_rn(h, r, h);
    return __fma_rn(__fma_rn(-g, g, x), h, g);
}

// exp(x) for |x| < 700.
__device__ __forceinline__ double exp_r(double x) {
    const double INV_L = 0x1.71547652b82fep+5, L1 = 0x1.62e42fee00000p-6, L2 = 0x1.a39ef35793c76p-38;
    const double A1 = 0x1.0000000000000p-1, A2 = 0x1.5555555555555p-3;
    const double A3 = 0x1.5555555555555p-5, A4 = 0x1.1111111111111p-7;
    const double A5 = 0x1.6c16c16c16c17p-10;
    const double RINT = 0x1.8p+52;
    const double t = __dadd_rn(__dmul_rn(x, INV_L), RINT);
    const int n = __double2loint(t);
    const double nf = __dsub_rn(t, RINT);
    const double r1 = __fma_rn(-nf, L1, x);   // nf L1 is exact: 32 + 16 bits
    const double r2 = -__dmul_rn(nf, L2);
    const double r = __dadd_rn(r1, r2);
    double q = __dadd_rn(A4, __dmul_rn(r, A5));
    q = __dadd_rn(A3, __dmul_rn(r, q));
    q = __dadd_rn(A2, __dmul_rn(r, q));
    q = __dadd_rn(A1, __dmul_rn(r, q));
    q = __dmul_rn(__dmul_rn(r, r), q);
    const double p = __dadd_rn(r1, __dadd_rn(r2, q));
    const double *tab = mgcm_rt_exp_tab_dev + (n & 31);
    const double sl = __ldg(tab), st = __ldg(tab + 32);
    const double v = __dadd_rn(sl, __dadd_rn(st, __dmul_rn(sl, p)));
    return __hiloint2double(__double2hiint(v) + ((n >> 5) << 20), __double2loint(v));
}

}  // namespace mgcm
