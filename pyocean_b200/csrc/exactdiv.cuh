// Correctly rounded division of binary64 values by the constants 3 and 6 in three FP64 operations, and by a divisor
// whose reciprocal is at hand.
//
// The reference divides by 6 three times per WENO face ((2v1 - 7v2 + 11v3)/6 ...) and by 3 in the RK3 flux
// combination.  An IEEE division is an iterative sequence of ~10 FP64 instructions; for these constant divisors
// the same correctly rounded result comes from one multiplication and two FMAs:
//
//   y  = RN(1/3)                      (a compile-time constant)
//   q  = RN(x * y)                    |q - x/3| <= ulp(x/3): x*y = (x/3)(1 + d), |d| = 2^-54, plus one rounding
//   r  = fma(-q, 3, x)                exact: x and 3q are multiples of ulp(x/3)/2 and |x - 3q| <= 3 ulp(x/3)
//   q' = RN(q + r * y) = RN(x/3)      the FMA's argument is x/3 + (x/3 - q) d, within 2^-54 ulp of x/3, while
//                                     x/3 is at least ulp/6 away from every rounding midpoint (x - 3m is an odd
//                                     multiple of ulp/2 for any midpoint m), so both round to the same double.
//
// This is Markstein's correction step for division with a correctly rounded reciprocal (P. Markstein, "IA-64 and
// Elementary Functions", 2000, ch. 8) specialised to the divisor 3; RN(1/6) is RN(1/3) / 2, so it holds for 6 too.
// Nonzero arguments near the ends of the exponent range (and inf, NaN) take the IEEE division, so the result equals
// `x / 3.0` / `x / 6.0` for every input.  tests/hostcore checks the identity on the host.
#pragma once

#ifdef __CUDACC__
#define PO_XD __host__ __device__ __forceinline__
#else
#include <math.h>
#define PO_XD inline
#endif

namespace po {

// x / 6 in three operations, for the callers that check their result's range themselves: correctly rounded, signed
// zeros included, for |x| = 0 or in [2^-1019, 2^1024); below that the quotient is subnormal and may round the other way
// on a tie, and an infinite x gives NaN.  The residual is formed as 6 q - x so that a zero keeps its sign.
PO_XD double div6_short(double x)
{
    const double y = 1.0 / 6.0;
    const double q = x * y;
    return fma(fma(6.0, q, -x), -y, q);
}

PO_XD double div3_short(double x)
{
    const double y = 1.0 / 3.0;
    const double q = x * y;
    return fma(fma(3.0, q, -x), -y, q);
}

#ifdef __CUDACC__
// Whether div6_short / div3_short round x as the division does: x is zero, or |x| in [2^-1000, 2^1000).
__device__ __forceinline__ bool short_range(double x)
{
    const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu;
    return h - (23u << 20) < (2000u << 20) || (h | (unsigned)__double2loint(x)) == 0u;
}

static __device__ __noinline__ double div_ieee(double x, double y) { return x / y; }
#endif

// x / 3 and x / 6 for every x: the short form in its range, else the division.
PO_XD double div3_exact(double x)
{
#ifdef __CUDA_ARCH__
    const double q = div3_short(x);
    return short_range(x) ? q : div_ieee(x, 3.0);
#else
    const double ax = fabs(x);
    return ax >= 0x1p-899 && ax <= 0x1p899 ? div3_short(x) : x / 3.0;
#endif
}

PO_XD double div6_exact(double x)
{
#ifdef __CUDA_ARCH__
    const double q = div6_short(x);
    return short_range(x) ? q : div_ieee(x, 6.0);
#else
    const double ax = fabs(x);
    return ax >= 0x1p-898 && ax <= 0x1p899 ? div6_short(x) : x / 6.0;
#endif
}

#ifdef __CUDACC__
// 1 / b for 2^-1000 < b < 2^1000 without range checks, for quot_rn: PTX's approximate reciprocal (rcp.approx.ftz.f64: it
// reads the upper 20 mantissa bits of b and gives as many; relative error e below 2^-18) and two Newton-Raphson steps
// y (1 + e) (P. Markstein, "IA-64 and Elementary Functions", 2000, ch. 8).  A step squares the relative error, so the
// result lies within 2^-72 of 1 / b before its own rounding: within (1/2 + eta) ulp with eta = 2^-19.
__device__ __forceinline__ double recip_newton(double b)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    y = fma(y, fma(-b, y, 1.0), y);
    return fma(y, fma(-b, y, 1.0), y);
}

// RN(a / b), b > 0, for quotients and residuals that stay normal: |a| >= 2^-960, |a / b| in [2^-1000, 2^1000]; or a = +-0,
// whose sign the residual's order keeps.  y: RN(1 / b), or recip_newton(b) where b is not near_two.
//
// One correction of q = RN(a y) by its exact residual r = a - b q (Markstein's, the same chapter): q + r y differs from
// a / b by (r / b)(b y - 1).  Scaled to b in [1, 2), a / b in [1, 2): a / b is no midpoint of two doubles and lies at least
// 2^-105 / b from the nearest, M.  Only a distance below 2^-100 can matter (the difference is smaller than that); then
// |a / b - q| is half an ulp, 2^-53 (three halves would take |a y - a / b| of an ulp, so b > 2 (1 - 2 eta)), and with
// |b y - 1| <= b (1 + 2 eta) 2^-54 the difference is at most b (1 + 2 eta) 2^-107, less than 2^-105 / b where
// b^2 (1 + 2 eta) < 4: for every b with eta = 0, else for b < 2 - 2^-18.
__device__ __forceinline__ double quot_rn(double a, double b, double y)
{
    const double q = a * y;
    return fma(fma(b, q, -a), -y, q);
}

// Whether recip_newton(b) may not serve quot_rn: the upper 18 mantissa bits of b are ones.  near_two_bits of several
// divisors can be compared by their maximum.
__device__ __forceinline__ unsigned near_two_bits(double b) { return (unsigned)__double2hiint(b) << 12; }
constexpr unsigned NEAR_TWO = 0xffffc000u;

// Divisors shared by several quotients: y = 1 / b once, three operations per quotient; 0 for a b outside
// [2^-400, 2^400] or near two.  quotient(a, b, y) is a / b; it takes the division for y = 0 and for an a that is neither 0
// nor in [2^-500, 2^500].
__device__ __forceinline__ double shared_recip(double b)
{
    const bool in = (unsigned)__double2hiint(b) - (623u << 20) < (800u << 20);         // b > 0 too
    return in && near_two_bits(b) < NEAR_TWO ? recip_newton(b) : 0.0;
}

__device__ __forceinline__ double quotient(double a, double b, double y)
{
    const unsigned h = (unsigned)__double2hiint(a) & 0x7fffffffu;
    const bool in = h - (523u << 20) < (1000u << 20) || (h | (unsigned)__double2loint(a)) == 0u;
    const double q = quot_rn(a, b, y);
    return in && y != 0.0 ? q : div_ieee(a, b);
}
#endif

}  // namespace po
