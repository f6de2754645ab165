// Correctly rounded division of binary64 values by the constants 3 and 6 in three FP64 operations, and by a divisor
// whose correctly rounded reciprocal is at hand.
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
// RN(1 / b) for 2^-1000 < b < 2^1000 without range checks: the hardware's approximate reciprocal (relative error e
// about 2^-20: it reads the upper 20 mantissa bits of b and gives as many), one cubic step y (1 + e + e^2), which leaves
// e^3 and the rounding (below one ulp), and Markstein's final step, after which y is the correctly rounded reciprocal
// unless b's mantissa is all ones and y came out below (P. Markstein, "IA-64 and Elementary Functions", 2000, ch. 8).
// For that mantissa 1 / b lies just above the middle of two doubles; the bit set below the approximation's last one
// makes it an overestimate there, e^3 negative, and y the upper neighbour, which the final step keeps.
__device__ __forceinline__ double recip_rn(double b)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    y = __hiloint2double(__double2hiint(y), (int)0x80000000);
    double e = fma(-b, y, 1.0);
    y = fma(y, fma(e, e, e), y);
    e = fma(-b, y, 1.0);
    return fma(y, e, y);
}

// RN(a / b), b > 0, from y = RN(1 / b) (the same chapter: the quotient a y is within one ulp, its residual is exact and
// one correction rounds correctly), for quotients and residuals that stay normal: |a| >= 2^-960, |a / b| in
// [2^-1000, 2^1000]; or a = +-0, whose sign the residual's order keeps.
__device__ __forceinline__ double quot_rn(double a, double b, double y)
{
    const double q = a * y;
    return fma(fma(b, q, -a), -y, q);
}

// Divisors shared by several quotients: y = RN(1 / b) once, three operations per quotient; 0 for a b outside
// [2^-400, 2^400].  quotient(a, b, y) is a / b; it takes the division for y = 0 and for an a that is neither 0 nor in
// [2^-500, 2^500].
__device__ __forceinline__ double shared_recip(double b)
{
    const bool in = (unsigned)__double2hiint(b) - (623u << 20) < (800u << 20);         // b > 0 too
    return in ? recip_rn(b) : 0.0;
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
