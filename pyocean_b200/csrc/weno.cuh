// WENO5 face reconstruction in FP64 with the reference's arithmetic.
//
// The face value of an upwind-ordered 5-cell stencil v1..v5 (v3 = the upwind cell) follows
// core/dynamics/sigma_baroclinic.py:204-233 (`_wval`): WENO5-Z (Borges et al. 2008, tau5 = |b2 - b0|, eps 1e-40) or
// WENO5-JS (Jiang & Shu 1996, eps 1e-6) when all five cells are valid, WENO3 (eps 1e-6) when v2..v4 are, else the
// upwind value.  Every operation is written in the reference's evaluation order; the translation unit is compiled
// with -fmad=false so no multiply-add is contracted, which makes the result bit-identical to the reference's
// IEEE-754 FP64 evaluation.  Where fewer instructions give the same correctly rounded numbers, they are used
// (weno5_full, exactdiv.cuh; x * 0.5 is x / 2 exactly).
#pragma once

#include "common.cuh"
#include "exactdiv.cuh"

namespace po {

// The full WENO5 value with IEEE divisions, the reference's operations one by one: the stencils outside the ranges
// of weno5_full's short divisions (not inlined: they are rare, and inlined their registers would count everywhere).
__device__ __noinline__ double weno5_ieee(double v1, double v2, double v3, double v4, double v5, bool z_variant)
{
    if ((__double_as_longlong(v1) | __double_as_longlong(v2) | __double_as_longlong(v3) | __double_as_longlong(v4) |
         __double_as_longlong(v5)) == 0)
        return 0.0;                                  // every cell +0: so is every term
    const double q0 = (2.0 * v1 - 7.0 * v2 + 11.0 * v3) / 6.0;
    const double q1 = (-v2 + 5.0 * v3 + 2.0 * v4) / 6.0;
    const double q2 = (2.0 * v3 + 5.0 * v4 - v5) / 6.0;
    const double c1312 = 13.0 / 12.0;
    double d = v1 - 2.0 * v2 + v3, e = v1 - 4.0 * v2 + 3.0 * v3;
    const double b0 = c1312 * (d * d) + 0.25 * (e * e);
    d = v2 - 2.0 * v3 + v4;
    e = v2 - v4;
    const double b1 = c1312 * (d * d) + 0.25 * (e * e);
    d = v3 - 2.0 * v4 + v5;
    e = 3.0 * v3 - 4.0 * v4 + v5;
    const double b2 = c1312 * (d * d) + 0.25 * (e * e);
    double a0, a1, a2;
    if (z_variant) {
        const double tau = fabs(b2 - b0);
        a0 = 0.1 * (1.0 + tau / (1e-40 + b0));
        a1 = 0.6 * (1.0 + tau / (1e-40 + b1));
        a2 = 0.3 * (1.0 + tau / (1e-40 + b2));
    } else {
        const double s0 = 1e-6 + b0, s1 = 1e-6 + b1, s2 = 1e-6 + b2;
        a0 = 0.1 / (s0 * s0);
        a1 = 0.6 / (s1 * s1);
        a2 = 0.3 / (s2 * s2);
    }
    return (a0 * q0 + a1 * q1 + a2 * q2) / (a0 + a1 + a2);
}

// The constants of weno5_full whose low word is not zero, in constant memory: an FP64 instruction takes them as an
// operand there, while an immediate would first be moved into a register pair.
static __constant__ double kWeno[6] = {13.0 / 12.0, 1e-40, 1e-6, 0.1, 0.6, 0.3};

// WENO5 value of a stencil whose five cells are valid: the numbers of weno5_ieee in fewer instructions.
//  * A product by a power of two is exact, so a - 2 b, a - 4 b and a + 0.25 b are one fma each with the same rounding
//    (0.25 (e e) may round in the subnormal range; beside the epsilon 1e-40 or 1e-6 that changes no bit).
//  * A face costs 73 FP64 instructions and about as many others; with four IEEE divisions and their checks it cost 92
//    and 225 (ncu, face pass of 384 x 384 x 50, T and S: 634 -> 379 warp instructions per warp of 64 faces with the
//    stencil classes, 317 -> 242 us).
//  * x / 6 takes three operations (div6_short), the four quotients a reciprocal and one correction each
//    (recip_newton, quot_rn), without range checks of their own.
//  * One check per face covers all of them.  The weights' denominators are below 2^800 (JS: their roots below 2^50):
//    with the epsilon below them, the reciprocals and quotients are normal numbers, and a quotient too small for an
//    exact residual is added to 1 and vanishes.  The face value is in [2^-800, 2^900): then the last residual is exact,
//    no term was infinite or NaN, and a candidate x / 6 below 2^-1019, which div6_short may round differently, is too
//    small against the others to be seen.  No divisor is near two (four of 2^18 faces have one).  Anything else, and the
//    value 0, goes to weno5_ieee.
template <bool ZV>
__device__ __forceinline__ double weno5_full(double v1, double v2, double v3, double v4, double v5)
{
    const double q0 = div6_short(fma(2.0, v1, -(7.0 * v2)) + 11.0 * v3);
    const double q1 = div6_short(fma(2.0, v4, 5.0 * v3 - v2));
    const double q2 = div6_short(fma(2.0, v3, 5.0 * v4) - v5);
    const double c1312 = kWeno[0];
    const double w3 = 3.0 * v3;
    double d = fma(-2.0, v2, v1) + v3, e = fma(-4.0, v2, v1) + w3;
    const double b0 = fma(0.25, e * e, c1312 * (d * d));
    d = fma(-2.0, v3, v2) + v4;
    e = v2 - v4;
    const double b1 = fma(0.25, e * e, c1312 * (d * d));
    d = fma(-2.0, v4, v3) + v5;
    e = fma(-4.0, v4, w3) + v5;
    const double b2 = fma(0.25, e * e, c1312 * (d * d));
    const double eps = ZV ? kWeno[1] : kWeno[2];
    const double g0 = eps + b0, g1 = eps + b1, g2 = eps + b2;
    const unsigned top = max(max((unsigned)__double2hiint(g0), (unsigned)__double2hiint(g1)),
                             (unsigned)__double2hiint(g2));
    constexpr unsigned lim = (1023u + (ZV ? 800u : 50u)) << 20;
    // the divisors of the three weights; their checks first, so that no bits of them stay in registers for the end (kept
    // there they cost a step at 512 x 512 x 50 1.5 % in spills)
    const double s0 = ZV ? g0 : g0 * g0, s1 = ZV ? g1 : g1 * g1, s2 = ZV ? g2 : g2 * g2;
    bool slow = max(max(near_two_bits(s0), near_two_bits(s1)), near_two_bits(s2)) >= NEAR_TWO || top >= lim;
    double a0, a1, a2;
    if (ZV) {
        const double tau = fabs(b2 - b0);
        a0 = kWeno[3] * (1.0 + quot_rn(tau, s0, recip_newton(s0)));
        a1 = kWeno[4] * (1.0 + quot_rn(tau, s1, recip_newton(s1)));
        a2 = kWeno[5] * (1.0 + quot_rn(tau, s2, recip_newton(s2)));
    } else {
        a0 = quot_rn(kWeno[3], s0, recip_newton(s0));
        a1 = quot_rn(kWeno[4], s1, recip_newton(s1));
        a2 = quot_rn(kWeno[5], s2, recip_newton(s2));
    }
    const double den = a0 + a1 + a2;
    slow = slow || near_two_bits(den) >= NEAR_TWO;
    const double w = quot_rn(a0 * q0 + a1 * q1 + a2 * q2, den, recip_newton(den));
    const unsigned size = (unsigned)__double2hiint(w) & 0x7fffffffu;
    constexpr unsigned lo = (1023u - 800u) << 20, hi = (1023u + 900u) << 20;
    if (size - lo >= hi - lo || slow) return weno5_ieee(v1, v2, v3, v4, v5, ZV);
    return w;
}

// WENO3 value of a stencil of which the middle three cells are valid.
__device__ __forceinline__ double weno3_value(double v2, double v3, double v4)
{
    const double c0 = (-v2 + 3.0 * v3) * 0.5, c1 = (v3 + v4) * 0.5;
    const double s0 = 1e-6 + (v3 - v2) * (v3 - v2), s1 = 1e-6 + (v4 - v3) * (v4 - v3);
    const double e0 = (1.0 / 3.0) / (s0 * s0);
    const double e1 = (2.0 / 3.0) / (s1 * s1);
    return (e0 * c0 + e1 * c1) / (e0 + e1);
}

// ---------------------------------------------------------------------------------------------------------------
// Mixed-precision WENO5 face value: the smoothness indicators, the nonlinear weights and the weighted candidate
// run in FP32 on the differences of the stencil from the upwind cell (formed in FP64, then rounded), normalised by
// their largest magnitude s; the result is added back to the FP64 upwind value: face = v3 + s * w(d/s).  Every
// quantity of the scheme is a function of these differences (q_r - v3 and beta_r are linear / quadratic forms in
// them), so the FP32 rounding acts on the local variation only (relative face error ~1e-7 of s, not of v3).  The
// normalisation keeps beta_r in [0, 40] so FP32 cannot overflow; WENO5-Z's epsilon, 1e-40 in FP64, becomes 1e-30 on
// the normalised scale (both are negligible against any non-zero beta_r, and both give the same limit when a
// beta_r vanishes).  Stencils whose variation is outside what the FP32 forms represent safely (s below 1e-30 or,
// for the absolute-epsilon forms WENO5-JS and WENO3, above 1e8) keep the FP64 arithmetic (weno5_ieee).

template <bool ZV>
__device__ __forceinline__ double weno5_full_mixed(double v1, double v2, double v3, double v4, double v5)
{
    const float e1 = (float)(v1 - v3), e2 = (float)(v2 - v3), e4 = (float)(v4 - v3), e5 = (float)(v5 - v3);
    const float sc = fmaxf(fmaxf(fabsf(e1), fabsf(e2)), fmaxf(fabsf(e4), fabsf(e5)));
    if (sc == 0.f) {
        if (v1 == v3 && v2 == v3 && v4 == v3 && v5 == v3) return v3;      // flat: every candidate is v3
        return weno5_ieee(v1, v2, v3, v4, v5, ZV);
    }
    if (!(sc > 1e-30f) || (!ZV && sc > 1e8f))
        return weno5_ieee(v1, v2, v3, v4, v5, ZV);
    const float inv = 1.f / sc;
    const float d1 = e1 * inv, d2 = e2 * inv, d4 = e4 * inv, d5 = e5 * inv;
    const float c1312 = 13.f / 12.f;
    float t = fmaf(-2.f, d2, d1), u = fmaf(-4.f, d2, d1);
    const float b0 = fmaf(c1312 * t, t, 0.25f * u * u);
    t = d2 + d4;
    u = d2 - d4;
    const float b1 = fmaf(c1312 * t, t, 0.25f * u * u);
    t = fmaf(-2.f, d4, d5);
    u = fmaf(-4.f, d4, d5);
    const float b2 = fmaf(c1312 * t, t, 0.25f * u * u);
    const float tau = fabsf(b2 - b0);
    float a0, a1, a2;
    if (ZV) {
        a0 = 0.1f * (1.f + __fdividef(tau, 1e-30f + b0));
        a1 = 0.6f * (1.f + __fdividef(tau, 1e-30f + b1));
        a2 = 0.3f * (1.f + __fdividef(tau, 1e-30f + b2));
    } else {
        // JS weights use an absolute epsilon (1e-6): un-normalise beta (s <= 1e8 keeps the squares finite)
        const float s2 = sc * sc;
        const float g0 = fmaf(s2, b0, 1e-6f), g1 = fmaf(s2, b1, 1e-6f), g2 = fmaf(s2, b2, 1e-6f);
        a0 = __fdividef(0.1f, g0 * g0);
        a1 = __fdividef(0.6f, g1 * g1);
        a2 = __fdividef(0.3f, g2 * g2);
    }
    // 6 (q_r - v3) / s
    const float p0 = fmaf(2.f, d1, -7.f * d2), p1 = fmaf(2.f, d4, -d2), p2 = fmaf(5.f, d4, -d5);
    const float num = fmaf(a0, p0, fmaf(a1, p1, a2 * p2));
    const float den = 6.f * (a0 + a1 + a2);
    return v3 + (double)(sc * __fdividef(num, den));
}

// WENO3 (absolute eps 1e-6): candidates v3 - e2/2 and v3 + e4/2
__device__ __forceinline__ double weno3_value_mixed(double v2, double v3, double v4)
{
    const float d2 = (float)(v2 - v3), d4 = (float)(v4 - v3);
    if (!(fmaxf(fabsf(d2), fabsf(d4)) <= 1e8f)) return weno3_value(v2, v3, v4);
    const float g0 = fmaf(d2, d2, 1e-6f), g1 = fmaf(d4, d4, 1e-6f);
    const float w0 = __fdividef(1.f / 3.f, g0 * g0), w1 = __fdividef(2.f / 3.f, g1 * g1);
    const float corr = __fdividef(fmaf(w1, 0.5f * d4, -w0 * 0.5f * d2), w0 + w1);
    return v3 + (double)corr;
}

template <bool ZV, bool MIX>
__device__ __forceinline__ double weno5_any(double v1, double v2, double v3, double v4, double v5)
{
    if (MIX) return weno5_full_mixed<ZV>(v1, v2, v3, v4, v5);
    return weno5_full<ZV>(v1, v2, v3, v4, v5);
}

template <bool MIX>
__device__ __forceinline__ double weno3_any(double v2, double v3, double v4)
{
    if (MIX) return weno3_value_mixed(v2, v3, v4);
    return weno3_value(v2, v3, v4);
}

}  // namespace po
