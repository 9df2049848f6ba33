// fp64.cuh -- FP64 reciprocal, square root and tests that spare the FP64 pipe.
//
// GB300 issues FP64 at 2 lanes per clock and SM (a warp instruction occupies the
// pipe for 16 cycles) against 128 lanes of FP32 and integer work, so the pair
// loops in FP64 are bound by the number of FP64 instructions. These helpers take
// their seeds from the FP32 special-function unit through integer moves of the
// bit patterns and spend FP64 instructions on the refinement alone.
//
// The refinements are the cubic members of Newton's family (Householder, "The
// Numerical Treatment of a Single Nonlinear Equation", 1970): with a seed of
// relative error e (|e| < 2^-21) one pass leaves e^3, below 2^-62. Arguments
// outside the seeds' range (|x| in [2^-100, 2^100]), zeros, infinities and NaN
// take the ordinary operators.
#pragma once

#include <math.h>

#include "common.cuh"

namespace azp
{
#ifdef __CUDACC__
AZP_D bool finite_bits(double a) { return (__double2hiint(a) & 0x7ff00000) != 0x7ff00000; }

// |x| in [2^-100, 2^100], by its exponent field
AZP_D bool seed_range(int hi) { return (uint32_t)((hi & 0x7fffffff) - 0x39b00000) < 0x0c800000u; }

// the float next to x towards zero (x in the seeds' range): the leading 24 bits
AZP_D float trunc_float(int hi, int lo)
{
    const uint32_t m = __funnelshift_l((uint32_t)lo, (uint32_t)(hi & 0x7fffffff) - 0x38000000u, 3);
    return __uint_as_float(m | ((uint32_t)hi & 0x80000000u));
}

// a normal float as a double, by its bits
AZP_D double widen(float f)
{
    const uint32_t b = __float_as_uint(f);
    return __hiloint2double((int)((((b & 0x7fffffffu) >> 3) + 0x38000000u) | (b & 0x80000000u)), (int)(b << 29));
}

// 1 / x: y (1 + e + e^2) with e = 1 - x y, for x (high word hi) in the seeds' range
AZP_D double rcp_in_range(double x, int hi)
{
    float s;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(trunc_float(hi, __double2loint(x))));
    const double y = widen(s);
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}
AZP_D double d_rcp(double x)
{
    const int hi = __double2hiint(x);
    if (!seed_range(hi)) return 1.0 / x;
    return rcp_in_range(x, hi);
}

// a / b: the product with 1 / b corrected once by its residual, which rounds it as the
// division does but for quotients within 2^-8 ulp or so of a rounding boundary and for |a|
// below 2^-900 (the bare product is an ulp off in 27 % of the cases). Where there is no
// residual (a infinite or not a number) the product stands.
AZP_D double d_div(double a, double b)
{
    const int hb = __double2hiint(b);
    if (!seed_range(hb)) return a / b;
    const double y = rcp_in_range(b, hb);
    const double q = a * y;
    const double r = fma(-q, b, a);
    return finite_bits(r) ? fma(r, y, q) : q;
}

// 1 / sqrt(x), x > 0: y (1 + e / 2 + 3 e^2 / 8) with e = 1 - x y^2
AZP_D double d_rsqrt(double x)
{
    const int hi = __double2hiint(x);
    if (hi < 0 || !seed_range(hi)) return 1.0 / sqrt(x);
    float s;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(trunc_float(hi, __double2loint(x))));
    const double y = widen(s);
    const double e = fma(-(x * y), y, 1.0);
    return fma(y * e, fma(e, 0.375, 0.5), y);
}

// sqrt(x) with 1 / sqrt(x) beside it; the root corrected once by its residual
AZP_D double d_sqrt(double x, double& rinv)
{
    const int hi = __double2hiint(x);
    if (hi < 0 || !seed_range(hi)) {
        const double r = sqrt(x);
        rinv = 1.0 / r;
        return r;
    }
    rinv = d_rsqrt(x);
    const double r = x * rinv;
    return fma(fma(-r, r, x), 0.5 * rinv, r);
}
AZP_D double d_sqrt(double x)
{
    double rinv;
    return d_sqrt(x, rinv);
}

// a < b for a >= 0 or NaN of either sign (false) and b >= 0, on the bit patterns. The
// comparison is unsigned: inf - inf gives a NaN whose sign bit is set, which a signed one
// would take for less than everything.
AZP_D bool less_nonneg(double a, double b)
{
    return (unsigned long long)__double_as_longlong(a) < (unsigned long long)__double_as_longlong(b);
}

// |a| > b for b >= 0 (NaN: true)
AZP_D bool magnitude_above(double a, double b)
{
    return (__double_as_longlong(a) & 0x7fffffffffffffffll) > __double_as_longlong(b);
}

// min_image1 that runs only where it changes v: |v| > L / 2. The body is out of
// line: as a predicated or speculated body its FP64 instructions would occupy the
// pipe for every pair.
static __device__ __noinline__ double min_image_call(double v, double L, double Linv) { return min_image1(v, L, Linv); }
AZP_D double min_image_if(double v, double half, double L, double Linv)
{
    if (magnitude_above(v, half)) v = min_image_call(v, L, Linv);
    return v;
}

// r^2 of a pair and whether it is below rcutsq as the oracle decides it (rsq_exact).
// cut: rcutsq and rcutsq (1 - 2^-48). Below the second the fused sum, within
// 2^-51 of the rounded one, decides; the pairs between take the exact one.
static __device__ __noinline__ bool below_exact(double dx, double dy, double dz, double rcutsq)
{
    return rsq_exact(dx, dy, dz) < rcutsq;
}
AZP_D bool pair_inside(double dx, double dy, double dz, const double* cut, double& rsq)
{
    rsq = fma(dz, dz, fma(dy, dy, dx * dx));
    return less_nonneg(rsq, cut[1]) || below_exact(dx, dy, dz, cut[0]);
}
AZP_D double cut_low(double rcutsq) { return rcutsq * (1.0 - 3.552713678800501e-15); }
#endif
}  // namespace azp
