// Logarithm, exponential and reciprocal of the friction solves, for arguments
// that the caller has checked (fm_log: positive and normal; fm_exp: |x| <= 700).
//
// Logarithm and exponential are table-driven after P. T. P. Tang (Table-driven
// implementation of the logarithm function, ACM TOMS 16(4), 1990; of the
// exponential function, ACM TOMS 15(2), 1989): a short table takes the argument
// to |r| <= 2^-8 (2^-7.5 for the exponential), and a short polynomial does the
// rest.  The FP64 pipe is this part's narrowest (a 64th of FP32), and an FP64
// operation or a conversion between FP32 and FP64 takes ~62 clocks of a chain
// and 16 of the SM's pipe, so the split is chosen to issue as few of both as
// possible: the polynomials' last terms are evaluated in FP32 beside the FP64
// chain (their rounding is below 2^-55, absolute for the logarithm and relative
// for the exponential), and the conversions are shifts and masks on the integer
// pipe.  Errors: the logarithm's below 3 x 2^-53 of the result + 2^-55, the
// exponential's below 1.3 x 2^-53 of it.  In a chain (clocks): logarithm 560 and
// exponential 691 (681 and 872 with conversion instructions); CUDA's log 1936 and
// exp 1650.
#pragma once
#include "friction_tables.cuh"

namespace qdfn {
namespace sim {

// x to the nearest FP32 (ties away from zero); below 2^-126 in magnitude to zero,
// |x| < 2^127
__device__ __forceinline__ float to_float(double x) {
    const unsigned h = (unsigned)__double2hiint(x), a = h & 0x7fffffffu;
    const unsigned l = (unsigned)__double2loint(x);
    const unsigned m = __funnelshift_l(l, a - 0x38000000u, 3) + ((l >> 28) & 1u);
    return __uint_as_float((a < 0x38100000u ? 0u : m) | (h & 0x80000000u));
}
// f as FP64; subnormals to zero, finite f
__device__ __forceinline__ double to_double(float f) {
    const unsigned u = __float_as_uint(f), a = u & 0x7fffffffu;
    const unsigned h = (a >> 3) + 0x38000000u;
    return __hiloint2double((int)((a < 0x00800000u ? 0u : h) | (u & 0x80000000u)), (int)(a < 0x00800000u ? 0u : u << 29));
}
__device__ __forceinline__ double to_double(int k) {
    return __hiloint2double(0x43300000, k ^ 0x80000000) - __hiloint2double(0x43300000, 0x80000000);
}

// 1/x to about an ulp, x normal and 1/x normal.  With an estimate y and e = 1 - x y,
// 1/x = y/(1 - e) = y (1 + e + e^2 + ...): the third-order member of Householder's
// family (A. S. Householder, The Numerical Treatment of a Single Nonlinear
// Equation, 1970), which leaves e^3 < 2^-60 of the hardware's 2^-20 estimate.
__device__ __forceinline__ double fm_rcp(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

__device__ __forceinline__ double fm_log(double x) {
    // x = 2^k m, m in [0x1.6a09ep-1, 0x1.6a09ep0); interval j of its significand
    const int ix = __double2hiint(x) - 0x3fe6a09e;
    const int k = ix >> 20;
    const double m = __hiloint2double(__double2hiint(x) - (k << 20), __double2loint(x));
    const double2 t = __ldg(kLogTab + ((ix >> 13) & 127));
    const double r = fma(m, t.x, -1.0);                       // |r| <= 2^-8
    const double r2 = r * r;
    const float f = to_float(r);
    // ln(1 + r) = r + r^2 (-1/2 + r/3 - r^2/4 + ...): the terms from r^2/4 on in FP32
    const float tail = f * f * fmaf(f, fmaf(f, fmaf(f, 0.14285715f, -0.16666667f), 0.2f), -0.25f);
    const double u = fma(r, 0.33333333333333331, -0.5) + to_double(tail);
    return fma(to_double(k), 0.69314718055994529, t.y) + fma(r2, u, r);
}

__device__ __forceinline__ double fm_exp(double x) {
    // x = n ln2/64 + r, n rounded in FP32 (|r| <= 2^-7.5 up to that rounding)
    const int n = __float2int_rn(to_float(x) * 92.332482f);
    const double nd = to_double(n);
    const double r = fma(nd, 0x1.718432a1b0e26p-41, fma(nd, -0x1.62e42ff000000p-7, x));   // ln2/64 = hi + lo
    const double T = __ldg(kExpTab + (n & 63));
    const double r2 = r * r;
    const float f = to_float(r);
    const float tail = f * f * fmaf(f, fmaf(f, 0.0013888889f, 0.0083333333f), 0.041666668f);
    const double u = fma(r, 0.16666666666666666, 0.5) + to_double(tail);
    const double y = fma(T, fma(r2, u, r), T);
    return __hiloint2double(__double2hiint(y) + ((n >> 6) << 20), __double2loint(y));
}

}  // namespace sim
}  // namespace qdfn
