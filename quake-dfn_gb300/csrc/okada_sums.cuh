// Okada (1992) DC3D displacement gradients of a rectangular dislocation as
// sums over its corners (Chinnery's notation), for pairs away from the
// singular lines of the source.
//
// The gradients are linear in a few corner functions -- 1/R, 1/R^3, X11, X32,
// Y11, Y32, ... and their products with xi -- whose coefficients (sin and cos
// of the dip, the medium, the slip, Q and Z) are the same at all four corners,
// and eta, Y~ and D~ only change between the two values of eta.  So the corner
// functions are summed first, over xi at each eta and then over eta with the
// powers of eta, Y~ and D~, and the nine (real source) or twelve (image)
// components are formed once from the sums, where okada.cuh forms every
// component at every corner for three slip directions (opening is zero here).
// The kernel is bound by the FP64 pipe, so what counts is the number of FP64
// operations: ~1,470 per pair of a fault network against ~7,540 (ncu, the
// source's and receiver's constants included; no divisions either: one
// reciprocal square root per corner gives R and 1/R, and 1/(R + xi),
// 1/(R + eta), 1/(R + D~) are reciprocals by Newton's iteration from the
// hardware's estimate).
//
// The formulas' own rounding is not small beside an entry: the corners nearly
// cancel in the far field, and more so where a factor blows up -- 1/cos^2(dip)
// in UB's K and J terms, R/(R + xi) and R/(R + eta) at receivers along or down
// a source's own plane.  The published formulas in FP64 carry an error of
// 1e-8 and more of a far block's largest entry there (113-bit arithmetic as the value),
// and another order of rounding gives another error of that size.  So that the
// entries are those of the published formulas in FP64 all the same:
//   R, R + xi, R + eta, X11, Y11 are formed and rounded as okada.cuh forms them
//     (to the last bit but for rare ties); the zeroing of |xi|, |eta|, |q| < 1e-6
//     inside R, Y~ and D~ alone is kept;
//   steep, not vertical sources (is_steep): K1, K3, J3, J6 at each corner by
//     okada.cuh's operations;
//   receivers along or down a source's plane, R/(R + xi) or R/(R + eta) above 64
//     at a corner of the real source (not `plain`): that source's part component
//     by component at each corner (real_corners), like okada.cuh; the image of
//     such a source lies far enough off;
//   where R + xi, R + eta or R + D~ is below 2^-30 R, or anything is not finite
//     (`ok`): the pair by okada.cuh.
// 2,200 blocks of 61 x 64 patches of a random network, the difference from
// okada.cuh over the block in the 2-norm, Kn and Ks apart: 6e-10 at most, 6e-12
// in the median (by corner sums alone 1.8e-8, and 5e-3 with sources at 89.9998
// degrees).
#pragma once
#include <cstring>

#include "okada.cuh"

namespace qdfn {
namespace okada {

#ifdef __CUDA_ARCH__
#define QDFN_HD __device__ __forceinline__
// estimates of 1/x and 1/sqrt(x) good to ~2^-20
QDFN_HD double rcp_est(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}
QDFN_HD double rsqrt_est(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}
#else
#define QDFN_HD inline __host__ __device__
QDFN_HD double rcp_est(double x) { return (double)(float)(1.0 / x); }
QDFN_HD double rsqrt_est(double x) { return (double)(float)(1.0 / sqrt(x)); }
#endif

// 1/x to about an ulp.  With an estimate y and e = 1 - x y, 1/x = y/(1 - e) =
// y (1 + e + e^2 + ...): the third-order member of Householder's family (A. S.
// Householder, The Numerical Treatment of a Single Nonlinear Equation, 1970);
// e^3 < 2^-60.
QDFN_HD double recip1(double x) {
    const double y = rcp_est(x), e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}
// R = sqrt(R2) and 1/R: the same family's 1/sqrt(R2) = y (1 - e)^(-1/2) =
// y (1 + e/2 + 3 e^2/8 + ...) with e = 1 - R2 y^2, then Newton's (Heron's) step
// for the root, r + (R2 - r^2)/(2 r), whose remainder is exact in one fused
// operation.
QDFN_HD void root(double R2, double& R, double& i1) {
    const double y = rsqrt_est(R2), e = fma(-(R2 * y), y, 1.0);
    i1 = fma(y * e, fma(e, 0.375, 0.5), y);
    const double r = R2 * i1;
    R = fma(fma(-r, r, R2), 0.5 * i1, r);
}
QDFN_HD long long dbits(double v) {
#ifdef __CUDA_ARCH__
    return __double_as_longlong(v);
#else
    long long b;
    memcpy(&b, &v, 8);
    return b;
#endif
}
// DCCON2's EPS rule, |v| < 1e-6 (compared as integers, like the checks below: an
// FP64 comparison takes the FP64 pipe)
QDFN_HD double zero_small(double v) {
    return (dbits(v) & 0x7fffffffffffffffll) < 0x3eb0c6f7a0b5ed8dll ? 0.0 : v;
}
QDFN_HD int hi_word(double v) { return (int)(dbits(v) >> 32); }
// x > 2^-BITS R (R >= 0; x NaN passes, R is checked)
template <int BITS = 30>
QDFN_HD bool well_above(double x, int hiR) {
    const int h = hi_word(x);
    return h > 0 && h > hiR - (BITS << 20);
}

// Per-source constants of the combination
struct Src {
    double SD, CD, iCD;          // iCD = 1/CD (unused where the dip is 90 degrees)
    double A1, A2, A3, A4, A5;   // DCCON0's ALP1..ALP5
    double D1, D2;               // strike and dip slip / 2 pi
    bool flat;                   // cos dip = 0
    bool steep;                  // is_steep(CD)
};

// Sources whose 1/cos^2(dip) is above 100 (84.3 to 95.7 degrees), the vertical
// ones apart.  At 80 degrees the difference from okada.cuh is that of 60.
QDFN_HD bool is_steep(double CD) { return CD != 0.0 && fabs(CD) < 0.1; }

// 1/x, correctly rounded but for rare ties (recip1 rounds otherwise one time in
// a hundred): Newton's step from a value within an ulp (Markstein 1990, cited at
// div_by in sim_device.cuh)
QDFN_HD double recip2(double x) {
    const double y = recip1(x);
    return fma(fma(-x, y, 1.0), y, y);
}
// x/d, correctly rounded but for rare ties: i = 1/d to about an ulp, then
// Markstein's correction of the quotient by its remainder
QDFN_HD double quotient(double x, double d, double i) {
    const double q = x * i;
    return fma(fma(-q, d, x), i, q);
}

// Corner functions, and differences of them over xi
struct Corner {
    double i1, i3, Xi3, X11, X32, Y11, XY11, XY32, xxY32, XxxY32;                       // both sources
    double i5, Xi5, xxi3, xxi5, Xxxi5, X53, Y32, xxY53, XxxY53, D11, XD11, D12, XD12;   // image
    double k1, k3, j3, j6;                                                              // image, |cos dip| < 0.1
};

template <bool IMG>
QDFN_HD Corner corner(const Src& s, double XI, double x, double ET, double e, double q2, double Q, double Y, double D,
                      bool& ok, bool& plain) {
    Corner c;
    const double x2 = x * x, e2 = e * e;
    const double R2 = x2 + e2 + q2;
    double R;
    root(R2, R, c.i1);
    const double RX = R + x, RE = R + e;
    const int hiR = hi_word(R);
    ok = ok && well_above(RX, hiR) && well_above(RE, hiR) && (unsigned)hiR < 0x46293e59u;   // R < 1e30
    const double i2 = c.i1 * c.i1;
    c.i3 = i2 * c.i1;
    c.Xi3 = XI * c.i3;
    if constexpr (!IMG) plain = plain && well_above<6>(RX, hiR) && well_above<6>(RE, hiR);
    c.X11 = recip1(R * RX);
    c.X32 = (R + RX) * c.X11 * c.X11 * c.i1;
    c.Y11 = recip1(R * RE);
    const double Y32 = (R + RE) * c.Y11 * c.Y11 * c.i1;
    c.XY11 = XI * c.Y11;
    c.XY32 = XI * Y32;
    c.xxY32 = x2 * Y32;
    c.XxxY32 = XI * c.xxY32;
    if constexpr (IMG) {
        const double RD = R + D;
        ok = ok && well_above(RD, hiR);
        const double iRD = recip1(RD);
        c.i5 = c.i3 * i2;
        c.Xi5 = XI * c.i5;
        c.xxi3 = x2 * c.i3;
        c.xxi5 = x2 * c.i5;
        c.Xxxi5 = XI * c.xxi5;
        const double R2x8 = 8.0 * R2, R9 = 9.0 * R;
        c.X53 = fma(R9, XI, fma(3.0, x2, R2x8)) * (c.X11 * c.X11 * c.X11) * i2;
        c.Y32 = Y32;
        const double Y53 = fma(R9, ET, fma(3.0, e2, R2x8)) * (c.Y11 * c.Y11 * c.Y11) * i2;
        c.xxY53 = x2 * Y53;
        c.XxxY53 = XI * c.xxY53;
        c.D11 = c.i1 * iRD;
        c.XD11 = XI * c.D11;
        c.D12 = c.D11 * iRD;
        c.XD12 = XI * c.D12;
        if (s.flat) {
            const double w = iRD * iRD;
            c.k1 = c.XD12;
            c.k3 = fma(x2, c.D12, -iRD);
            c.j3 = XI * w * fma(-q2, c.D11, 0.5);
            c.j6 = Y * w * fma(-x2, c.D11, 0.5);
        } else if (s.steep) {   // by okada.cuh's operations, in its order and rounding
            const double D11 = recip2(R * RD), Y11 = recip2(R * RE);
            const double j2 = quotient(XI * Y, RD, iRD) * D11, j5 = -(D + quotient(Y * Y, RD, iRD)) * D11;
            c.k1 = quotient(XI * (D11 - Y11 * s.SD), s.CD, s.iCD);
            c.k3 = quotient(Q * Y11 - Y * D11, s.CD, s.iCD);
            c.j3 = quotient(c.k1 - j2 * s.SD, s.CD, s.iCD);
            c.j6 = quotient(c.k3 - j5 * s.SD, s.CD, s.iCD);
        } else {
            c.k1 = c.k3 = c.j3 = c.j6 = 0.0;
        }
    }
    return c;
}

QDFN_HD Corner minus(const Corner& a, const Corner& b, bool img, bool kj) {
    Corner d;
    d.i1 = a.i1 - b.i1; d.i3 = a.i3 - b.i3; d.Xi3 = a.Xi3 - b.Xi3; d.X11 = a.X11 - b.X11; d.X32 = a.X32 - b.X32;
    d.Y11 = a.Y11 - b.Y11; d.XY11 = a.XY11 - b.XY11; d.XY32 = a.XY32 - b.XY32; d.xxY32 = a.xxY32 - b.xxY32;
    d.XxxY32 = a.XxxY32 - b.XxxY32;
    if (img) {
        d.i5 = a.i5 - b.i5; d.Xi5 = a.Xi5 - b.Xi5; d.xxi3 = a.xxi3 - b.xxi3; d.xxi5 = a.xxi5 - b.xxi5;
        d.Xxxi5 = a.Xxxi5 - b.Xxxi5; d.X53 = a.X53 - b.X53; d.Y32 = a.Y32 - b.Y32; d.xxY53 = a.xxY53 - b.xxY53;
        d.XxxY53 = a.XxxY53 - b.XxxY53; d.D11 = a.D11 - b.D11; d.XD11 = a.XD11 - b.XD11; d.D12 = a.D12 - b.D12;
        d.XD12 = a.XD12 - b.XD12;
        if (kj) { d.k1 = a.k1 - b.k1; d.k3 = a.k3 - b.k3; d.j3 = a.j3 - b.j3; d.j6 = a.j6 - b.j6; }
    }
    return d;
}

// Corner sums of both sources
struct Sums {
    double i1 = 0, i3 = 0, Di3 = 0, Yi3 = 0, Ei3 = 0, Xi3 = 0, XDi3 = 0, XYi3 = 0, Y11 = 0, XY11 = 0, XY32 = 0,
           xxY32 = 0, XxxY32 = 0, X11 = 0, DX11 = 0, YX11 = 0, EX11 = 0, YX32 = 0, DX32 = 0, EYX32 = 0, EDX32 = 0;
};
QDFN_HD void add(Sums& s, const Corner& c, double ET, double Y, double D) {
    s.i1 += c.i1; s.i3 += c.i3; s.Xi3 += c.Xi3; s.Y11 += c.Y11; s.XY11 += c.XY11; s.XY32 += c.XY32;
    s.xxY32 += c.xxY32; s.XxxY32 += c.XxxY32; s.X11 += c.X11;
    s.Di3 = fma(D, c.i3, s.Di3); s.Yi3 = fma(Y, c.i3, s.Yi3); s.Ei3 = fma(ET, c.i3, s.Ei3);
    s.XDi3 = fma(D, c.Xi3, s.XDi3); s.XYi3 = fma(Y, c.Xi3, s.XYi3);
    s.DX11 = fma(D, c.X11, s.DX11); s.YX11 = fma(Y, c.X11, s.YX11); s.EX11 = fma(ET, c.X11, s.EX11);
    const double yx = Y * c.X32, dx = D * c.X32;
    s.YX32 += yx; s.DX32 += dx;
    s.EYX32 = fma(ET, yx, s.EYX32); s.EDX32 = fma(ET, dx, s.EDX32);
}

// Gradients of Okada_DC3D_Vector (UXX,UYX,UZX,UXY,UYY,UZY,UXZ,UYZ,UZZ) for
// slip (DISL1, DISL2, 0): real_sums() sets U to the real source's part (UA),
// image_sums() adds the image's (UA + UB and UC).  False where the pair is too
// close to a singular line; `plain` as in the notes above, else unchanged.
QDFN_HD bool real_sums(const Src& s, double X, double Y, double Z, double DEPTH, double AL, double AW, double U[9],
                       bool& plain) {
    const double SD = s.SD, CD = s.CD, A1 = s.A1, A2 = s.A2, D1 = s.D1, D2 = s.D2;
    const double XP = X + AL, XM = X - AL, xp = zero_small(XP), xm = zero_small(XM);
    bool ok = true;
    const double d = DEPTH + Z, P = Y * CD + d * SD, Q = Y * SD - d * CD, q = zero_small(Q), q2 = q * q;
    Sums t;
#pragma unroll 1
    for (int K = 0; K < 2; ++K) {
        const double ET = K == 0 ? P + AW : P - AW, e = zero_small(ET);
        const double Yt = e * CD + q * SD, Dt = e * SD - q * CD;
        const Corner a = corner<false>(s, K == 0 ? XP : XM, K == 0 ? xp : xm, ET, e, q2, Q, Yt, Dt, ok, plain);
        const Corner b = corner<false>(s, K == 0 ? XM : XP, K == 0 ? xm : xp, ET, e, q2, Q, Yt, Dt, ok, plain);
        add(t, minus(a, b, false, false), ET, Yt, Dt);
    }
    const double EY = fma(-q, t.Yi3, SD * t.i1), EZ = fma(q, t.Di3, CD * t.i1);
    const double FY = fma(SD, t.xxY32, t.Di3), FZ = fma(CD, t.xxY32, t.Yi3);
    const double XFY = fma(SD, t.XxxY32, t.XDi3), XFZ = fma(CD, t.XxxY32, t.XYi3);
    const double GY = fma(2 * SD, t.X11, -q * t.YX32), GZ = fma(2 * CD, t.X11, q * t.DX32);
    const double EGY = fma(2 * SD, t.EX11, -q * t.EYX32), EGZ = fma(2 * CD, t.EX11, q * t.EDX32);
    const double QY = Q * t.Y11, QX3 = A2 * Q * t.Xi3, EY2 = A2 * EY, EZ2 = A2 * EZ;
    const double a0 = D1 * (-A1 * QY - A2 * Q * t.xxY32) - D2 * QX3;
    const double a1 = -D1 * QX3 + D2 * (-0.5 * QY - A2 * Q * t.Ei3);
    const double a2 = D1 * (A1 * t.XY11 + A2 * q2 * t.XY32) + D2 * (A1 * t.i1 + A2 * q2 * t.i3);
    const double a3 = D1 * (A1 * SD * t.XY11 + A2 * XFY + 0.5 * t.DX11) + D2 * EY2;
    const double a4 = D1 * EY2 + D2 * (A1 * t.DX11 + 0.5 * SD * t.XY11 + A2 * EGY);
    const double a5 = D1 * (A1 * fma(CD, t.i1, SD * QY) - A2 * Q * FY) + D2 * (A1 * t.YX11 - A2 * Q * GY);
    const double a6 = D1 * (A1 * CD * t.XY11 + A2 * XFZ + 0.5 * t.YX11) + D2 * EZ2;
    const double a7 = D1 * EZ2 + D2 * (A1 * t.YX11 + 0.5 * CD * t.XY11 + A2 * EGZ);
    const double a8 = D1 * (A1 * fma(-SD, t.i1, CD * QY) - A2 * Q * FZ) - D2 * (A1 * t.DX11 + A2 * Q * GZ);
    U[0] = -a0; U[1] = fma(-CD, a1, SD * a2); U[2] = -fma(SD, a1, CD * a2);
    U[3] = -a3; U[4] = fma(-CD, a4, SD * a5); U[5] = -fma(SD, a4, CD * a5);
    U[6] = a6; U[7] = fma(CD, a7, -SD * a8); U[8] = fma(SD, a7, CD * a8);
    return ok;
}

// real_sums() with the components formed at each corner, in the operations and the
// order of okada.cuh's ua() up to divisions by R, which are products with 1/R.
// ~770 operations against ~330.
QDFN_HD bool real_corners(const Src& s, double X, double Y, double Z, double DEPTH, double AL, double AW, double U[9]) {
    const double SD = s.SD, CD = s.CD, A1 = s.A1, A2 = s.A2, D1 = s.D1, D2 = s.D2;
    const double d = DEPTH + Z, P = Y * CD + d * SD, Q = Y * SD - d * CD, q = zero_small(Q), q2 = q * q;
    const double A2Q = A2 * Q;
    bool ok = true;
    for (int k = 0; k < 9; ++k) U[k] = 0.0;
#pragma unroll 1
    for (int j = 0; j < 4; ++j) {
        const double XI = (j & 1) ? X - AL : X + AL, ET = (j & 2) ? P - AW : P + AW;
        const double x = zero_small(XI), e = zero_small(ET), x2 = x * x;
        double R, i1;
        root(x2 + e * e + q2, R, i1);
        const double RX = R + x, RE = R + e;
        const int hiR = hi_word(R);
        ok = ok && well_above(RX, hiR) && well_above(RE, hiR) && (unsigned)hiR < 0x46293e59u;   // R < 1e30
        const double Yt = e * CD + q * SD, Dt = e * SD - q * CD, i3 = i1 * i1 * i1;
        const double X11 = recip1(R * RX), X32 = (R + RX) * X11 * X11 * i1;
        const double Y11 = recip1(R * RE), Y32 = (R + RE) * Y11 * Y11 * i1;
        const double XY = XI * Y11, QY = Q * Y11, xxY = x2 * Y32, Qi = Q * i3;
        const double qi = q * i3, EY = SD * i1 - Yt * qi, EZ = CD * i1 + Dt * qi;
        const double FY = Dt * i3 + xxY * SD, FZ = Yt * i3 + xxY * CD;
        const double GY = 2.0 * X11 * SD - Yt * q * X32, GZ = 2.0 * X11 * CD + Dt * q * X32;
        const double A2X = A2 * XI, A1XY = A1 * XY, aq = A2X * Qi, h = 0.5 * XY, A2E = A2 * ET;
        const double ad = A1 * Dt * X11, ay = A1 * Yt * X11, ey = A2 * EY, ez = A2 * EZ;
        const double a0 = D1 * (-A1 * QY - A2 * x2 * Q * Y32) - D2 * aq;
        const double a1 = -D1 * aq + D2 * (-0.5 * QY - A2E * Qi);
        const double a2 = D1 * (A1XY + A2X * q2 * Y32) + D2 * (A1 * i1 + A2 * q2 * i3);
        const double a3 = D1 * (A1XY * SD + A2X * FY + 0.5 * Dt * X11) + D2 * ey;
        const double a4 = D1 * ey + D2 * (ad + h * SD + A2E * GY);
        const double a5 = D1 * (A1 * (CD * i1 + QY * SD) - A2Q * FY) + D2 * (ay - A2Q * GY);
        const double a6 = D1 * (A1XY * CD + A2X * FZ + 0.5 * Yt * X11) + D2 * ez;
        const double a7 = D1 * ez + D2 * (ay + h * CD + A2E * GZ);
        const double a8 = D1 * (-A1 * (SD * i1 - QY * CD) - A2Q * FZ) + D2 * (-ad - A2Q * GZ);
        const double sg = j == 0 || j == 3 ? 1.0 : -1.0;
        U[0] = fma(-sg, a0, U[0]); U[1] = fma(sg, a2 * SD - a1 * CD, U[1]); U[2] = fma(-sg, a1 * SD + a2 * CD, U[2]);
        U[3] = fma(-sg, a3, U[3]); U[4] = fma(sg, a5 * SD - a4 * CD, U[4]); U[5] = fma(-sg, a4 * SD + a5 * CD, U[5]);
        U[6] = fma(sg, a6, U[6]); U[7] = fma(sg, a7 * CD - a8 * SD, U[7]); U[8] = fma(sg, a7 * SD + a8 * CD, U[8]);
    }
    return ok;
}

QDFN_HD bool image_sums(const Src& s, double X, double Y, double Z, double DEPTH, double AL, double AW, double U[9]) {
    const double SD = s.SD, CD = s.CD, A1 = s.A1, A2 = s.A2, A3 = s.A3, A4 = s.A4, A5 = s.A5, D1 = s.D1, D2 = s.D2;
    const double XP = X + AL, XM = X - AL, xp = zero_small(XP), xm = zero_small(XM);
    const bool kj = s.flat || s.steep;
    bool ok = true, none = true;
    const double d = DEPTH - Z, P = Y * CD + d * SD, Q = Y * SD - d * CD, q = zero_small(Q), q2 = q * q;
    Sums t;
    double Y32 = 0, xxi3 = 0, xxi5 = 0, Xxxi5 = 0, xxY53 = 0, XxxY53 = 0;
    double Ci3 = 0, CEi3 = 0, Ci5 = 0, CEi5 = 0, CYi5 = 0, CDi5 = 0, CXi5 = 0, CEXi5 = 0, CYXi5 = 0, CDXi5 = 0;
    double CX11 = 0, CX32 = 0, CEX32 = 0, CYX32 = 0, CDX32 = 0, YYX32 = 0, YDX32 = 0, DDX32 = 0;
    double CYX53 = 0, CDX53 = 0, CYEX53 = 0, CDEX53 = 0;
    double J2 = 0, J5 = 0, XD11 = 0, YD11 = 0, k1 = 0, k3 = 0, j3 = 0, j6 = 0;
#pragma unroll 1
    for (int K = 0; K < 2; ++K) {
        const double ET = K == 0 ? P + AW : P - AW, e = zero_small(ET);
        const double Yt = e * CD + q * SD, Dt = e * SD - q * CD, C = Dt + Z;
        const Corner a = corner<true>(s, K == 0 ? XP : XM, K == 0 ? xp : xm, ET, e, q2, Q, Yt, Dt, ok, none);
        const Corner b = corner<true>(s, K == 0 ? XM : XP, K == 0 ? xm : xp, ET, e, q2, Q, Yt, Dt, ok, none);
        const Corner c = minus(a, b, true, kj);
        add(t, c, ET, Yt, Dt);
        Y32 += c.Y32; xxi3 += c.xxi3; xxi5 += c.xxi5; Xxxi5 += c.Xxxi5; xxY53 += c.xxY53; XxxY53 += c.XxxY53;
        const double c3 = C * c.i3, c5 = C * c.i5, cx5 = C * c.Xi5;
        Ci3 += c3; CEi3 = fma(ET, c3, CEi3);
        Ci5 += c5; CEi5 = fma(ET, c5, CEi5); CYi5 = fma(Yt, c5, CYi5); CDi5 = fma(Dt, c5, CDi5);
        CXi5 += cx5; CEXi5 = fma(ET, cx5, CEXi5); CYXi5 = fma(Yt, cx5, CYXi5); CDXi5 = fma(Dt, cx5, CDXi5);
        CX11 = fma(C, c.X11, CX11);
        const double cx32 = C * c.X32, yx = Yt * c.X32, dx = Dt * c.X32;
        CX32 += cx32; CEX32 = fma(ET, cx32, CEX32); CYX32 = fma(Yt, cx32, CYX32); CDX32 = fma(Dt, cx32, CDX32);
        YYX32 = fma(Yt, yx, YYX32); YDX32 = fma(Yt, dx, YDX32); DDX32 = fma(Dt, dx, DDX32);
        const double cy53 = C * Yt * c.X53, cd53 = C * Dt * c.X53;
        CYX53 += cy53; CDX53 += cd53; CYEX53 = fma(ET, cy53, CYEX53); CDEX53 = fma(ET, cd53, CDEX53);
        J2 = fma(Yt, c.XD12, J2);
        J5 -= fma(Dt, c.D11, Yt * Yt * c.D12);
        XD11 += c.XD11; YD11 = fma(Yt, c.D11, YD11);
        if (kj) { k1 += c.k1; k3 += c.k3; j3 += c.j3; j6 += c.j6; }
    }
    // UB's K and J terms
    double K1, K3, J3, J6;
    if (s.flat) {
        K1 = Q * k1; K3 = SD * k3; J3 = j3; J6 = j6;
    } else if (s.steep) {
        K1 = k1; K3 = k3; J3 = j3; J6 = j6;
    } else {
        K1 = fma(-SD, t.XY11, XD11) * s.iCD;
        K3 = fma(Q, t.Y11, -YD11) * s.iCD;
        J3 = fma(-SD, J2, K1) * s.iCD;
        J6 = fma(-SD, J5, K3) * s.iCD;
    }
    const double K2 = fma(SD, K3, t.i1), K4 = fma(CD, t.XY11, -SD * K1);
    const double J1 = fma(CD, J5, -SD * J6), J4 = fma(SD, J3, fma(-CD, J2, -t.XY11));
    const double EY = fma(-q, t.Yi3, SD * t.i1), EZ = fma(q, t.Di3, CD * t.i1);
    const double FY = fma(SD, t.xxY32, t.Di3), FZ = fma(CD, t.xxY32, t.Yi3);
    const double XFY = fma(SD, t.XxxY32, t.XDi3), XFZ = fma(CD, t.XxxY32, t.XYi3);
    const double GY = fma(2 * SD, t.X11, -q * t.YX32), GZ = fma(2 * CD, t.X11, q * t.DX32);
    const double EGY = fma(2 * SD, t.EX11, -q * t.EYX32), EGZ = fma(2 * CD, t.EX11, q * t.EDX32);
    const double QY = Q * t.Y11, QX3 = Q * t.Xi3;
    // UA + UB, row by row: the shared functions' coefficients are A2 - 1
    // (or A1, 1/2 less 1), then UB's half-space terms
    const double Am = A2 - 1.0, w1 = A3 * SD, w2 = A3 * SD * CD;   // SDCD = SD * CD
    const double a0 = D1 * (-A1 * QY - Am * Q * t.xxY32 - w1 * J1) + D2 * (-Am * QX3 + w2 * J4);
    const double a1 = D1 * (-Am * QX3 - w1 * J2) + D2 * (0.5 * QY - Am * Q * t.Ei3 + w2 * J5);
    const double a2 = D1 * (A1 * t.XY11 + Am * q2 * t.XY32 - w1 * J3) +
                      D2 * (A1 * t.i1 + Am * q2 * t.i3 + w2 * J6);
    const double a3 = D1 * (A1 * SD * t.XY11 + Am * XFY - 0.5 * t.DX11 + w1 * (t.XY11 + J4)) +
                      D2 * (Am * EY + w2 * J1);
    const double a4 = D1 * (Am * EY + w1 * (t.i1 + J5)) +
                      D2 * (A1 * t.DX11 - 0.5 * SD * t.XY11 + Am * EGY + w2 * J2);
    const double a5 = D1 * (A1 * fma(CD, t.i1, SD * QY) - Am * Q * FY - w1 * (QY - J6)) +
                      D2 * (A1 * t.YX11 - Am * Q * GY + w2 * J3);
    const double a6 = D1 * (A1 * CD * t.XY11 + Am * XFZ - 0.5 * t.YX11 + w1 * K1) + D2 * (Am * EZ - w2 * K3);
    const double a7 = D1 * (Am * EZ + w1 * YD11) +
                      D2 * (A1 * t.YX11 - 0.5 * CD * t.XY11 + Am * EGZ - w2 * XD11);
    const double a8 = D1 * (A1 * fma(-SD, t.i1, CD * QY) - Am * Q * FZ + w1 * K2) -
                      D2 * (A1 * t.DX11 + Am * Q * GZ + w2 * K4);
    // UC
    const double H = Q * CD - Z, SD3 = 3.0 * SD, Q3 = 3.0 * Q;
    const double Y0 = t.Y11 - t.xxY32;
    const double Z32 = fma(SD, t.i3, -H * Y32), Z0 = Z32 - fma(SD3, xxi5, -H * xxY53);
    const double XZ32 = fma(SD, t.Xi3, -H * t.XY32), XZ0 = XZ32 - fma(SD3, Xxxi5, -H * XxxY53);
    const double xxZ32 = fma(SD, xxi3, -H * t.xxY32);
    const double XQQ = fma(Z, t.XY32, XZ32 + XZ0);
    const double XPY = fma(CD, t.Xi3, Q * SD * t.XY32), XPZ = fma(SD, t.Xi3, -Q * CD * t.XY32);
    const double XQQY = fma(3.0, CDXi5, -SD * XQQ), XQQZ = fma(3.0, CYXi5, fma(-CD, XQQ, Q * t.XY32));
    const double CDR = Ci3 + t.Di3, YY0 = fma(-CD, Y0, t.Yi3);
    const double CYQ = Q3 * CYi5, CDQ = Q3 * CDi5, QZ0 = Q * Z0;
    const double u = fma(SD, CDR, -CYQ), v = fma(CD, CDR, CDQ);   // CDR SD - C Y QR, CDR CD + C D QR
    const double c0 = D1 * (A4 * CD * t.XY11 - A5 * Q * XZ32) + D2 * (A4 * CD * t.i1 - SD * QY - A5 * Q * Ci3);
    const double c1 = D1 * (A4 * fma(CD, t.i1, 2 * SD * QY) - A5 * Q * Ci3) + D2 * (A4 * t.YX11 - A5 * Q * CEX32);
    const double c2 = D1 * (A4 * CD * QY - A5 * (CEi3 - Z * t.Y11 + xxZ32)) +
                      D2 * (-t.DX11 - SD * t.XY11 - A5 * fma(-q2, CX32, CX11));
    const double c3 = D1 * (A4 * CD * Y0 - A5 * QZ0) +
                      D2 * (-A4 * CD * t.Xi3 + A5 * Q3 * CXi5 + SD * Q * t.XY32);
    const double c4 = D1 * (-A4 * fma(CD, t.Xi3, 2 * Q * SD * t.XY32) + A5 * Q3 * CXi5) +
                      D2 * (-A4 * t.Yi3 + A5 * Q3 * CEi5);
    const double c5 = D1 * (-A4 * CD * Q * t.XY32 + A5 * fma(3.0, CEXi5, -XQQ)) +
                      D2 * (t.Di3 - SD * Y0 + A5 * fma(-3.0 * q2, Ci5, Ci3));
    const double c6 = -D1 * (A4 * CD * XPY + A5 * XQQY) + D2 * (-A4 * t.Ei3 + SD * SD * Y0 - A5 * u);
    const double c7 = D1 * (2 * A4 * SD * fma(-SD, Y0, t.Di3) - CD * t.Yi3 - A5 * (u - t.Ei3)) +
                      D2 * (A4 * (t.X11 - YYX32) - A5 * (fma(2 * Q, CD * CX32, CDX32) - Q * CYEX53));
    const double c8 = D1 * (-A4 * Q * t.i3 + SD * YY0 + A5 * (v - SD * fma(CD, Y0, QZ0))) +
                      D2 * (SD * XPY + YDX32 + A5 * (fma(2 * Q, SD * CX32, CYX32) - q2 * CYX53));
    const double c9 = D1 * (A4 * CD * XPZ - A5 * XQQZ) + D2 * (-Q * t.i3 + SD * CD * Y0 - A5 * v);
    const double c10 = D1 * (2 * A4 * SD * YY0 + CD * t.Di3 - A5 * v) +
                       D2 * (A4 * YDX32 - A5 * (fma(-2 * Q, SD * CX32, CYX32) + Q * CDEX53));
    const double c11 = D1 * (CD * YY0 - A5 * (u - SD * SD * Y0 + CD * QZ0)) +
                       D2 * (-SD * XPZ + t.X11 - DDX32 - A5 * (fma(-2 * Q, CD * CX32, CDX32) - q2 * CDX53));
    const double p1 = fma(Z, c4, a1), p2 = fma(Z, c5, a2), m1 = fma(-Z, c4, a1), m2 = fma(-Z, c5, a2);
    const double p4 = fma(Z, c7, a4), p5 = fma(Z, c8, a5), m4 = fma(-Z, c7, a4), m5 = fma(-Z, c8, a5);
    const double p7 = fma(Z, c10, a7) + c1, p8 = fma(Z, c11, a8) + c2;
    const double m7 = fma(-Z, c10, a7) - c1, m8 = fma(-Z, c11, a8) - c2;
    U[0] += fma(Z, c3, a0);
    U[1] += fma(CD, p1, -SD * p2);
    U[2] += fma(SD, m1, CD * m2);
    U[3] += fma(Z, c6, a3);
    U[4] += fma(CD, p4, -SD * p5);
    U[5] += fma(SD, m4, CD * m5);
    U[6] += fma(Z, c9, a6) + c0;
    U[7] += fma(CD, p7, -SD * p8);
    U[8] += fma(SD, m7, CD * m8);
    return ok;
}

}  // namespace okada
}  // namespace qdfn
