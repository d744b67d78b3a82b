// Stresses of a triangular dislocation in an elastic half-space (Nikkhoo &
// Walter 2015, GJI; MIT-licensed original by M. Nikkhoo), one (receiver, source)
// pair per thread, as the shear and normal stiffness of the pair.  Follows
// scripts/Functions_TDstressHS.jl (TDstressHS :2-130, TDstressFS :133-286,
// TDstress_HarFunc :289-335, TensTrans :338, CoordTrans :365, trimodefinder :393,
// TDSetupS :433, AngSetupFSC_S :467); the strains of the angular dislocations
// (AngDisStrain :577, AngDisStrainFSC :654-1034) are in tdhs_terms.cuh.  Points
// on a TD edge give NaN, as in the reference (:262-267).
//
// Shear and normal stiffness of one (receiver, source) pair of triangles in a
// half-space, projected on the receiver's unit vectors
// as it is formed:
//   Kn = n . S n,  Ks = v . S n,  S = 2 mu E + lambda tr(E)
// With E = A e A^T for a part's local axes A, n . E n = n' . e n' with n' = A^T n
// (and v . E n likewise), so each part's strains are contracted where they are
// formed with the receiver's vectors in the part's axes, instead of being
// rotated back tensor by tensor (eleven rotations of ~75 operations a pair).
//
// What depends on the source alone -- axes, angles and their sines, the sides'
// geometry -- is formed by the *_consts functions, once per source where many
// receivers share it, by the reference's operations to the last bit: the stress
// is sensitive to the last bits of the angles (an ulp in one moves an entry by
// up to 3e-10 of the row's largest).  So are the local coordinates, distances
// and the sums r + z that cancel near a side's axis.
#pragma once
#include <math_constants.h>

#include "qdfn_internal.h"
#include "tdhs_terms.cuh"

namespace qdfn {
namespace tdhs {

// r = A * (x1,x2,x3) with A a 3x3 given column-major.
__device__ void coord_trans(double x1, double x2, double x3, const double* A, double r[3]) {
    r[0] = A[0] * x1 + A[3] * x2 + A[6] * x3;
    r[1] = A[1] * x1 + A[4] * x2 + A[7] * x3;
    r[2] = A[2] * x1 + A[5] * x2 + A[8] * x3;
}

__device__ void cross3(const double a[3], const double b[3], double c[3]) {
    c[0] = a[1] * b[2] - a[2] * b[1];
    c[1] = a[2] * b[0] - a[0] * b[2];
    c[2] = a[0] * b[1] - a[1] * b[0];
}
__device__ double norm3(const double a[3]) { return sqrt(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]); }

// Full space: the triangle in its own axes (normal, strike, dip), origin P2
struct TriFs {
    double ax[9];                    // rows: normal, strike, dip
    double P2[3], p1[3], p3[3];
    double sv[3][2];                 // strike and dip components of -e13, e12, e23
    double sinA[3], cosA[3];         // of (vertex angle - pi)
    double den;                      // trimodefinder's denominator
};
// Free-surface correction of one side
struct TriSide {
    double c, s;                     // horizontal direction of the side
    double yAB[3], b[3];
    double sinB[2], cosB[2], cotB[2], icosB[2];   // of beta, of pi - beta
    bool skip;                       // a vertical side
};

__device__ inline void unit_axes(const double P1[3], const double P2[3], const double P3[3], bool image, double N[3],
                                 double S[3], double D[3]) {
    double d21[3] = {P2[0] - P1[0], P2[1] - P1[1], P2[2] - P1[2]};
    double d31[3] = {P3[0] - P1[0], P3[1] - P1[1], P3[2] - P1[2]};
    cross3(d21, d31, N);
    const double nn = norm3(N);
    for (int k = 0; k < 3; ++k) N[k] = N[k] / nn;
    const double eZ[3] = {0, 0, 1};
    cross3(eZ, N, S);
    if (norm3(S) == 0) {             // a horizontal triangle
        S[0] = 0; S[1] = N[2]; S[2] = 0;
        if (image && P1[2] > 0)
            for (int k = 0; k < 3; ++k) S[k] = -S[k];
    }
    const double ns = norm3(S);
    for (int k = 0; k < 3; ++k) S[k] = S[k] / ns;
    cross3(N, S, D);
}

__device__ inline void fs_consts(const double P1[3], const double P2[3], const double P3[3], TriFs& f) {
    double N[3], S[3], D[3];
    unit_axes(P1, P2, P3, true, N, S, D);
    const double At[9] = {N[0], S[0], D[0], N[1], S[1], D[1], N[2], S[2], D[2]};
    for (int k = 0; k < 3; ++k) { f.ax[k] = N[k]; f.ax[3 + k] = S[k]; f.ax[6 + k] = D[k]; f.P2[k] = P2[k]; }
    coord_trans(P1[0] - P2[0], P1[1] - P2[1], P1[2] - P2[2], At, f.p1);
    coord_trans(P3[0] - P2[0], P3[1] - P2[1], P3[2] - P2[2], At, f.p3);
    double e12[3], e13[3], e23[3];
    const double d[3] = {0 - f.p1[0], 0 - f.p1[1], 0 - f.p1[2]};
    double n = norm3(d);
    for (int k = 0; k < 3; ++k) e12[k] = d[k] / n;
    const double d2[3] = {f.p3[0] - f.p1[0], f.p3[1] - f.p1[1], f.p3[2] - f.p1[2]};
    n = norm3(d2);
    for (int k = 0; k < 3; ++k) e13[k] = d2[k] / n;
    const double d3[3] = {f.p3[0] - 0, f.p3[1] - 0, f.p3[2] - 0};
    n = norm3(d3);
    for (int k = 0; k < 3; ++k) e23[k] = d3[k] / n;
    const double ang[3] = {acos(e12[0] * e13[0] + e12[1] * e13[1] + e12[2] * e13[2]),
                           acos(-e12[0] * e23[0] + -e12[1] * e23[1] + -e12[2] * e23[2]),
                           acos(e23[0] * e13[0] + e23[1] * e13[1] + e23[2] * e13[2])};
    for (int k = 0; k < 3; ++k) {
        f.sinA[k] = sin(-CUDART_PI + ang[k]);
        f.cosA[k] = cos(-CUDART_PI + ang[k]);
    }
    for (int k = 0; k < 2; ++k) { f.sv[0][k] = -e13[1 + k]; f.sv[1][k] = e12[1 + k]; f.sv[2][k] = e23[1 + k]; }
    const double x1 = f.p1[1], y1 = f.p1[2], x3 = f.p3[1], y3 = f.p3[2];   // trimodefinder's p1, p3; p2 = 0
    f.den = (0 - y3) * (x1 - x3) + (x3 - 0) * (y1 - y3);
}

// The slip in the fixed axes, for the sides' corrections
__device__ inline void slip_fixed(const double P1[3], const double P2[3], const double P3[3], double Ss, double Ds,
                                  double b[3]) {
    double N[3], S[3], D[3];
    unit_axes(P1, P2, P3, false, N, S, D);
    const double A[9] = {N[0], N[1], N[2], S[0], S[1], S[2], D[0], D[1], D[2]};
    coord_trans(0.0, Ss, Ds, A, b);
}
__device__ inline void side_consts(const double PA[3], const double PB[3], const double bxyz[3], TriSide& t) {
    const double SV[3] = {PB[0] - PA[0], PB[1] - PA[1], PB[2] - PA[2]};
    const double beta = acos(-SV[2] / norm3(SV));
    t.skip = fabs(beta) < 1e-16 || fabs(CUDART_PI - beta) < 1e-16;
    const double h[3] = {SV[0], SV[1], 0};
    const double n1 = norm3(h);
    t.c = h[0] / n1;
    t.s = h[1] / n1;
    t.yAB[0] = t.c * SV[0] + t.s * SV[1]; t.yAB[1] = t.s * SV[0] + -t.c * SV[1]; t.yAB[2] = -SV[2];
    t.b[0] = t.c * bxyz[0] + t.s * bxyz[1]; t.b[1] = t.s * bxyz[0] + -t.c * bxyz[1]; t.b[2] = -bxyz[2];
#pragma unroll 1
    for (int k = 0; k < 2; ++k) {
        const double g = k == 0 ? beta : CUDART_PI - beta;
        t.sinB[k] = sin(g);
        t.cosB[k] = cos(g);
        t.cotB[k] = 1.0 / tan(g);
        t.icosB[k] = 1.0 / t.cosB[k];
    }
}

// Receiver
struct TriRecv {
    double X[3], n[3], v[3];
};
// Running contractions: n . E n, v . E n and tr E
struct TriSum {
    double nn = 0, vn = 0, tr = 0;
};
__device__ __forceinline__ void contract(const double e[6], double n0, double n1, double n2, double v0, double v1,
                                         double v2, double f, TriSum& s) {
    // e scaled by f; t = e n
    const double t0 = fma(e[0], n0, fma(e[3], n1, e[4] * n2));
    const double t1 = fma(e[3], n0, fma(e[1], n1, e[5] * n2));
    const double t2 = fma(e[4], n0, fma(e[5], n1, e[2] * n2));
    s.nn = fma(f, fma(t0, n0, fma(t1, n1, t2 * n2)), s.nn);
    s.vn = fma(f, fma(t0, v0, fma(t1, v1, t2 * v2)), s.vn);
    s.tr = fma(f, e[0] + e[1] + e[2], s.tr);
}

// Full-space part (TDstressFS): false on the triangle's edge, where the
// reference gives NaN
__device__ __forceinline__ bool fs_part(const TriFs& f, const TriRecv& R, double Ss, double Ds, double nu, double M2,
                                        double scale, TriSum& s) {
    const double dx = R.X[0] - f.P2[0], dy = R.X[1] - f.P2[1], dz = R.X[2] - f.P2[2];
    const double x = f.ax[0] * dx + f.ax[1] * dy + f.ax[2] * dz;
    const double y = f.ax[3] * dx + f.ax[4] * dy + f.ax[5] * dz;
    const double z = f.ax[6] * dx + f.ax[7] * dy + f.ax[8] * dz;
    const double n0 = fma(f.ax[0], R.n[0], fma(f.ax[1], R.n[1], f.ax[2] * R.n[2]));
    const double n1 = fma(f.ax[3], R.n[0], fma(f.ax[4], R.n[1], f.ax[5] * R.n[2]));
    const double n2 = fma(f.ax[6], R.n[0], fma(f.ax[7], R.n[1], f.ax[8] * R.n[2]));
    const double v0 = fma(f.ax[0], R.v[0], fma(f.ax[1], R.v[1], f.ax[2] * R.v[2]));
    const double v1 = fma(f.ax[3], R.v[0], fma(f.ax[4], R.v[1], f.ax[5] * R.v[2]));
    const double v2 = fma(f.ax[6], R.v[0], fma(f.ax[7], R.v[1], f.ax[8] * R.v[2]));
    // trimodefinder
    const double x1 = f.p1[1], y1 = f.p1[2], x3 = f.p3[1], y3 = f.p3[2];
    const double a = ((0 - y3) * (y - x3) + (x3 - 0) * (z - y3)) / f.den;
    const double b = ((y3 - y1) * (y - x3) + (x1 - x3) * (z - y3)) / f.den;
    const double c = 1 - a - b;
    double sgn = 1.0;
    if (a <= 0 && b > c && c > a) sgn = -1.0;
    if (b <= 0 && c > a && a > b) sgn = -1.0;
    if (c <= 0 && a > b && b > c) sgn = -1.0;
    if ((a == 0 && b >= 0 && c >= 0) || (a >= 0 && b == 0 && c >= 0) || (a >= 0 && b >= 0 && c == 0)) {
        if (x == 0) return false;
        sgn = 1.0;
    }
#pragma unroll 1
    for (int k = 0; k < 3; ++k) {
        const double s1 = sgn * f.sv[k][0], s2 = sgn * f.sv[k][1];
        const double py = k == 0 ? f.p1[1] : k == 1 ? 0.0 : f.p3[1], pz = k == 0 ? f.p1[2] : k == 1 ? 0.0 : f.p3[2];
        const double ry = y - py, rz = z - pz;
        double e[6];
        ang_strain(x, s2 * ry - s1 * rz, s1 * ry + s2 * rz, f.sinA[k], f.cosA[k], s2 * Ss - s1 * Ds,
                   s1 * Ss + s2 * Ds, nu, M2, e);
        contract(e, n0, fma(s2, n1, -s1 * n2), fma(s1, n1, s2 * n2), v0, fma(s2, v1, -s1 * v2), fma(s1, v1, s2 * v2),
                 scale, s);
    }
    return true;
}

// Free-surface correction of one side (AngSetupFSC_S)
__device__ __forceinline__ void side_part(const TriSide& t, const double PA[3], const double PB[3], const TriRecv& R,
                                          double nu, double N1, double M2, double scale, TriSum& s) {
    if (t.skip) return;
    const double dx = R.X[0] - PA[0], dy = R.X[1] - PA[1], dz = R.X[2] - PA[2];
    const double yA[3] = {t.c * dx + t.s * dy, t.s * dx + -t.c * dy, -dz};
    const bool first = yA[0] >= 0;
    const int k = first ? 1 : 0;
    const double f = first ? -1.0 : 1.0;
    const double n0 = f * fma(t.c, R.n[0], t.s * R.n[1]), n1 = f * fma(t.s, R.n[0], -t.c * R.n[1]), n2 = -R.n[2];
    const double v0 = f * fma(t.c, R.v[0], t.s * R.v[1]), v1 = f * fma(t.s, R.v[0], -t.c * R.v[1]), v2 = -R.v[2];
    // (with the local axes 0 and 1 turned round where `first`, the components
    // xz and yz that AngSetupFSC_S negates come out right)
#pragma unroll 1
    for (int end = 0; end < 2; ++end) {
        const double y0 = end ? yA[0] - t.yAB[0] : yA[0], y1 = end ? yA[1] - t.yAB[1] : yA[1];
        const double y2 = end ? yA[2] - t.yAB[2] : yA[2];
        double v[6];
        ang_strain_fsc(f * y0, f * y1, y2, t.sinB[k], t.cosB[k], t.cotB[k], t.icosB[k], f * t.b[0], f * t.b[1], t.b[2],
                       nu, N1, M2, end ? -PB[2] : -PA[2], v);
        contract(v, n0, n1, n2, v0, v1, v2, end ? scale : -scale, s);
    }
}

}  // namespace tdhs
}  // namespace qdfn
