// Triangular-patch stiffness kernel (TDstressHS), one thread per
// (receiver, source) pair, FP64.  Follows StiffnessMatrix_ByParts_Calculation_Tri
// (scripts/Functions_BuildInputFile.jl:551-594).
#include <cuda_runtime.h>

#include <algorithm>

#include "assemble_kernels.h"
#include "qdfn_internal.h"
#include "tdhs.cuh"

namespace qdfn {
namespace {

constexpr int kMaxSrcTile = 8;   // sources of a block's turn, their constants in shared memory

// What the pairs of one source share
struct TriSource {
    tdhs::TriFs fs[2];       // the source and its image
    tdhs::TriSide side[3];
    double P[3][3], Ss, Ds;
    bool flat;               // all vertices at z = 0
};

// the medium and the scales of the strains
struct Medium {
    double G, lam, nu, N1, M2, c_fs, c_fsc;
};
__device__ __forceinline__ Medium medium(double G, double nu_in) {
    Medium m;
    m.G = G;
    m.lam = 2 * G * nu_in / (1 - 2 * nu_in);
    m.nu = 1 / (1 + m.lam / G) / 2;
    m.N1 = 1 - 2 * m.nu;
    m.M2 = 2 - 2 * m.nu;
    m.c_fs = 1 / (8 * CUDART_PI * (1 - m.nu));
    m.c_fsc = 1 / (4 * CUDART_PI * (1 - m.nu));
    return m;
}
// For a source in the free surface the image's shear stresses on horizontal
// planes count with the other sign, which is the receiver's vectors mirrored
// in the image part.
__device__ __forceinline__ tdhs::TriRecv image_receiver(const tdhs::TriRecv& R, bool flat) {
    tdhs::TriRecv Q = R;
    if (flat) {
        Q.n[2] = -Q.n[2];
        Q.v[2] = -Q.v[2];
    }
    return Q;
}
__device__ __forceinline__ tdhs::TriRecv receiver(const double* centre, const double* nhat, const double* shat,
                                                  int64_t r) {
    tdhs::TriRecv R;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        R.X[k] = centre[r * 3 + k];
        R.n[k] = nhat[r * 3 + k];
        R.v[k] = shat[r * 3 + k];
    }
    return R;
}
__device__ __forceinline__ void stiffness(const Medium& m, const tdhs::TriRecv& R, const tdhs::TriSum& s, bool edge,
                                          double& ks, double& kn) {
    const double nn = R.n[0] * R.n[0] + R.n[1] * R.n[1] + R.n[2] * R.n[2];
    const double vn = R.v[0] * R.n[0] + R.v[1] * R.n[1] + R.v[2] * R.n[2];
    kn = edge ? CUDART_NAN : fma(2 * m.G, s.nn, m.lam * s.tr * nn);
    ks = edge ? CUDART_NAN : fma(2 * m.G, s.vn, m.lam * s.tr * vn);
}

// A block takes kAsmThreads receivers, one per thread, and up to kMaxSrcTile
// sources at a time, whose constants (angles, sines, axes: ~3,000 FP64
// operations a source) its first three warps form in shared memory: the
// triangles on one, their images on the next, the sides on the third.  Bound by
// the FP64 pipe (~8,000 operations a pair; 43,500 with the published formulas'
// divisions and every constant formed per pair): 1,100 x 1,100 triangles 138.9 ->
// 21.1 ms.
__global__ void __launch_bounds__(kAsmThreads)
k_assemble_tri(int64_t n_src, const double* __restrict__ P1, const double* __restrict__ P2,
               const double* __restrict__ P3, const double* __restrict__ rake, int64_t n_recv,
               const double* __restrict__ centre, const double* __restrict__ nhat,
               const double* __restrict__ shat, double G, double nu, double* __restrict__ Ks,
               double* __restrict__ Kn, int64_t ld, int layout, int tile) {
    __shared__ TriSource src[kMaxSrcTile];
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool mine = r < n_recv;
    const Medium m = medium(G, nu);
    const tdhs::TriRecv R = receiver(centre, nhat, shat, mine ? r : 0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int64_t s0 = (int64_t)blockIdx.y * tile; s0 < n_src; s0 += (int64_t)gridDim.y * tile) {
        const int ns = (int)min((int64_t)tile, n_src - s0);
        __syncthreads();
        const int k = warp == 2 ? lane / 3 : lane;   // the source this lane works for
        if (warp < 3 && k < ns) {
            double P[3][3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                P[0][c] = P1[(s0 + k) * 3 + c];
                P[1][c] = P2[(s0 + k) * 3 + c];
                P[2][c] = P3[(s0 + k) * 3 + c];
            }
            const double Ss = -cosd_d(rake[s0 + k]), Ds = sind_d(rake[s0 + k]);
            TriSource& t = src[k];
            if (warp == 2) {
                const int j = lane % 3;
                double b[3];
                tdhs::slip_fixed(P[0], P[1], P[2], Ss, Ds, b);
                const double* A = j == 0 ? P[0] : j == 1 ? P[1] : P[2];
                const double* B = j == 0 ? P[1] : j == 1 ? P[2] : P[0];
                tdhs::side_consts(A, B, b, t.side[j]);
            } else {
                if (warp == 0) {
#pragma unroll
                    for (int c = 0; c < 9; ++c) t.P[c / 3][c % 3] = P[c / 3][c % 3];
                    t.Ss = Ss;
                    t.Ds = Ds;
                    t.flat = P[0][2] == 0 && P[1][2] == 0 && P[2][2] == 0;
                } else {
                    P[0][2] = -P[0][2]; P[1][2] = -P[1][2]; P[2][2] = -P[2][2];
                }
                tdhs::fs_consts(P[0], P[1], P[2], t.fs[warp]);
            }
        }
        __syncthreads();
        if (!mine) continue;
#pragma unroll 1
        for (int q = 0; q < ns; ++q) {
            const TriSource& t = src[q];
            tdhs::TriSum sum;
            bool in = true;
#pragma unroll 1
            for (int image = 0; image < 2; ++image)
                in = tdhs::fs_part(t.fs[image], image_receiver(R, image && t.flat), t.Ss, t.Ds, m.nu, m.M2, m.c_fs,
                                   sum) && in;
#pragma unroll 1
            for (int j = 0; j < 3; ++j)
                tdhs::side_part(t.side[j], t.P[j], t.P[j == 2 ? 0 : j + 1], R, m.nu, m.N1, m.M2, m.c_fsc, sum);
            const int64_t idx = layout == QDFN_LAYOUT_COL ? (s0 + q) * ld + r : r * ld + s0 + q;
            stiffness(m, R, sum, !in, Ks[idx], Kn[idx]);
        }
    }
}

// One thread per (receiver, source) pair of an index list: the entries that
// adaptive cross approximation asks for (rows and columns of admissible
// blocks) or any gathered set.  Same arithmetic as k_assemble_tri, with the
// source's constants formed by each thread part by part (~3,000 operations more
// a pair, but no thread waits for others').  256 blocks of 64 x 64: 155.7 -> 19.8
// ms.
__global__ void __launch_bounds__(kAsmThreads)
k_assemble_tri_pairs(int64_t npairs, const int64_t* __restrict__ ridx, const int64_t* __restrict__ sidx,
                     const double* __restrict__ P1, const double* __restrict__ P2, const double* __restrict__ P3,
                     const double* __restrict__ rake, const double* __restrict__ centre,
                     const double* __restrict__ nhat, const double* __restrict__ shat, double G, double nu,
                     double* __restrict__ Ks, double* __restrict__ Kn) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= npairs) return;
    const int64_t s = sidx[k];
    const Medium m = medium(G, nu);
    const tdhs::TriRecv R = receiver(centre, nhat, shat, ridx[k]);
    double P[3][3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        P[0][c] = P1[s * 3 + c];
        P[1][c] = P2[s * 3 + c];
        P[2][c] = P3[s * 3 + c];
    }
    const double Ss = -cosd_d(rake[s]), Ds = sind_d(rake[s]);
    const bool flat = P[0][2] == 0 && P[1][2] == 0 && P[2][2] == 0;
    tdhs::TriSum sum;
    bool in = true;
#pragma unroll 1
    for (int image = 0; image < 2; ++image) {
        const double sg = image ? -1.0 : 1.0;
        const double A[3] = {P[0][0], P[0][1], sg * P[0][2]}, B[3] = {P[1][0], P[1][1], sg * P[1][2]},
                     C[3] = {P[2][0], P[2][1], sg * P[2][2]};
        tdhs::TriFs f;
        tdhs::fs_consts(A, B, C, f);
        in = tdhs::fs_part(f, image_receiver(R, image && flat), Ss, Ds, m.nu, m.M2, m.c_fs, sum) && in;
    }
    double b[3];
    tdhs::slip_fixed(P[0], P[1], P[2], Ss, Ds, b);
#pragma unroll 1
    for (int j = 0; j < 3; ++j) {
        double A[3], B[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            A[c] = j == 0 ? P[0][c] : j == 1 ? P[1][c] : P[2][c];
            B[c] = j == 0 ? P[1][c] : j == 1 ? P[2][c] : P[0][c];
        }
        tdhs::TriSide t;
        tdhs::side_consts(A, B, b, t);
        tdhs::side_part(t, A, B, R, m.nu, m.N1, m.M2, m.c_fsc, sum);
    }
    stiffness(m, R, sum, !in, Ks[k], Kn[k]);
}

}  // namespace

void launch_assemble_tri_pairs(cudaStream_t st, int64_t npairs, const int64_t* ridx, const int64_t* sidx,
                               const double* P1, const double* P2, const double* P3, const double* rake,
                               const double* centre, const double* nhat, const double* shat, double G, double nu,
                               double* Ks, double* Kn) {
    const int64_t nb = (npairs + kAsmThreads - 1) / kAsmThreads;
    k_assemble_tri_pairs<<<(unsigned)nb, kAsmThreads, 0, st>>>(npairs, ridx, sidx, P1, P2, P3, rake, centre, nhat,
                                                             shat, G, nu, Ks, Kn);
}

// Sources per block and turn: their constants take a turn ~1,300 FP64
// operations in sequence beside ~8,000 per source and receiver, whatever their
// number, so 8 where that leaves four rounds of the resident blocks, down to 1
// for small calls.
void launch_assemble_tri(cudaStream_t st, int64_t n_src, const double* P1, const double* P2, const double* P3,
                         const double* rake, int64_t n_recv, const double* centre, const double* nhat,
                         const double* shat, double G, double nu, double* Ks, double* Kn, int64_t ld, int layout) {
    const int64_t gx = (n_recv + kAsmThreads - 1) / kAsmThreads;
    int tile = kMaxSrcTile;
    while (tile > 1 && gx * ((n_src + tile - 1) / tile) < (int64_t)8 * num_sms()) tile /= 2;
    const int64_t gy = std::min<int64_t>((n_src + tile - 1) / tile, 65535);
    k_assemble_tri<<<dim3((unsigned)gx, (unsigned)gy), kAsmThreads, 0, st>>>(
        n_src, P1, P2, P3, rake, n_recv, centre, nhat, shat, G, nu, Ks, Kn, ld, layout, tile);
}

}  // namespace qdfn
