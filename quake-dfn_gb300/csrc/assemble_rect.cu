// Rectangular-patch stiffness kernel (Okada DC3D), one thread per
// (receiver, source) pair, FP64.  Follows StiffnessMatrix_ByParts_Calculation_Rec
// (scripts/Functions_BuildInputFile.jl:386-512).
#include <cuda_runtime.h>

#include <algorithm>

#include "assemble_kernels.h"
#include "qdfn_internal.h"
#include "okada_sums.cuh"

namespace qdfn {
namespace {

constexpr int kMaxSrcTile = 8;   // sources of a block's turn, their constants in shared memory

// What a pair needs of its source and of its receiver
struct SrcConst {
    okada::Src o;
    double cx, cy, cz, AL, AW, cs, sn, strike, DISL1, DISL2;
};
struct RecvConst {
    double cx, cy, cz, strike, cdp, sdp, crk, srk, cs, sn;
};

// The receiver in the source's axes
struct Local {
    double X, Y, Z;
};
__device__ __forceinline__ Local local(const SrcConst& c, const RecvConst& r) {
    const double Xd = r.cx - c.cx, Yd = r.cy - c.cy;
    return {Xd * c.cs - Yd * c.sn, Xd * c.sn + Yd * c.cs, -r.cz};
}

// Ks and Kn of the displacement gradients U
__device__ __forceinline__ void stiffness(const SrcConst& c, const RecvConst& r, double lam, double G,
                                          const double (&U)[9], double& ks, double& kn) {
    // Hooke's law in the source frame (:462-467)
    const double tr = lam * (U[0] + U[4] + U[8]);
    const double sxx = fma(2 * G, U[0], tr), syy = fma(2 * G, U[4], tr), szz = fma(2 * G, U[8], tr);
    const double sxy = (U[3] + U[1]) * G, sxz = (U[6] + U[2]) * G, syz = (U[7] + U[5]) * G;
    // sigma' = R sigma R^T with R = R_dip R_strike(-relative strike)
    // (:480-492); sigma'_13, sigma'_23, sigma'_33 are R (sigma R_3), R_i
    // the rows of R.  cos and sin of the relative strike from the two
    // strikes' (exactly 1 and 0 where they are equal).
    const bool same = r.strike == c.strike;
    const double cr = same ? 1.0 : r.cs * c.cs - r.sn * c.sn, sr = same ? 0.0 : -(r.cs * c.sn + r.sn * c.cs);
    const double R20 = r.sdp * sr, R21 = r.sdp * cr, R22 = r.cdp;
    const double t0 = fma(sxx, R20, fma(sxy, R21, sxz * R22));
    const double t1 = fma(sxy, R20, fma(syy, R21, syz * R22));
    const double t2 = fma(sxz, R20, fma(syz, R21, szz * R22));
    const double S02 = fma(cr, t0, -sr * t1);
    const double S12 = fma(r.cdp, fma(sr, t0, cr * t1), -r.sdp * t2);
    kn = -fma(R20, t0, fma(R21, t1, R22 * t2));
    ks = r.crk * S02 + r.srk * S12;
}

// A pair by okada.cuh.  Out of line: its registers stay out of the usual path.
__device__ __noinline__ void general_pair(const SrcConst& c, const RecvConst& r, double lam, double G, double* ks,
                                          double* kn) {
    const okada::Src& o = c.o;
    const okada::C0 c0{o.A1, o.A2, o.A3, o.A4, o.A5, o.SD, o.CD, o.SD * o.SD, o.CD * o.CD, o.SD * o.CD};
    const Local p = local(c, r);
    double U[9];
    okada::dc3d_gradients(c0, p.X, p.Y, p.Z, c.cz, c.AL, c.AL, c.AW, c.AW, c.DISL1, c.DISL2, 0.0, U);
    stiffness(c, r, lam, G, U, *ks, *kn);
}

// Adds the real source's part, corner by corner, to a pair that has the rest
__device__ __noinline__ void add_real_source(const SrcConst& c, const RecvConst& r, double lam, double G, double* ks,
                                             double* kn) {
    const Local p = local(c, r);
    double U[9], s, n;
    okada::real_corners(c.o, p.X, p.Y, p.Z, c.cz, c.AL, c.AW, U);
    stiffness(c, r, lam, G, U, s, n);
    *ks += s;
    *kn += n;
}

// A block takes kAsmThreads receivers, one per thread, and `tile` sources at a
// time: what depends on the source alone (sines and cosines, the medium) is
// formed once per block and turn, what depends on the receiver alone once.  The
// pairs that need their real source's part corner by corner (4 % of a fault
// network's, in 10 % of its warps) go to a list in shared memory, which the
// block's threads work off at the turn's end without gaps.  (In their own warps:
// 105 ms of the network below, 2.38 of the two faults.)
// Bound by the FP64 pipe.  Against one pair per thread and turn with all of
// okada.cuh: 5,850 x 5,850 patches of a network 473.6 -> 93.5 ms, 800 x 800 of
// two faults 9.79 -> 2.08 ms, 61 x 64 (122 warps: the length of one pair's chain)
// 252 -> 69 us.
template <bool GENERAL>   // all pairs by okada.cuh (the self-check's)
__global__ void __launch_bounds__(kAsmThreads)
k_assemble_rect(int64_t n_src, const double* __restrict__ src, int64_t n_recv,
                const double* __restrict__ recv, double G, double nu, double* __restrict__ Ks,
                double* __restrict__ Kn, int64_t ld, int layout, int tile) {
    __shared__ SrcConst sc[kMaxSrcTile];
    __shared__ RecvConst rc[kAsmThreads];
    __shared__ unsigned short list[kMaxSrcTile * kAsmThreads];   // source k, thread t: k * kAsmThreads + t
    __shared__ int listed;
    const int64_t r0 = (int64_t)blockIdx.x * kAsmThreads;
    const bool mine = r0 + threadIdx.x < n_recv;
    const double lam = 2 * G * nu / (1 - 2 * nu);
    const double alpha = (lam + G) / (lam + 2 * G);
    {
        const double* rr = recv + (mine ? r0 + threadIdx.x : 0) * 8;
        RecvConst r;
        r.cx = rr[0]; r.cy = rr[1]; r.cz = rr[2]; r.strike = rr[5];
        r.cdp = cosd_d(-rr[6]); r.sdp = sind_d(-rr[6]);
        r.crk = cosd_d(rr[7]); r.srk = sind_d(rr[7]);
        r.cs = cosd_d(rr[5]); r.sn = sind_d(rr[5]);
        rc[threadIdx.x] = r;
    }
    const RecvConst r = rc[threadIdx.x];
    for (int64_t s0 = (int64_t)blockIdx.y * tile; s0 < n_src; s0 += (int64_t)gridDim.y * tile) {
        const int ns = (int)min((int64_t)tile, n_src - s0);
        auto index = [&](int k, int t) {
            return layout == QDFN_LAYOUT_COL ? (s0 + k) * ld + r0 + t : (r0 + t) * ld + s0 + k;
        };
        __syncthreads();
        if (threadIdx.x == 0) listed = 0;
        if (threadIdx.x < ns) {
            const double* ss = src + (s0 + threadIdx.x) * 8;
            SrcConst c;
            const okada::C0 c0 = okada::dccon0(alpha, ss[6]);
            c.o.SD = c0.SD; c.o.CD = c0.CD;
            c.o.flat = c0.CD == 0.0;
            c.o.steep = okada::is_steep(c0.CD);
            c.o.iCD = c.o.flat ? 0.0 : 1.0 / c0.CD;
            c.o.A1 = c0.ALP1; c.o.A2 = c0.ALP2; c.o.A3 = c0.ALP3; c.o.A4 = c0.ALP4; c.o.A5 = c0.ALP5;
            c.DISL1 = cosd_d(ss[7]); c.DISL2 = sind_d(ss[7]);
            c.o.D1 = c.DISL1 / 6.283185307179586; c.o.D2 = c.DISL2 / 6.283185307179586;
            c.cx = ss[0]; c.cy = ss[1]; c.cz = ss[2]; c.AL = ss[3] / 2; c.AW = ss[4] / 2;
            c.strike = ss[5];
            c.cs = cosd_d(-ss[5]); c.sn = sind_d(-ss[5]);
            sc[threadIdx.x] = c;
        }
        __syncthreads();
        if (mine) {
            for (int k = 0; k < ns; ++k) {
                const SrcConst& c = sc[k];
                const int64_t idx = index(k, threadIdx.x);
                if constexpr (GENERAL) {
                    general_pair(c, rc[threadIdx.x], lam, G, Ks + idx, Kn + idx);
                    continue;
                }
                const Local p = local(c, r);
                double U[9];
                bool plain = true;
                bool ok = okada::real_sums(c.o, p.X, p.Y, p.Z, c.cz, c.AL, c.AW, U, plain);
                double sum = 0.0;
#pragma unroll
                for (int i = 0; i < 9; ++i) {
                    sum += U[i];
                    if (!plain) U[i] = 0.0;
                }
                ok = ok && isfinite(sum);
                ok = okada::image_sums(c.o, p.X, p.Y, p.Z, c.cz, c.AL, c.AW, U) && ok;
                sum = 0.0;
#pragma unroll
                for (int i = 0; i < 9; ++i) sum += U[i];
                if (ok && isfinite(sum)) {
                    double ks, kn;
                    stiffness(c, r, lam, G, U, ks, kn);
                    Kn[idx] = kn;
                    Ks[idx] = ks;
                    if (!plain) list[atomicAdd(&listed, 1)] = (unsigned short)(k * kAsmThreads + threadIdx.x);
                } else {
                    general_pair(c, rc[threadIdx.x], lam, G, Ks + idx, Kn + idx);
                }
            }
        }
        if constexpr (!GENERAL) {
            __syncthreads();
            for (int n = threadIdx.x; n < listed; n += kAsmThreads) {
                const int k = list[n] / kAsmThreads, t = list[n] % kAsmThreads;
                const int64_t idx = index(k, t);
                add_real_source(sc[k], rc[t], lam, G, Ks + idx, Kn + idx);
            }
        }
    }
}

}  // namespace

// Sources per block and turn: a turn costs a thread ~250 FP64 operations of its
// receiver's and sources' sines and cosines beside ~1,400 per pair, so 8 where
// that still leaves four rounds of the GPU's resident blocks (two per SM at 255
// registers), down to 1 for small calls, where every pair starts at once.
void launch_assemble_rect(cudaStream_t st, int64_t n_src, const double* src, int64_t n_recv, const double* recv,
                          double G, double nu, double* Ks, double* Kn, int64_t ld, int layout, bool general) {
    const int64_t gx = (n_recv + kAsmThreads - 1) / kAsmThreads;
    int tile = kMaxSrcTile;
    while (tile > 1 && gx * ((n_src + tile - 1) / tile) < (int64_t)8 * num_sms()) tile /= 2;
    const int64_t gy = std::min<int64_t>((n_src + tile - 1) / tile, 65535);
    auto* k = general ? k_assemble_rect<true> : k_assemble_rect<false>;
    k<<<dim3((unsigned)gx, (unsigned)gy), kAsmThreads, 0, st>>>(n_src, src, n_recv, recv, G, nu, Ks, Kn, ld, layout,
                                                               tile);
}

}  // namespace qdfn
