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

// What a pair needs of its source
struct SrcConst {
    okada::Src o;
    double cx, cy, cz, AL, AW, cs, sn, strike, dip, DISL1, DISL2;
};

// The gradients by okada.cuh, for the few pairs near a singular line of the
// source.  Out of line: its registers stay out of the usual path.
__device__ __noinline__ void general_gradients(double alpha, double dip, double X, double Y, double Z, double depth,
                                               double AL, double AW, double DISL1, double DISL2, double* U) {
    okada::dc3d_gradients(okada::dccon0(alpha, dip), X, Y, Z, depth, AL, AL, AW, AW, DISL1, DISL2, 0.0, U);
}

// A block takes kAsmThreads receivers, one per thread, and `tile` sources at a
// time: what depends on the source alone (sines and cosines, the medium) is
// formed once per block and turn, what depends on the receiver alone once per
// turn.  Bound by the FP64 pipe.  Against one pair per thread and turn with all
// of okada.cuh: 5,850 x 5,850 patches 473.6 -> 86.6 ms, 800 x 800 9.80 -> 1.84
// ms, 61 x 64 (122 warps: the length of one pair's chain) 252 -> 64 us.
__global__ void __launch_bounds__(kAsmThreads)
k_assemble_rect(int64_t n_src, const double* __restrict__ src, int64_t n_recv,
                const double* __restrict__ recv, double G, double nu, double* __restrict__ Ks,
                double* __restrict__ Kn, int64_t ld, int layout, int tile) {
    __shared__ SrcConst sc[kMaxSrcTile];
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool mine = r < n_recv;
    const double lam = 2 * G * nu / (1 - 2 * nu);
    const double alpha = (lam + G) / (lam + 2 * G);
    const double* rr = recv + (mine ? r : 0) * 8;
    const double rcx = rr[0], rcy = rr[1], rcz = rr[2], rstr = rr[5];
    const double cdp = cosd_d(-rr[6]), sdp = sind_d(-rr[6]);
    const double crk = cosd_d(rr[7]), srk = sind_d(rr[7]);
    const double rcs = cosd_d(rstr), rsn = sind_d(rstr);
    for (int64_t s0 = (int64_t)blockIdx.y * tile; s0 < n_src; s0 += (int64_t)gridDim.y * tile) {
        const int ns = (int)min((int64_t)tile, n_src - s0);
        __syncthreads();
        if (threadIdx.x < ns) {
            const double* ss = src + (s0 + threadIdx.x) * 8;
            SrcConst c;
            const okada::C0 c0 = okada::dccon0(alpha, ss[6]);
            c.o.SD = c0.SD; c.o.CD = c0.CD;
            c.o.flat = c0.CD == 0.0;
            c.o.iCD = c.o.flat ? 0.0 : 1.0 / c0.CD;
            c.o.A1 = c0.ALP1; c.o.A2 = c0.ALP2; c.o.A3 = c0.ALP3; c.o.A4 = c0.ALP4; c.o.A5 = c0.ALP5;
            c.DISL1 = cosd_d(ss[7]); c.DISL2 = sind_d(ss[7]);
            c.o.D1 = c.DISL1 / 6.283185307179586; c.o.D2 = c.DISL2 / 6.283185307179586;
            c.cx = ss[0]; c.cy = ss[1]; c.cz = ss[2]; c.AL = ss[3] / 2; c.AW = ss[4] / 2;
            c.strike = ss[5]; c.dip = ss[6];
            c.cs = cosd_d(-ss[5]); c.sn = sind_d(-ss[5]);
            sc[threadIdx.x] = c;
        }
        __syncthreads();
        if (!mine) continue;
        for (int k = 0; k < ns; ++k) {
            const SrcConst& c = sc[k];
            const double Xd = rcx - c.cx, Yd = rcy - c.cy;
            const double X = Xd * c.cs - Yd * c.sn;
            const double Y = Xd * c.sn + Yd * c.cs;
            const double Z = -rcz;
            double U[9];
            bool ok = okada::corner_sums(c.o, X, Y, Z, c.cz, c.AL, c.AW, U);
            double sum = 0.0;
#pragma unroll
            for (int i = 0; i < 9; ++i) sum += U[i];
            if (!(ok && isfinite(sum))) {
                double W[9];
                general_gradients(alpha, c.dip, X, Y, Z, c.cz, c.AL, c.AW, c.DISL1, c.DISL2, W);
#pragma unroll
                for (int i = 0; i < 9; ++i) U[i] = W[i];
            }
            // Hooke's law in the source frame (:462-467)
            const double tr = lam * (U[0] + U[4] + U[8]);
            const double sxx = fma(2 * G, U[0], tr), syy = fma(2 * G, U[4], tr), szz = fma(2 * G, U[8], tr);
            const double sxy = (U[3] + U[1]) * G, sxz = (U[6] + U[2]) * G, syz = (U[7] + U[5]) * G;
            // sigma' = R sigma R^T with R = R_dip R_strike(-relative strike)
            // (:480-492); sigma'_13, sigma'_23, sigma'_33 are R (sigma R_3), R_i
            // the rows of R.  cos and sin of the relative strike from the two
            // strikes' (exactly 1 and 0 where they are equal).
            const bool same = rstr == c.strike;
            const double cr = same ? 1.0 : rcs * c.cs - rsn * c.sn, sr = same ? 0.0 : -(rcs * c.sn + rsn * c.cs);
            const double R20 = sdp * sr, R21 = sdp * cr, R22 = cdp;
            const double t0 = fma(sxx, R20, fma(sxy, R21, sxz * R22));
            const double t1 = fma(sxy, R20, fma(syy, R21, syz * R22));
            const double t2 = fma(sxz, R20, fma(syz, R21, szz * R22));
            const double S02 = fma(cr, t0, -sr * t1);
            const double S12 = fma(cdp, fma(sr, t0, cr * t1), -sdp * t2);
            const double S22 = fma(R20, t0, fma(R21, t1, R22 * t2));
            const int64_t s = s0 + k;
            const int64_t idx = layout == QDFN_LAYOUT_COL ? s * ld + r : r * ld + s;
            Kn[idx] = -S22;
            Ks[idx] = crk * S02 + srk * S12;
        }
    }
}

}  // namespace

// Sources per block and turn: a turn costs a thread ~250 FP64 operations of its
// receiver's and sources' sines and cosines beside ~1,340 per pair, so 8 where
// that still leaves four rounds of the GPU's resident blocks (two per SM at 255
// registers), down to 1 for small calls, where every pair starts at once.
void launch_assemble_rect(cudaStream_t st, int64_t n_src, const double* src, int64_t n_recv, const double* recv,
                          double G, double nu, double* Ks, double* Kn, int64_t ld, int layout) {
    const int64_t gx = (n_recv + kAsmThreads - 1) / kAsmThreads;
    int tile = kMaxSrcTile;
    while (tile > 1 && gx * ((n_src + tile - 1) / tile) < (int64_t)8 * num_sms()) tile /= 2;
    const int64_t gy = std::min<int64_t>((n_src + tile - 1) / tile, 65535);
    k_assemble_rect<<<dim3((unsigned)gx, (unsigned)gy), kAsmThreads, 0, st>>>(n_src, src, n_recv, recv, G, nu, Ks, Kn,
                                                                             ld, layout, tile);
}

}  // namespace qdfn
