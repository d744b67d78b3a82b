// Launchers and argument blocks of the adjoint kernels (adjoint.cu), used by
// the adjoint driver in sim.cu.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "qdfn_internal.h"

namespace qdfn {

constexpr int kAdjMaxInst = 4;

// One reverse step's per-patch inputs and outputs ([R][N] unless noted).
struct AdjLocalArgs {
    int64_t N, Ns;
    int R, dr, interp_at_told;
    double eta, sigma_min;
    // the step: state before (prev) and after (cur), its TLD, sigma, solver
    const double *Vprev, *Dprev, *thprev, *Vcur, *tld, *sig;
    const unsigned char* sw;
    const double *dt, *Tprev;          // [R]: the step's dt and the time before it
    // run constants
    const double *pa, *pb, *pDc, *F0, *la, *lth0, *kself /*[N]*/, *mass, *omega, *tau0;
    int64_t n_ext;
    const double *ext_t, *ext_n, *ext_s, *ext_p;
    // adjoints of the step's outputs
    const double *lV, *lD, *lth, *lA;
    // adjoints of its inputs (D_old local part, V_old, theta_old, TLD, sigma)
    double *oDloc, *oVold, *oThold, *oTLD, *oSig;
    double *ga, *gb, *gDc;             // parameter gradients, accumulated
    double *blk_dt, *blk_tx;           // [blocks][R] partial sums
    int* err;                          // set when a residual's derivative vanishes
};

// Transposed products over the tile-contiguous operator (rpb rows per block).
struct AdjTransArgs {
    int64_t N, rpb, nrb;
    int64_t gx;                        // column blocks per row block
    const void *E, *Kn;
    const double *x_s, *x_n;           // [R][N]: lambda_TLD (E^T) and lambda_sigma (Kn^T)
    double* part;                      // [nrb][2][R][N]
};

int adj_local(const AdjLocalArgs& a, cudaStream_t st);
int adj_local_blocks(int64_t RN);
int adj_transpose_prepare(int prec, int R, int64_t rpb);
// out = dloc - E^T x_s + Kn^T x_n, and zero = 0
int adj_transpose(int prec, int R, const AdjTransArgs& a, const double* dloc, double* out, double* zero,
                  cudaStream_t st);

// The adjoint of a reverse step's Dt and T, and the seeds of the state it ends
// at (V null: the seeds alone, for the last state).
struct AdjControlArgs {
    int64_t N, Ns, state;              // the state's number in the window
    int R, nblk, told;
    double rupture_dt, max_dt, switch_v, dt_cut;
    const double *V, *A;               // [R][N] the state the step's Dt was chosen from
    const double *dt_now, *dt_prev;    // [R]
    const unsigned char* unstable;
    const int* has_unstable;
    const double *blk_dt, *blk_tx;     // [nblk][R] from adj_local
    double *lamT, *carry;              // [R], kept from step to step
    const int64_t *seed_off, *seed_patch;   // [states * R + 1], [seeds]
    const double* seed_val;            // [seeds][3]: dV, dD, dT
    double *lV, *lD, *lA;
};
int adj_control(const AdjControlArgs& a, cudaStream_t st);

}  // namespace qdfn
