// Device self-checks of the arithmetic helpers, exposed for the test suite and
// evaluated on caller arrays: the reciprocal-based division the friction solves
// use in place of IEEE division (sim_device.cuh div_by); their logarithm,
// exponential, reciprocal and conversions (friction_math.cuh); the square root and
// the quotients of the rectangle kernel (okada_sums.cuh); and the patch solvers
// one by one (sim_device.cuh), which the step loop chooses among by operands.
#include <cuda_runtime.h>

#include "okada_sums.cuh"
#include "qdfn_internal.h"
#include "sim_device.cuh"

namespace qdfn {
namespace {

__global__ void k_check_division(int64_t n, const double* __restrict__ x, const double* __restrict__ d,
                                 double* __restrict__ q) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    q[i] = sim::div_by(x[i], sim::recip(d[i]));
}

__device__ double math_value(int which, double x, double d) {
    double R, i1;
    switch (which) {
        case 0: return sim::fm_log(x);
        case 1: return sim::fm_exp(x);
        case 2: return sim::fm_rcp(x);
        case 3: return sim::to_float(x);
        case 4: return sim::to_double((float)x);
        case 5: return sim::to_double((int)x);
        case 6: return okada::recip1(x);
        case 7: return okada::recip2(x);
        case 8: return okada::quotient(x, d, okada::recip1(d));
        case 9: okada::root(x, R, i1); return R;
        default: okada::root(x, R, i1); return i1;
    }
}
__global__ void k_check_math(int which, int64_t n, const double* __restrict__ x, const double* __restrict__ d,
                             double* __restrict__ y) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = math_value(which, x[i], d[i]);
}

// a patch's operands in the caller's order, and what a solver returns
constexpr int kSolveIn = 17, kSolveOut = 10;
__global__ void k_check_solve(int which, int64_t n, const double* __restrict__ in, double eta, double alpha, int dr,
                              double switch_v, double* __restrict__ out) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool pair = which >= 4, high = (which & 1) != 0;
    const int64_t i = pair ? t / 2 : t;   // (a pair of lanes leaves together)
    if (i >= n) return;
    const double* x = in + i * kSolveIn;
    sim::PatchIn p;
    p.DispOld = x[0]; p.FrictionOld = x[1]; p.ThetaOld = x[2]; p.VOld = x[3]; p.Friction0 = x[4]; p.a = x[5];
    p.b = x[6]; p.Dc = x[7]; p.K_Self = x[8]; p.Omega = x[9]; p.Mass = x[10]; p.sigma = x[11]; p.TLD = x[12];
    p.dtau = x[13]; p.sigma_old = x[14]; p.tau0 = x[15];
    const double Dt = x[16];
    p.ra = 1.0 / p.a; p.rDc = 1.0 / p.Dc; p.rDt = 1.0 / Dt;
    sim::PatchOut o{};
    int err = 0;
    bool taken = true;
    if (which == 0) taken = sim::solve_lowv_newton(p, Dt, eta, alpha, dr, o);
    else if (which == 1) taken = sim::solve_highv_usual(p, Dt, eta, alpha, dr, o);
    else o = sim::solve_reference(p, high, pair, Dt, eta, alpha, dr, switch_v, err);
    if (pair && (t & 1)) return;
    double* y = out + i * kSolveOut;
    y[0] = taken; y[1] = o.V; y[2] = o.Friction; y[3] = o.Disp; y[4] = o.Theta; y[5] = o.Dt;
    y[6] = o.Instab; y[7] = o.Flag; y[8] = o.Iterations; y[9] = err;
}

}  // namespace
}  // namespace qdfn

using namespace qdfn;

extern "C" int qdfn_check_division(int64_t n, const double* x, const double* d, double* q, void* stream) {
    if (n < 0) return fail(QDFN_ERR_INVALID, "n < 0");
    if (n == 0) return QDFN_OK;
    if (!x || !d || !q) return fail(QDFN_ERR_INVALID, "null pointer");
    const int64_t blocks = (n + 255) / 256;
    if (blocks > 2147483647LL) return fail(QDFN_ERR_INVALID, "n too large");
    k_check_division<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(n, x, d, q);
    QDFN_CUDA(cudaGetLastError());
    return QDFN_OK;
}

extern "C" int qdfn_check_math(int which, int64_t n, const double* x, const double* d, double* y, void* stream) {
    if (which < 0 || which > 10) return fail(QDFN_ERR_INVALID, "no such function");
    if (n < 0) return fail(QDFN_ERR_INVALID, "n < 0");
    if (n == 0) return QDFN_OK;
    if (!x || !d || !y) return fail(QDFN_ERR_INVALID, "null pointer");
    const int64_t blocks = (n + 255) / 256;
    if (blocks > 2147483647LL) return fail(QDFN_ERR_INVALID, "n too large");
    k_check_math<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(which, n, x, d, y);
    QDFN_CUDA(cudaGetLastError());
    return QDFN_OK;
}

extern "C" int qdfn_check_solve(int which, int64_t n, const double* in, double eta, double alpha, int evolution_dr,
                                double switch_v, double* out, void* stream) {
    if (which < 0 || which > 5) return fail(QDFN_ERR_INVALID, "no such solver");
    if (n < 0) return fail(QDFN_ERR_INVALID, "n < 0");
    if (n == 0) return QDFN_OK;
    if (!in || !out) return fail(QDFN_ERR_INVALID, "null pointer");
    const int64_t blocks = ((which >= 4 ? 2 * n : n) + 127) / 128;
    if (blocks > 2147483647LL) return fail(QDFN_ERR_INVALID, "n too large");
    k_check_solve<<<(unsigned)blocks, 128, 0, (cudaStream_t)stream>>>(which, n, in, eta, alpha, evolution_dr, switch_v,
                                                                     out);
    QDFN_CUDA(cudaGetLastError());
    return QDFN_OK;
}
