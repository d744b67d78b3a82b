// Device self-checks of the arithmetic helpers, exposed for the test suite and
// evaluated on caller arrays: the reciprocal-based division the friction solves
// use in place of IEEE division (sim_device.cuh div_by); their logarithm,
// exponential, reciprocal and conversions (friction_math.cuh); the square root and
// the quotients of the rectangle kernel (okada_sums.cuh).
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
