// The integer functions of normal64.cuh and explog64.cuh on the device (their
// seeds are the device's reciprocal root and reciprocal there), one kernel
// each.  Built and called by tests/test_integer_functions_gpu.py.
#include "explog64.cuh"

#include <cstddef>

using namespace vsmc_cuda;

namespace
{

__global__ void k_polar(
    const uint64_t *u, size_t n, double *r, double *s, double *c)
{
    const size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
    if (i >= n)
        return;
    r[i] = n64_radius(u[i]);
    n64_sincos(u[i], s[i], c[i]);
}

__global__ void k_explog(int op, const double *x, const uint32_t *w,
    const uint32_t *d, size_t n, double *r)
{
    const size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
    if (i >= n)
        return;
    r[i] = op == 0 ? exp_of_negative(-x[i])
        : op == 1  ? -log_of_fraction(x[i])
                   : n64_neg_log_over(w[i], d[i]);
}

int done()
{
    return cudaGetLastError() == cudaSuccess &&
            cudaDeviceSynchronize() == cudaSuccess
        ? 0
        : 1;
}

} // namespace

extern "C" int polar(
    const uint64_t *u, size_t n, double *r, double *s, double *c)
{
    k_polar<<<static_cast<unsigned>((n + 255) / 256), 256>>>(u, n, r, s, c);
    return done();
}

extern "C" int explog(int op, const double *x, const uint32_t *w,
    const uint32_t *d, size_t n, double *r)
{
    k_explog<<<static_cast<unsigned>((n + 255) / 256), 256>>>(
        op, x, w, d, n, r);
    return done();
}
