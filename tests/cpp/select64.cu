// The FP64 filter's copy kernel launched on buffers of the test's: the
// library's own translation unit, compiled here, with its other functions
// taken from libvsmc_cuda.  Built and called by
// tests/test_pf64_select_gpu.py.
#include "pf64.cu"

using namespace vsmc_cuda;

// err: kErrWords words; out: the mean (2 doubles); host: 3 words.  scal[2] is
// the weight that every particle gets.
extern "C" int select64(uint32_t n, uint32_t ld, double *state, double *W,
    const int *idx, double *scal, uint32_t *err, double *part, double *out,
    uint32_t *host)
{
    Step64 a = {};
    a.n = n;
    a.state = state;
    a.ld = ld;
    a.W = W;
    a.scal = scal;
    a.h_mean = out;
    a.err = err;
    a.host = reinterpret_cast<Pf64Host *>(host);
    k_select64<<<select_grid(n), kSelB>>>(a, state, idx, part);
    if (cudaGetLastError() != cudaSuccess)
        return 1;
    return cudaDeviceSynchronize() == cudaSuccess ? 0 : 2;
}

extern "C" uint32_t select64_blocks(uint32_t n)
{
    return static_cast<uint32_t>(select_grid(n));
}
