// Device-side resampling / weight building blocks shared by the C ABI
// (resample.cu) and the FP64 filter driver (pf64.cu).
#pragma once

#include "common.cuh"
#include "seqsum.cuh"

namespace vsmc_cuda
{

// the words of new_err past the sums' tickets
constexpr int kErrTail = 4;     // uniforms left to the last particle
constexpr int kErrTicket = 5;   // ticket of another last-block reduction
constexpr int kErrMax = 6;      // key of the largest log-weight (two words)

// Threads of a block where each element takes many FP64 instructions (19
// cycles of an SM each): small blocks spread a short vector over all SMs.
constexpr int kB64 = 64;

inline int grid64(size_t n) { return grid_for(n ? n : 1, kB64, 1, 32); }

// Order-preserving unsigned key of a double for the running maximum (an
// integer atomic); 0, the key of nothing, and NaN stand for -inf, as fmax
// from -inf passes NaN over.
__device__ __forceinline__ unsigned long long max_key(double v)
{
    const unsigned long long b =
        static_cast<unsigned long long>(__double_as_longlong(v));
    if ((b & 0x7FFFFFFFFFFFFFFFull) > 0x7FF0000000000000ull)
        return 0;
    return (b >> 63) ? ~b : b | 0x8000000000000000ull;
}

__device__ __forceinline__ double from_max_key(unsigned long long k)
{
    if (k == 0)
        return -static_cast<double>(INFINITY);
    return __longlong_as_double(static_cast<long long>(
        (k >> 63) ? k & 0x7FFFFFFFFFFFFFFFull : ~k));
}


// What is known of a uniform sequence: nothing; non-decreasing, non-negative
// and free of NaN; that, and u_j within [j / n, (j + 1) / n] up to rounding.
enum class UniformOrder { Any, Sorted, Near };

int rep_index_device(size_t m, size_t n, const int *rep, int *idx,
    uint32_t *err, Scratch &scratch, cudaStream_t st);
// the counts of a scheme, queued (the residual schemes wait for their split);
// *N gets the uniforms, err[kErrTail] those left to the last particle
int scheme_enqueue(size_t m, size_t n, const vsmc_cuda_rng &rng,
    const double *w, int *rep, int scheme, uint32_t *err, size_t *N,
    Scratch &scratch, cudaStream_t st);
// the engine past the words the scheme's sequence of N uniforms consumed
void scheme_advance(
    vsmc_cuda_rng &rng, size_t m, size_t N, int scheme, uint32_t tail);
int scheme_device(size_t m, size_t n, vsmc_cuda_rng *rng, const double *w,
    int *rep, int scheme, Scratch &scratch, cudaStream_t st);
int weight_sums(SeqArgs a, const double *v, double *W, double *ess,
    cudaStream_t st);
int weight_normalize_device(size_t n, const double *v, double *W,
    double *ess_dev, uint32_t *err, Scratch &scratch, cudaStream_t st);
int weight_set_log_device(size_t n, const double *lw, double *W,
    double *ess_dev, uint32_t *err, Scratch &scratch, cudaStream_t st);
int weight_set_equal_device(size_t n, double *W, double *ess_dev,
    uint32_t *err, Scratch &scratch, cudaStream_t st);
int weight_add_log_device(size_t n, const double *l, double *W,
    double *ess_dev, uint32_t *err, Scratch &scratch, cudaStream_t st);
template <typename T>
int monitor_mean_device(size_t n, size_t dim, size_t ld, const T *state,
    const double *W, double *out, Scratch &scratch, cudaStream_t st);
template <typename T>
int state_copy_device(size_t n, size_t dim, size_t ld, const int *idx,
    T *state, uint32_t *err, cudaStream_t st);

} // namespace vsmc_cuda
