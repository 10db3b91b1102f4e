// Left-to-right double summation: buffers, entry points (the passes are in
// seqsum.cuh).
#include "common.cuh"
#include "seqsum.cuh"

#include <algorithm>

namespace vsmc_cuda
{

uint32_t *new_err(Scratch &scratch, cudaStream_t st)
{
    uint32_t *err = scratch.get<uint32_t>(kErrWords);
    if (err == nullptr)
        return nullptr;
    const cudaError_t e =
        cudaMemsetAsync(err, 0, kErrWords * sizeof(uint32_t), st);
    if (e != cudaSuccess) {
        set_last_cuda_error(e);
        return nullptr;
    }
    return err;
}

int seq_args(size_t n, uint32_t *err, bool allow_inf, Scratch &scratch,
    SeqArgs *a)
{
    if (n >= (size_t(1) << 31))
        return VSMC_CUDA_ERR_SIZE;
    const size_t nt = (n + kSeqTile - 1) / kSeqTile;
    const size_t most = std::min<size_t>(
        static_cast<size_t>(num_sms()) * kSeqOcc, kSeqMaxRanges);
    const size_t nb = std::min(nt, most);
    const size_t tb = (nt + nb - 1) / nb;
    size_t bytes = 0;
    auto place = [&bytes](size_t b) {
        const size_t at = bytes;
        bytes += (b + 255) / 256 * 256;
        return at;
    };
    const size_t ntt = nb * (tb + 1);
    const size_t oP = place(sizeof(double) * (nb + 1));
    const size_t oR = place(sizeof(uint64_t) * (nb + 1));
    const size_t oF = place(sizeof(uint32_t) * (nb + 1));
    const size_t oS = place(sizeof(uint64_t) * (nb + 1));
    const size_t otP = place(sizeof(double) * ntt);
    const size_t otR = place(sizeof(uint64_t) * ntt);
    const size_t otF = place(sizeof(uint32_t) * ntt);
    const size_t oT = place(2 * sizeof(double));
    const size_t nl = n <= kSeqSmall ? 0 : n; // the lists
    const size_t oA = place(sizeof(uint64_t) * nl);
    const size_t oE = place(sizeof(uint32_t) * nl);
    const size_t oX = place(sizeof(uint16_t) * nl);
    char *b = scratch.get<char>(bytes);
    if (b == nullptr)
        return VSMC_CUDA_ERR_ALLOC;
    a->n = static_cast<uint32_t>(n);
    a->nt = static_cast<uint32_t>(nt);
    a->tb = static_cast<uint32_t>(tb);
    a->blocks = static_cast<uint32_t>(nb);
    int lg = 0;
    while ((size_t(1) << lg) < n)
        ++lg;
    const int mexp = lg < 11 ? 40 : 51 - lg; // m = 2^-mexp
    a->flo = 1ull << (53 - mexp);
    a->fhi = (1ull << 52) - a->flo;
    a->P = reinterpret_cast<double *>(b + oP);
    a->R = reinterpret_cast<uint64_t *>(b + oR);
    a->F = reinterpret_cast<uint32_t *>(b + oF);
    a->start = reinterpret_cast<uint64_t *>(b + oS);
    a->tP = reinterpret_cast<double *>(b + otP);
    a->tR = reinterpret_cast<uint64_t *>(b + otR);
    a->tF = reinterpret_cast<uint32_t *>(b + otF);
    a->total = reinterpret_cast<double *>(b + oT);
    a->inv = a->total + 1;
    a->adj = reinterpret_cast<uint64_t *>(b + oA);
    a->pos = reinterpret_cast<uint32_t *>(b + oE);
    a->bex = reinterpret_cast<uint16_t *>(b + oX);
    a->err = err;
    a->allow_inf = allow_inf ? 1 : 0;
    return VSMC_CUDA_OK;
}

int seqsum_device(size_t n, const double *x, double *prefix, double *total,
    uint32_t *err, Scratch &scratch, cudaStream_t st, bool allow_inf)
{
    if (n == 0) {
        if (total)
            VSMC_CUDA_TRY(cudaMemsetAsync(total, 0, sizeof(double), st));
        return VSMC_CUDA_OK;
    }
    SeqArgs a;
    int rc = seq_args(n, err, allow_inf, scratch, &a);
    if (rc != VSMC_CUDA_OK)
        return rc;
    if (total)
        a.total = total;
    a.inv = nullptr;
    return prefix ? seq_scan(a, SeqLoad{x}, SeqStore{prefix, a.n}, st)
                  : seq_total(a, SeqLoad{x}, st);
}

int err_status(uint32_t e)
{
    if (e & DEV_ERR_NONFINITE)
        return VSMC_CUDA_ERR_NONFINITE;
    if (e & DEV_ERR_COUNTS)
        return VSMC_CUDA_ERR_ARG;
    return e ? VSMC_CUDA_ERR_INTERNAL : VSMC_CUDA_OK;
}

int read_err(uint32_t *err_dev, cudaStream_t st, int *status)
{
    uint32_t e = 0;
    VSMC_CUDA_TRY(cudaMemcpyAsync(
        &e, err_dev, sizeof(e), cudaMemcpyDeviceToHost, st));
    VSMC_CUDA_TRY(cudaStreamSynchronize(st));
    *status = err_status(e);
    return VSMC_CUDA_OK;
}

} // namespace vsmc_cuda

using namespace vsmc_cuda;

extern "C" int vsmc_cuda_sequential_sum(size_t n, const double *x,
    double *prefix, double *total_dev, void *stream)
{
    if ((x == nullptr && n) || (prefix == nullptr && total_dev == nullptr))
        return VSMC_CUDA_ERR_ARG;
    cudaStream_t st = as_stream(stream);
    Scratch scratch(st);
    uint32_t *err = new_err(scratch, st);
    if (err == nullptr)
        return VSMC_CUDA_ERR_ALLOC;
    int rc = seqsum_device(n, x, prefix, total_dev, err, scratch, st);
    if (rc != VSMC_CUDA_OK)
        return rc;
    int status = VSMC_CUDA_OK;
    rc = read_err(err, st, &status);
    return rc != VSMC_CUDA_OK ? rc : status;
}
