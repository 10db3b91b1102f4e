// FP64 bootstrap filter with the reference's arithmetic step for step: the
// Weight class's normalized doubles and left-to-right sums
// (core/weight.hpp:145-230), the scheme functors with the sequential
// resampling engine (core/particle.hpp:170-197), rep -> index with the
// reference slot layout and the in-place copy, then the Monitor's weighted
// mean (core/monitor.hpp:242-268).  Only libm (exp / log / sincos / log1p)
// differs from the reference, so a run tracks the oracle closely.  The step
// reads the ESS back to decide on resampling, as Particle::resample does.
//
// A step is three launches and one host wait:
//   move   every particle moves; the largest log-weight lw = log(W) + l and
//          the largest l are found (integer atomics);
//   exp    W = exp(lw - max), and block sums of the evidence's terms
//          W exp(l - max l);
//   weigh  both left-to-right sums, the normalized weights, ESS, evidence,
//          the decision and, without a resample, the weighted mean: one
//          cluster up to 16384 particles, the passes of seqsum.cuh above.
// The decision and the error word go to mapped host memory.  A resample adds
// the uniforms, the counts, the slots and one pass that copies particles,
// sets the weights and takes the mean.  move and exp are bound by the FP64
// pipe (19 cycles of an SM per warp's instruction), so they run in 64-thread
// blocks over all SMs: at 2^14 particles a step took 320 us with 256-thread
// blocks on 16 to 64 SMs, about 60 launches and four waits.
#include "explog64.cuh"
#include "pf_internal.cuh"
#include "pf_model.cuh"
#include "resample_internal.cuh"
#include "seqsum.cuh"

#include <algorithm>
#include <cmath>
#include <new>

namespace vsmc_cuda
{

// What the host reads after a step (mapped pinned memory).
struct Pf64Host {
    uint32_t err;
    uint32_t resample; // ESS < threshold * n
    uint32_t tail;     // uniforms left to the last particle (a resample's)
};

struct Pf64State {
    int *rep = nullptr;
    int *idx = nullptr;
    double *scal = nullptr; // [0] ess, [1] log-evidence, [2] 1 / n normalized,
                            // [4], [5] sums, [6], [7] the maxima's keys
    double *ll = nullptr; // the step's log-likelihoods, then its log-weights
    double *part = nullptr; // sums of blocks
    uint32_t *err = nullptr; // kErrWords words (resample_internal.cuh)
    Pf64Host *host = nullptr, *host_dev = nullptr;
    Scratch *work = nullptr; // the sums' buffers, ll
    SeqArgs seq = {};
    vsmc_cuda_rng reng = {};
    bool pending = false; // the engine has yet to pass the last resample
    size_t pending_n = 0; // its uniforms
};

namespace
{

constexpr int kSelB = 128;

// Move, log-likelihood and log-weight of every particle (into ll[0 .. n) and
// ll[n .. 2 n)); the largest log-weight into key[0], the largest
// log-likelihood into key[1].  The weights are read after a resample too: a
// caller may have written them (vsmc_cuda_pf_state).
__global__ void __launch_bounds__(kB64) k_move64(uint32_t n, uint32_t ld,
    uint32_t t, uint32_t seed, CvConst<double> c, const double *obs,
    double *s, double *ll, const double *W, unsigned long long *key)
{
    pdl_begin();
    const double ox = obs[2 * t + 0], oy = obs[2 * t + 1];
    unsigned long long m = 0, ml = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x) {
        const u32x4 w = particle_block(t, seed, i);
        double X, Y, VX, VY;
        double z1, z2;
        normal_pair_d(w.x, w.y, z1, z2);
        if (t == 0) {
            double z3, z4;
            normal_pair_d(w.z, w.w, z3, z4);
            X = __dmul_rn(c.sd_pos0, z1);
            Y = __dmul_rn(c.sd_pos0, z2);
            VX = __dmul_rn(c.sd_vel0, z3);
            VY = __dmul_rn(c.sd_vel0, z4);
        } else {
            X = s[i];
            Y = s[ld + i];
            VX = s[2 * ld + i];
            VY = s[3 * ld + i];
            cv_move(c, __dmul_rn(c.sigma_a, z1), __dmul_rn(c.sigma_a, z2), X,
                Y, VX, VY);
        }
        s[i] = X;
        s[ld + i] = Y;
        s[2 * ld + i] = VX;
        s[3 * ld + i] = VY;
        const double l = cv_loglik(c, ox, oy, X, Y);
        const double lw =
            t == 0 ? l : __dadd_rn(log_of_fraction(W[i]), l);
        ll[i] = l;
        ll[static_cast<size_t>(n) + i] = lw;
        m = max(m, max_key(lw));
        ml = max(ml, max_key(l));
    }
    __shared__ unsigned long long sh[2];
    m = warp_reduce(m, OpMax());
    ml = warp_reduce(ml, OpMax());
    if (threadIdx.x == 32) {
        sh[0] = m;
        sh[1] = ml;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicMax(key, max(m, sh[0]));
        atomicMax(key + 1, max(ml, sh[1]));
    }
}

// W = exp(lw - max), and the block's sum of W exp(l - max l) over the weights
// before the step (1 each at t == 0) into part.  The evidence is the log of
// these sums' tree sum, not of the left-to-right sum of the new weights: its
// n roundings in a row, and that of log(W) + l, made an increment's error
// 3e-15 at 2^14 and 2.4e-14 at 2^20 particles, against 1.5e-16.
__global__ void __launch_bounds__(kB64) k_exp64(uint32_t n, uint32_t t,
    const double *ll, double *W, const unsigned long long *key, double *part)
{
    pdl_begin();
    const double m = from_max_key(key[0]), ml = from_max_key(key[1]);
    double ev = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x) {
        const double e = exp_of_negative(ll[i] - ml);
        ev += t == 0 ? e : W[i] * e;
        W[i] = exp_of_negative(ll[static_cast<size_t>(n) + i] - m);
    }
    __shared__ double sh;
    ev = warp_reduce(ev, OpAdd());
    if (threadIdx.x == 32)
        sh = ev;
    __syncthreads();
    if (threadIdx.x == 0)
        part[blockIdx.x] = ev + sh;
}

// where a step's results go
struct Step64 {
    uint32_t n, t;
    double threshold;
    const double *state;
    size_t ld;
    double *W, *scal;
    double *h_mean, *h_ess, *h_logz;
    int *h_res;
    uint32_t *err;
    unsigned long long *key;
    const double *part; // the evidence's block sums
    uint32_t nb;
    Pf64Host *host;
};

// The step's records, by one thread: the evidence increment is
// log sum_i W_{t-1,i} exp(l_i) = max l + log(sum) with the sum of k_exp64's
// terms (over n equal weights at t = 0).
__device__ __forceinline__ void step64_record(
    const Step64 &a, double sum, double ess)
{
    const bool res = ess < a.threshold * static_cast<double>(a.n);
    const double mass = a.t == 0 ? sum / static_cast<double>(a.n) : sum;
    const double logz = (a.t == 0 ? 0.0 : a.scal[1]) +
        (from_max_key(a.key[1]) + log(mass));
    a.scal[0] = ess;
    a.scal[1] = logz;
    a.h_ess[a.t] = ess;
    a.h_logz[a.t] = logz;
    a.h_res[a.t] = res ? 1 : 0;
    a.key[0] = a.key[1] = 0; // for the next step's maxima
    a.host->err = atomicOr(a.err, 0u);
    // (the host reads these after waiting for the stream: no fence, which took
    // a microsecond of the step)
    a.host->resample = res ? 1 : 0;
}

__global__ void __launch_bounds__(kSeqBlock) k_record64(const Step64 a)
{
    pdl_begin();
    __shared__ double sh[kSeqBlock / 32 + 1];
    double sum = 0;
    for (uint32_t b = threadIdx.x; b < a.nb; b += kSeqBlock)
        sum += a.part[b];
    sum = block_reduce(sum, OpAdd(), 0.0, sh);
    if (threadIdx.x == 0)
        step64_record(a, sum, a.scal[5]);
}

// Normalization, ESS, records and (without a resample) the weighted mean of
// up to kSeqSmall particles, by one cluster.
__global__ void __launch_bounds__(kSeqBlock) k_weigh64(
    SeqArgs q, const Step64 a)
{
    pdl_begin();
    namespace cg = cooperative_groups;
    const cg::cluster_group cl = cg::this_cluster();
    SeqClusterSmem &S = seq_cluster_smem(q);
    __shared__ double s_inv, s_mass, s_mean[2], sh[kSeqBlock / 32 + 1];
    __shared__ bool s_res;
    const uint32_t tile = cl.block_rank();
    double w[kSeqItems], sq[kSeqItems];
    seq_load(SeqLoad{a.W}, tile, q.n, w);
    // the evidence's block sums (at most 256), by a warp of the first block
    // while another thread divides
    constexpr int kP = static_cast<int>(kSeqSmall) / kB64 / 32;
    const bool adds = tile == 0 && threadIdx.x >= 32 && threadIdx.x < 64;
    double part[kP];
#pragma unroll
    for (int k = 0; k < kP; ++k) {
        const uint32_t b = threadIdx.x % 32 + 32 * k;
        part[k] = adds && b < a.nb ? a.part[b] : 0.0;
    }
    const double total = seq_cluster_total(cl, q, w, S);
    if (threadIdx.x == 0)
        s_inv = 1.0 / total;
    if (adds) {
#pragma unroll
        for (int d = kP / 2; d > 0; d /= 2)
#pragma unroll
            for (int k = 0; k < d; ++k)
                part[k] += part[k + d];
        const double s = warp_reduce(part[0], OpAdd());
        if (threadIdx.x == 32)
            s_mass = s;
    }
    __syncthreads();
    const double inv = s_inv;
#pragma unroll
    for (int k = 0; k < kSeqItems; ++k) {
        const uint32_t i = seq_striped(tile, k);
        w[k] = __dmul_rn(inv, w[k]);
        if (i < q.n)
            a.W[i] = w[k];
        sq[k] = __dmul_rn(w[k], w[k]);
    }
    const double tsq = seq_cluster_total(cl, q, sq, S);
    if (threadIdx.x == 0) {
        const double ess = 1.0 / tsq;
        s_res = ess < a.threshold * static_cast<double>(a.n);
        if (tile == 0)
            step64_record(a, s_mass, ess);
    }
    __syncthreads();
    if (s_res) // the same in every block
        return;
    double m[2] = {0.0, 0.0};
#pragma unroll
    for (int k = 0; k < kSeqItems; ++k) {
        const uint32_t i = seq_striped(tile, k);
        if (i < q.n) {
            m[0] += w[k] * a.state[i];
            m[1] += w[k] * a.state[a.ld + i];
        }
    }
#pragma unroll
    for (int d = 0; d < 2; ++d) {
        const double v = block_reduce(m[d], OpAdd(), 0.0, sh);
        if (threadIdx.x == 0)
            s_mean[d] = v;
    }
    cl.sync();
    if (tile == 0 && threadIdx.x < 2) {
        double v = 0;
        for (uint32_t b = 0; b < cl.num_blocks(); ++b)
            v += *cl.map_shared_rank(&s_mean[threadIdx.x], b);
        a.h_mean[2 * a.t + threadIdx.x] = v;
    }
    cl.sync(); // the sums are read
}

// After a resample: particles copied to the empty slots (parents keep
// theirs, so in place), every weight 1 / n normalized, and the mean of the
// result: block sums, added by the last block (its ticket; nothing waits).
// After an error of the counts or slots nothing is copied: idx may be an
// earlier resample's then, whose copies from slots that are not parents would
// overlap.
__global__ void __launch_bounds__(kSelB) k_select64(
    const Step64 a, double *state, const int *idx, double *part)
{
    pdl_begin();
    __shared__ double sh[kSelB / 32 + 1];
    __shared__ bool last;
    const double w = a.scal[2];
    const bool copy = __ldcg(a.err) == 0;
    double m[2] = {0.0, 0.0};
    for (uint32_t i = blockIdx.x * kSelB + threadIdx.x; i < a.n;
         i += gridDim.x * kSelB) {
        const uint32_t j = copy ? static_cast<uint32_t>(idx[i]) : i;
        if (j >= a.n) {
            atomicOr(a.err, DEV_ERR_INTERNAL);
            continue;
        }
        const double x = state[j], y = state[a.ld + j];
        if (j != i) {
            const double vx = state[2 * a.ld + j], vy = state[3 * a.ld + j];
            state[i] = x;
            state[a.ld + i] = y;
            state[2 * a.ld + i] = vx;
            state[3 * a.ld + i] = vy;
        }
        a.W[i] = w;
        m[0] += w * x;
        m[1] += w * y;
    }
#pragma unroll
    for (int d = 0; d < 2; ++d) {
        const double v = block_reduce(m[d], OpAdd(), 0.0, sh);
        if (threadIdx.x == 0)
            part[2 * blockIdx.x + d] = v;
    }
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(a.err + kErrTicket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last)
        return;
    __threadfence();
#pragma unroll
    for (int d = 0; d < 2; ++d) {
        double v = 0;
        for (uint32_t b = threadIdx.x; b < gridDim.x; b += kSelB)
            v += __ldcg(part + 2 * b + d);
        v = block_reduce(v, OpAdd(), 0.0, sh);
        if (threadIdx.x == 0)
            a.h_mean[2 * a.t + d] = v;
    }
    if (threadIdx.x == 0) {
        a.err[kErrTicket] = 0;
        a.host->tail = a.err[kErrTail];
        a.host->err = atomicOr(a.err, 0u);
    }
}

__global__ void k_equal64(const double *W, double *scal)
{
    if (threadIdx.x == 0 && blockIdx.x == 0)
        scal[2] = W[0];
}

int select_grid(size_t n) { return grid_for(n, kSelB, 1, 4); }

} // namespace

int pf64_create(vsmc_cuda_pf *pf)
{
    Pf64State *p = new (std::nothrow) Pf64State;
    if (p == nullptr)
        return VSMC_CUDA_ERR_ALLOC;
    pf->p64 = p;
    const size_t n = pf->n;
    cudaStream_t st = pf->stream;
    auto get = [](auto **q, size_t bytes) {
        void *v = nullptr;
        const cudaError_t e = device_malloc(&v, bytes);
        *q = static_cast<std::remove_pointer_t<decltype(q)>>(v);
        return e == cudaSuccess;
    };
    const size_t blocks = std::max(2 * select_grid(n), grid64(n));
    if (!get(&p->rep, sizeof(int) * n) || !get(&p->idx, sizeof(int) * n) ||
        !get(&p->scal, sizeof(double) * 8) ||
        !get(&p->part, sizeof(double) * blocks) ||
        !get(&p->err, sizeof(uint32_t) * kErrWords) ||
        cudaHostAlloc(reinterpret_cast<void **>(&p->host), sizeof(Pf64Host),
            cudaHostAllocMapped) != cudaSuccess ||
        cudaHostGetDevicePointer(reinterpret_cast<void **>(&p->host_dev),
            p->host, 0) != cudaSuccess)
        return VSMC_CUDA_ERR_ALLOC;
    p->work = new (std::nothrow) Scratch(st);
    if (p->work == nullptr)
        return VSMC_CUDA_ERR_ALLOC;
    p->ll = p->work->get<double>(2 * n);
    if (p->ll == nullptr)
        return VSMC_CUDA_ERR_ALLOC;
    VSMC_CUDA_TRY(cudaMemsetAsync(p->err, 0, sizeof(uint32_t) * kErrWords, st));
    int rc = seq_args(n, p->err, false, *p->work, &p->seq);
    if (rc != VSMC_CUDA_OK)
        return rc;
    // the weight that Weight::set_equal leaves in every slot
    double *W = static_cast<double *>(pf->weight);
    {
        Scratch scratch(st);
        rc = weight_set_equal_device(n, W, nullptr, p->err, scratch, st);
        if (rc != VSMC_CUDA_OK)
            return rc;
    }
    k_equal64<<<1, 1, 0, st>>>(W, p->scal);
    VSMC_CUDA_CHECK_LAUNCH();
    return VSMC_CUDA_OK;
}

void pf64_destroy(vsmc_cuda_pf *pf)
{
    Pf64State *p = pf->p64;
    if (p == nullptr)
        return;
    delete p->work;
    cudaFree(p->rep);
    cudaFree(p->idx);
    cudaFree(p->scal);
    cudaFree(p->part);
    cudaFree(p->err);
    if (p->host)
        cudaFreeHost(p->host);
    delete p;
    pf->p64 = nullptr;
}

// both sums and the weights of more than kSeqSmall particles
static int weigh_large(vsmc_cuda_pf *pf, const Step64 &a)
{
    Pf64State *p = pf->p64;
    cudaStream_t st = pf->stream;
    SeqArgs q = p->seq;
    q.total = p->scal + 4;
    int rc = weight_sums(q, a.W, a.W, p->scal + 5, st);
    if (rc != VSMC_CUDA_OK)
        return rc;
    launch_after(k_record64, 1, kSeqBlock, 0, st, a);
    VSMC_CUDA_CHECK_LAUNCH();
    return VSMC_CUDA_OK;
}

int pf64_step(vsmc_cuda_pf *pf, bool first)
{
    Pf64State *p = pf->p64;
    cudaStream_t st = pf->stream;
    const size_t n = pf->n;
    const uint32_t t = static_cast<uint32_t>(pf->t);
    const bool small = n <= kSeqSmall;
    Step64 a = {};
    a.n = static_cast<uint32_t>(n);
    a.t = t;
    a.threshold = pf->threshold;
    a.state = static_cast<const double *>(pf->state);
    a.ld = pf->stride;
    a.W = static_cast<double *>(pf->weight);
    a.scal = p->scal;
    a.h_mean = pf->h_mean;
    a.h_ess = pf->h_ess;
    a.h_logz = pf->h_logz;
    a.h_res = pf->h_res;
    a.err = p->err;
    a.key = reinterpret_cast<unsigned long long *>(p->scal + 6);
    a.part = p->part;
    a.nb = static_cast<uint32_t>(grid64(n));
    a.host = p->host_dev;
    double *S = static_cast<double *>(pf->state);
    if (first) {
        // Sampler::initialize: resampling engine key {0, seed}, counter
        // {0, 0, 1, 0}
        vsmc_cuda_rng_init(&p->reng, VSMC_CUDA_PHILOX4X32, 0);
        const uint64_t key[2] = {0, pf->seed};
        vsmc_cuda_rng_set_key(&p->reng, 2, key);
        const uint64_t ctr[4] = {0, 0, 1, 0};
        vsmc_cuda_rng_set_ctr(&p->reng, 4, ctr);
        p->pending = false;
        VSMC_CUDA_TRY(
            cudaMemsetAsync(p->err, 0, sizeof(uint32_t) * kErrWords, st));
        VSMC_CUDA_TRY(cudaMemsetAsync(a.key, 0, 2 * sizeof(*a.key), st));
    }
    const CvConst<double> c = make_cv_const<double>(pf->model);
    launch_after(k_move64, a.nb, kB64, 0, st, a.n,
        static_cast<uint32_t>(a.ld), t, pf->seed, c, pf->obs, S, p->ll, a.W,
        a.key);
    launch_after(k_exp64, a.nb, kB64, 0, st, a.n, t, p->ll, a.W, a.key,
        p->part);
    VSMC_CUDA_CHECK_LAUNCH();
    int rc = small ? seq_cluster_launch(k_weigh64, p->seq, st, a)
                   : weigh_large(pf, a);
    if (rc != VSMC_CUDA_OK)
        return rc;
    VSMC_CUDA_TRY(cudaStreamSynchronize(st));
    rc = err_status(p->host->err);
    if (rc != VSMC_CUDA_OK)
        return rc;
    Scratch scratch(st);
    if (p->host->resample) {
        if (p->pending) { // the last resample's words are known by now
            scheme_advance(p->reng, n, p->pending_n, pf->scheme, p->host->tail);
            p->pending = false;
        }
        size_t N = 0;
        rc = scheme_enqueue(n, n, p->reng, a.W, p->rep, pf->scheme, p->err,
            &N, scratch, st);
        if (rc != VSMC_CUDA_OK)
            return rc;
        rc = rep_index_device(n, n, p->rep, p->idx, p->err, scratch, st);
        if (rc != VSMC_CUDA_OK)
            return rc;
        launch_after(k_select64, select_grid(n), kSelB, 0, st, a, S,
            p->idx, p->part);
        VSMC_CUDA_CHECK_LAUNCH();
        p->pending = true;
        p->pending_n = N;
    } else if (!small) {
        rc = monitor_mean_device<double>(
            n, 2, pf->stride, S, a.W, pf->h_mean + 2 * t, scratch, st);
    }
    return rc;
}

// Waits for the last step's resample and returns its errors, which the step's
// own wait did not see.
int pf64_finish(vsmc_cuda_pf *pf)
{
    VSMC_CUDA_TRY(cudaStreamSynchronize(pf->stream));
    return err_status(pf->p64->host->err);
}

} // namespace vsmc_cuda
