// vsmc_cuda_filter.cuh - the fused FP32 particle-filter step of libvsmc_cuda
// for any user model, compiled with nvcc (sm_103a) into the user's program.
//
// In the reference a model is the user's per-particle `eval_sp` inside a
// MoveBase / MoveOMP functor: eval_pre once per step, eval_sp per particle,
// eval_post once (smp/backend_base.hpp:243-363, smp/backend_omp.hpp:93-105),
// followed by Weight::add_log (core/weight.hpp:168-173).  Here the model is a
// device functor and one kernel does all of it: it reads every particle
// (through the resampling index after a resample), moves it, evaluates its
// log-likelihood, updates its FP32 log-weight and reduces, per block,
// (max, sum exp, sum exp^2) of the new log-weights and the weighted sums of
// the first `monitor_dim` state components.  The last block to finish
// combines the blocks' records in FP64 into the ESS, the log-evidence
// increment, the monitor mean and the resampling decision.  The library
// (vsmc_cuda.h) owns the buffers and the resampling passes; this header only
// adds the model-dependent kernel.  The library's own constant-velocity
// filter is an instance of the same template.
//
// A model is a trivially copyable struct (it is a kernel argument):
//
//   struct MyModel {
//       static constexpr int dim = 4;         // state components, <= 8
//       static constexpr int monitor_dim = 2; // leading components whose
//                                             // weighted mean is recorded
//       struct step_type { ... };             // per-step constants
//       // eval_pre: once per thread and step (t = step index)
//       __device__ step_type step(uint32_t t) const;
//       // t = 0: draw the initial particle (x is uninitialized on entry)
//       __device__ void init(const step_type &, vsmc_cuda::ParticleRng &,
//           float (&x)[dim]) const;
//       // t >= 1: propagate x in place (eval_sp)
//       __device__ void move(const step_type &, vsmc_cuda::ParticleRng &,
//           float (&x)[dim]) const;
//       // log g(y_t | x) of the moved particle, added to its log-weight
//       __device__ float log_likelihood(const step_type &,
//           const float (&x)[dim]) const;
//   };
//
// and one step is
//
//   vsmc_cuda_pf_step_desc d;
//   vsmc_cuda_pf_step_desc_get(pf, &d);         // buffers of the next step
//   vsmc_cuda::pf_step_launch(d, model);        // this header's kernel
//   vsmc_cuda_pf_step_commit(pf);               // resampling, next buffers
//
// (vsmc_cuda_sampler.cuh wraps this in Sampler<T> classes).  Randomness comes
// from the ParticleRng the kernel hands the model: the Philox4x32 stream
// with key {t, seed} and counters {1.., i, 0, 0} of particle i (the slot
// index, after resampling).
#ifndef VSMC_CUDA_FILTER_CUH
#define VSMC_CUDA_FILTER_CUH

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "vsmc_cuda.h"
#include "vsmc_cuda_device.cuh"

namespace vsmc_cuda
{

constexpr int kPfBlock = 256;
constexpr int kPfTile = kPfBlock * 4; // particles per block and tile
constexpr int kMaxFilterDim = 8;
constexpr int kMaxMonitorDim = 4;

// Device-side error word bits of the filter scalars (written with atomicOr).
enum : unsigned {
    DEV_ERR_NONFINITE = 1u, // NaN / inf / negative weight where forbidden
    DEV_ERR_BOUND = 2u,     // an exactness or iteration bound was exceeded
    DEV_ERR_INTERNAL = 4u,  // an index left its range
    DEV_ERR_TIMEOUT = 16u,  // a bounded wait gave up
};

// Device-resident filter scalars (one per filter; the library allocates
// them, this kernel and the library's resampling passes share the layout).
struct PfScalars {
    double M;    // max of the stored log-weights after the last weighting
    double S;    // sum exp(lw - M)
    double logz; // cumulative log-evidence
    double ess;
    double mean[kMaxMonitorDim]; // monitor: weighted mean after the step
    uint64_t Q;          // fixed-point CDF total of the pending resample
    uint64_t qrcp;       // floor((2^128 - 1) / (Q << qz)) - 2^64
    uint64_t qG;         // systematic: ceil(a Q / 2^32) for the shared word a
    uint64_t qgam;       // systematic: floor(2^64 qG / Q)
    uint64_t qm;         // floor(2^(64 + qs) n / Q) (when qs > 0)
    uint64_t qgs;        // floor(2^qs qG / Q)
    uint32_t qz;         // leading zero bits of Q
    uint32_t qs;         // fraction bits of the n / Q reciprocal (0: unused)
    uint32_t done3;      // completion counter of the resampling passes
    uint32_t step;       // next step index t
    int32_t resampled;   // last step resampled: weights equal, lw stale
    int32_t gather;      // state must be read through idx (after a resample)
    uint32_t done;       // completion counter of the fused step
    uint32_t done2;      // completion counter of the other reductions
    uint32_t err;        // DEV_ERR_* bits
    uint32_t nempty;     // empty slots of the pending resample
    uint32_t rindex;     // resampling engine: next word index in gen(rctr)
    uint32_t rkey[2];
    uint32_t rctr[4];
    float Mf; // M as a float (the batched filters' kernels read it per tile)
};

// Per-block record of the fused step: new log-weights' block max m, sum
// exp(lw - m), sum exp(2 (lw - m)), and sum exp(lw - m) x_d for the
// monitored components.
struct PfPartial {
    double m, s, s2;
    double mon[kMaxMonitorDim];
    double prev[kMaxMonitorDim]; // previous-step monitor sums (Previous)
    double prev_w;
};

// Kernel arguments (from vsmc_cuda_pf_step_desc).
struct PfStepArgs {
    const float *in; // state before the step: dim rows of `stride`
    float *out;      // state after the step
    float *lw;       // log-weights, updated in place
    const int32_t *idx;
    const uint32_t *srcs;
    PfPartial *part;
    PfScalars *sc;
    double *h_mean, *h_ess, *h_logz;
    int *h_res;
    size_t stride;
    uint32_t n, seed, max_steps;
    double threshold; // resample when ESS < threshold * n (< 0: never)
    int mon_prev;     // PfMon::Previous (the filter's own runs)
};

// ------------------------------------------------- weighted accumulation

// Running (max, sum exp, sum exp^2, monitored weighted sums) of log-weights,
// all relative to the running max, in FP32.  A plain aggregate (it also
// lives in shared memory); start from lse_empty().
template <int MD>
struct LseMon {
    float m, s, s2;
    float mon[MD > 0 ? MD : 1];

    // Both without branches: the side with the larger max keeps its sums,
    // the other's are scaled by e = exp(its max - the larger one).  A weight
    // that is -inf or NaN, and an empty side, add nothing (e = 0).
    template <int D>
    __device__ __forceinline__ void push(float v, const float (&x)[D])
    {
        const bool up = v > m;
        const bool ok = v > -INFINITY; // -inf and NaN carry no weight
        const float e = ok ? __expf(up ? m - v : v - m) : 0.0f;
        s = fmaf(up ? s : 1.0f, e, up ? 1.0f : s);
        s2 = fmaf((up ? s2 : 1.0f) * e, e, up ? 1.0f : s2);
#pragma unroll
        for (int d = 0; d < MD; ++d) {
            const float y = fmaf(up ? mon[d] : e, up ? e : x[d],
                up ? x[d] : mon[d]);
            mon[d] = ok ? y : mon[d];
        }
        m = up ? v : m;
    }

    __device__ __forceinline__ void merge(const LseMon &o)
    {
        const bool up = o.m > m;
        const float lo = up ? m : o.m, hi = up ? o.m : m;
        const float e = lo > -INFINITY ? __expf(lo - hi) : 0.0f;
        s = fmaf(up ? s : o.s, e, up ? o.s : s);
        s2 = fmaf((up ? s2 : o.s2) * e, e, up ? o.s2 : s2);
#pragma unroll
        for (int d = 0; d < MD; ++d)
            mon[d] = fmaf(up ? mon[d] : o.mon[d], e, up ? o.mon[d] : mon[d]);
        m = hi;
    }

    __device__ __forceinline__ LseMon shfl_xor(int lanes) const
    {
        LseMon o = *this;
        o.m = __shfl_xor_sync(0xFFFFFFFFu, m, lanes);
        o.s = __shfl_xor_sync(0xFFFFFFFFu, s, lanes);
        o.s2 = __shfl_xor_sync(0xFFFFFFFFu, s2, lanes);
#pragma unroll
        for (int d = 0; d < MD; ++d)
            o.mon[d] = __shfl_xor_sync(0xFFFFFFFFu, mon[d], lanes);
        return o;
    }
};

template <int MD>
__device__ __forceinline__ LseMon<MD> lse_empty()
{
    LseMon<MD> a;
    a.m = -INFINITY;
    a.s = 0.0f;
    a.s2 = 0.0f;
#pragma unroll
    for (int d = 0; d < (MD > 0 ? MD : 1); ++d)
        a.mon[d] = 0.0f;
    return a;
}

// ------------------------------------------------------------ particle I/O

__device__ __forceinline__ float4 pf_ld4(const float *p)
{
    return __ldcs(reinterpret_cast<const float4 *>(p));
}

__device__ __forceinline__ void pf_st4(float *p, float4 v)
{
    __stcs(reinterpret_cast<float4 *>(p), v);
}

__device__ __forceinline__ float pf_get(const float4 &v, int k)
{
    return k == 0 ? v.x : (k == 1 ? v.y : (k == 2 ? v.z : v.w));
}

__device__ __forceinline__ void pf_set(float4 &v, int k, float f)
{
    if (k == 0)
        v.x = f;
    else if (k == 1)
        v.y = f;
    else if (k == 2)
        v.z = f;
    else
        v.w = f;
}

// Source slot of slot i after a resample: idx[i] >= 0 is the slot itself
// (a parent keeps its slot), idx[i] = -(e + 1) is the e-th empty slot,
// filled from srcs[e] (the layout of resample/transform.hpp:116-133).
__device__ __forceinline__ uint32_t pf_source(
    const uint32_t *srcs, int32_t v)
{
    return v >= 0 ? static_cast<uint32_t>(v) : __ldcg(srcs + (-v - 1));
}

// Rows of particles i0..i0+3, gathered through the index after a resample.
// A group of four slots that all keep their own particles takes one float4
// per row.
template <int D>
__device__ __forceinline__ void pf_load_group(
    const PfStepArgs &a, uint32_t i0, bool gather, float4 (&R)[D])
{
    if (gather) {
        const int4 I = __ldcs(reinterpret_cast<const int4 *>(a.idx + i0));
        const int b = static_cast<int>(i0);
        if (I.x == b && I.y == b + 1 && I.z == b + 2 && I.w == b + 3) {
#pragma unroll
            for (int d = 0; d < D; ++d)
                R[d] = pf_ld4(a.in + d * a.stride + i0);
        } else {
            uint32_t s0 = pf_source(a.srcs, I.x);
            uint32_t s1 = pf_source(a.srcs, I.y);
            uint32_t s2 = pf_source(a.srcs, I.z);
            uint32_t s3 = pf_source(a.srcs, I.w);
            if (max(max(s0, s1), max(s2, s3)) >= a.n) {
                // an index outside the particles: record it, read slot 0
                atomicOr(&a.sc->err, DEV_ERR_INTERNAL);
                s0 = s0 < a.n ? s0 : 0;
                s1 = s1 < a.n ? s1 : 0;
                s2 = s2 < a.n ? s2 : 0;
                s3 = s3 < a.n ? s3 : 0;
            }
#pragma unroll
            for (int d = 0; d < D; ++d) {
                const float *r = a.in + d * a.stride;
                R[d] = make_float4(r[s0], r[s1], r[s2], r[s3]);
            }
        }
    } else {
#pragma unroll
        for (int d = 0; d < D; ++d)
            R[d] = pf_ld4(a.in + d * a.stride + i0);
    }
}

// The monitor's place in the step.  Current: the step's own weighted mean
// of the moved particles, reduced with the evidence (a host reading the
// monitor after every step, as Sampler<T> does).  Previous: the previous
// step's monitor, from the particles this step reads (weights
// exp(lw_prev - M_prev), or equal after a resample); the filter's own runs,
// where it costs one exponential and no pass after a resample.
enum class PfMon { Current, Previous };

template <int MD>
struct PrevSums {
    float x[MD > 0 ? MD : 1];
    float w;
};

// One particle: draw or move, weight, accumulate.
template <class Model, bool First, PfMon Mon, int MD, int AMD>
__device__ __forceinline__ void pf_particle(const Model &model,
    const typename Model::step_type &ctx, uint32_t t, uint32_t seed,
    uint32_t i, int resampled, float Mprev, float (&x)[Model::dim], float &lw,
    LseMon<AMD> &acc, PrevSums<MD> &prev)
{
    ParticleRng rng(t, seed, i);
    float lw_old = 0.0f;
    if (First) {
        model.init(ctx, rng, x);
    } else {
        lw_old = resampled ? 0.0f : lw - Mprev;
        if (Mon == PfMon::Previous) {
            const float wo = resampled ? 1.0f : __expf(lw_old);
#pragma unroll
            for (int d = 0; d < MD; ++d)
                prev.x[d] = fmaf(wo, x[d], prev.x[d]);
            prev.w += wo;
        }
        model.move(ctx, rng, x);
    }
    lw = lw_old + model.log_likelihood(ctx, x);
    acc.push(lw, x);
}

// ------------------------------------------------- FP64 block reductions
//
// An FP64 instruction of a warp takes 19 cycles of its SM, so the sums below
// split the values over the lanes as they go: NV values over 32 lanes in
// about NV + 4 additions, not 5 NV.  Every addition is the same pair as in a
// plain butterfly, so the results are the same bits.

// v[0..NV) summed over the warp; value k ends in lane warp_sum_lane<NV>(k)
// (in v[0] there).
template <int NV>
__device__ __forceinline__ void warp_sum_split(double (&v)[NV])
{
    const int lane = threadIdx.x & 31;
    int n = NV;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        if (n > 1) {
            const int h = (n + 1) / 2;
            const bool up = (lane & d) != 0;
#pragma unroll
            for (int i = 0; i < (NV + 1) / 2; ++i)
                if (i < h) {
                    const double hi = i + h < n ? v[i + h] : 0.0;
                    const double keep = up ? hi : v[i];
                    const double send = up ? v[i] : hi;
                    v[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, d);
                }
            n = h;
        } else {
            v[0] += __shfl_xor_sync(0xFFFFFFFFu, v[0], d);
        }
    }
}

template <int NV>
__host__ __device__ constexpr int warp_sum_lane(int k)
{
    int lane = 0, n = NV;
    for (int d = 16; d > 0; d >>= 1)
        if (n > 1) {
            const int h = (n + 1) / 2;
            if (k >= h) {
                lane |= d;
                k -= h;
            }
            n = h;
        }
    return lane;
}

// the value warp_sum_split leaves in the calling lane (NV and more: none)
template <int NV>
__device__ __forceinline__ int warp_sum_value()
{
    const int lane = threadIdx.x & 31;
    int v = NV;
#pragma unroll
    for (int k = 0; k < NV; ++k)
        if (lane == warp_sum_lane<NV>(k))
            v = k;
    return v;
}

// ------------------------------------------------------------ fused step

// Shared memory of a step's reductions.
template <class Model, PfMon Mon>
struct PfStepSmem {
    static constexpr int kW = kPfBlock / 32;
    static constexpr int AMD = Mon == PfMon::Current ? Model::monitor_dim : 0;
    LseMon<AMD> shw[kW];
    float shp[kMaxMonitorDim + 1][kW];
    double shd[2 + 2 * kMaxMonitorDim + 1][kW];
    float shmax[kW];
};

// One block's share of step t: its tiles of particles moved and weighted, and
// their sums left in *p (by warp 0; the caller orders the write).
template <class Model, bool First, PfMon Mon>
__device__ __forceinline__ void pf_step_record(const PfStepArgs &a,
    const Model &model, uint32_t t, int resampled, bool gather, float Mprev,
    PfPartial *p, PfStepSmem<Model, Mon> &sh)
{
    constexpr int D = Model::dim;
    constexpr int MD = Model::monitor_dim;
    // the evidence sums carry the monitor only for the current-step mode
    constexpr int AMD = Mon == PfMon::Current ? MD : 0;
    const typename Model::step_type ctx = model.step(t);
    const uint32_t n = a.n;
    LseMon<AMD> acc = lse_empty<AMD>();
    PrevSums<MD> prev;
#pragma unroll
    for (int d = 0; d < (MD > 0 ? MD : 1); ++d)
        prev.x[d] = 0.0f;
    prev.w = 0.0f;

    const uint32_t ntiles = (n + kPfTile - 1) / kPfTile;
    for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const uint32_t i0 = tile * kPfTile + threadIdx.x * 4;
        if (i0 + 3 < n) {
            float4 R[D];
            float4 LW = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (!First) {
                pf_load_group<D>(a, i0, gather, R);
                if (!resampled)
                    LW = pf_ld4(a.lw + i0);
            } else {
#pragma unroll
                for (int d = 0; d < D; ++d)
                    R[d] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                float x[D];
#pragma unroll
                for (int d = 0; d < D; ++d)
                    x[d] = pf_get(R[d], k);
                float l = pf_get(LW, k);
                pf_particle<Model, First, Mon, MD, AMD>(model, ctx, t, a.seed,
                    i0 + k, resampled, Mprev, x, l, acc, prev);
#pragma unroll
                for (int d = 0; d < D; ++d)
                    pf_set(R[d], k, x[d]);
                pf_set(LW, k, l);
            }
#pragma unroll
            for (int d = 0; d < D; ++d)
                pf_st4(a.out + d * a.stride + i0, R[d]);
            pf_st4(a.lw + i0, LW);
        } else {
            for (uint32_t i = i0; i < n && i < i0 + 4; ++i) {
                float x[D];
                float l = 0.0f;
                if (!First) {
                    uint32_t src = gather ? pf_source(a.srcs, a.idx[i]) : i;
                    if (src >= n) {
                        atomicOr(&a.sc->err, DEV_ERR_INTERNAL);
                        src = 0;
                    }
#pragma unroll
                    for (int d = 0; d < D; ++d)
                        x[d] = a.in[d * a.stride + src];
                    l = resampled ? 0.0f : a.lw[i];
                } else {
#pragma unroll
                    for (int d = 0; d < D; ++d)
                        x[d] = 0.0f;
                }
                pf_particle<Model, First, Mon, MD, AMD>(
                    model, ctx, t, a.seed, i, resampled, Mprev, x, l, acc,
                    prev);
#pragma unroll
                for (int d = 0; d < D; ++d)
                    a.out[d * a.stride + i] = x[d];
                a.lw[i] = l;
            }
        }
    }

    // ---- warp level in FP32
#pragma unroll
    for (int d = 16; d > 0; d >>= 1)
        acc.merge(acc.shfl_xor(d));
    constexpr bool prev_on = !First && Mon == PfMon::Previous;
    if (prev_on) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
            for (int d = 0; d < MD; ++d)
                prev.x[d] += __shfl_xor_sync(0xFFFFFFFFu, prev.x[d], o);
            prev.w += __shfl_xor_sync(0xFFFFFFFFu, prev.w, o);
        }
    }
    // ---- block level in FP32 (warp 0 merges the warps' records), then one
    // FP64 record per block
    constexpr int kW = kPfBlock / 32;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) {
        sh.shw[wid] = acc;
        if (prev_on) {
#pragma unroll
            for (int d = 0; d < MD; ++d)
                sh.shp[d][wid] = prev.x[d];
            sh.shp[kMaxMonitorDim][wid] = prev.w;
        }
    }
    __syncthreads();
    if (wid == 0) {
        LseMon<AMD> w = lse_empty<AMD>();
        if (lane < kW)
            w = sh.shw[lane];
#pragma unroll
        for (int d = kW / 2; d > 0; d >>= 1)
            w.merge(w.shfl_xor(d));
        if (lane == 0) {
            p->m = w.m;
            p->s = w.s;
            p->s2 = w.s2;
#pragma unroll
            for (int d = 0; d < kMaxMonitorDim; ++d)
                p->mon[d] = d < AMD ? w.mon[d < AMD ? d : 0] : 0.0;
        }
    } else if (wid == 1) {
        // the warps' monitor sums in FP64: eight lanes a component (the
        // last one, the weights), summed pairwise
        static_assert(kW == 8, "eight lanes a component");
        constexpr int kC = MD + 1;
#pragma unroll
        for (int c0 = 0; c0 <= kMaxMonitorDim; c0 += 4) {
            const int c = c0 + lane / 8;
            double x = prev_on && c < kC
                ? static_cast<double>(
                      sh.shp[c < MD ? c : kMaxMonitorDim][lane % 8])
                : 0.0;
            if (prev_on && c0 < kC)
#pragma unroll
                for (int o = 4; o > 0; o >>= 1)
                    x += __shfl_xor_sync(0xFFFFFFFFu, x, o);
            if (lane % 8 == 0 && c <= kMaxMonitorDim) {
                // component MD is the weights; unused ones are zero
                if (c == MD)
                    p->prev_w = x;
                else if (c < MD)
                    p->prev[c] = x;
                else
                    p->prev[c - 1] = 0.0;
            }
        }
    }
}

// The step's result from every block's record, in FP64, into sc (the
// filter's scalars) and, if write, the histories; by one whole block, whose
// warps 0 and 1 finish.  Every block that runs it gets the same bits.  Local:
// the records are this block's own (plain loads, shared memory allowed).
template <class Model, bool First, PfMon Mon, bool Local = false>
__device__ __forceinline__ void pf_step_combine(const PfStepArgs &a,
    const PfPartial *part, uint32_t nblk, PfScalars &sc, bool write,
    uint32_t t, int resampled, PfStepSmem<Model, Mon> &sh)
{
    constexpr int MD = Model::monitor_dim;
    constexpr int AMD = Mon == PfMon::Current ? MD : 0;
    constexpr bool prev_on = !First && Mon == PfMon::Previous;
    constexpr int kW = kPfBlock / 32;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t n = a.n;
    auto ld = [](const double *p) { return Local ? *p : __ldcg(p); };
    // S, S2, then the sums this mode has: the step's own monitor, or the
    // previous step's and its weights
    constexpr int NV = 2 + AMD + (prev_on ? MD + 1 : 0);
    const double prev_mass = resampled ? static_cast<double>(n) : sc.S;
    float M = -INFINITY;
    double tot = 0; // lane k of the finishing warps: value k
    if (nblk == 1) {
        // one record: the sums are its own (every factor is exp(M - M) = 1,
        // or not a number for an infinite M)
        M = static_cast<float>(ld(&part->m));
        if (lane < NV)
            tot = lane == 0 ? ld(&part->s)
                : lane == 1 ? ld(&part->s2)
                : lane < 2 + AMD ? ld(&part->mon[lane - 2])
                : lane < NV - 1  ? ld(&part->prev[lane - 2 - AMD])
                                 : ld(&part->prev_w);
        if (M == INFINITY && lane < 2 + AMD) // (no FP64 operation)
            tot = __longlong_as_double(0x7FF8000000000000ll);
        __syncthreads(); // sc.S is read
    } else {
        for (uint32_t b = threadIdx.x; b < nblk; b += blockDim.x)
            M = fmaxf(M, static_cast<float>(ld(&part[b].m)));
#pragma unroll
        for (int d = 16; d > 0; d >>= 1)
            M = fmaxf(M, __shfl_xor_sync(0xFFFFFFFFu, M, d));
        if (lane == 0)
            sh.shmax[wid] = M;
        __syncthreads();
        M = sh.shmax[0];
#pragma unroll
        for (int w = 1; w < kW; ++w)
            M = fmaxf(M, sh.shmax[w]);
        double v[NV] = {};
        if (wid * 32 < static_cast<int>(nblk)) { // records for this warp
            for (uint32_t b = threadIdx.x; b < nblk; b += blockDim.x) {
                const double pm = ld(&part[b].m);
                if (pm > -INFINITY) {
                    const double f = __expf(static_cast<float>(pm) - M);
                    v[0] += ld(&part[b].s) * f;
                    v[1] += ld(&part[b].s2) * f * f;
#pragma unroll
                    for (int d = 0; d < AMD; ++d)
                        v[2 + d] += ld(&part[b].mon[d]) * f;
                }
                if (prev_on) {
#pragma unroll
                    for (int d = 0; d < MD; ++d)
                        v[2 + AMD + d] += ld(&part[b].prev[d]);
                    v[NV - 1] += ld(&part[b].prev_w);
                }
            }
            warp_sum_split(v);
        }
        const int mine = warp_sum_value<NV>();
        if (mine < NV)
            sh.shd[mine][wid] = v[0];
        __syncthreads();
        if (lane < NV)
            for (int w = 0; w < kW && w * 32 < static_cast<int>(nblk); ++w)
                tot += sh.shd[lane][w];
    }
    // two warps finish, each with the totals: the quotients in the lanes of
    // warp 0, the logarithms in two lanes of warp 1
    if (wid > 1)
        return;
    const double S = __shfl_sync(0xFFFFFFFFu, tot, 0);
    const double M1 = static_cast<double>(M);
    const bool rec = write && t < a.max_steps;
    if (wid == 1) {
        const double lg = log(lane == 1 ? prev_mass : S);
        const double lg_prev = __shfl_sync(0xFFFFFFFFu, lg, 1);
        if (lane == 0) {
            sc.logz += M1 + lg - lg_prev;
            if (rec)
                a.h_logz[t] = sc.logz;
        }
        return;
    }
    const double S2 = __shfl_sync(0xFFFFFFFFu, tot, 1);
    const double PW = __shfl_sync(0xFFFFFFFFu, tot, NV - 1);
    // lane 1: ESS; a monitor component in its own lane: its mean
    const double quot = (lane == 1 ? S * S : tot) /
        (lane == 1 ? S2 : (prev_on && lane >= 2 + AMD ? PW : S));
    const double ess = __shfl_sync(0xFFFFFFFFu, quot, 1);
    if (prev_on && write && t >= 1 && t - 1 < a.max_steps && lane >= 2 + AMD &&
        lane < 2 + AMD + MD)
        a.h_mean[static_cast<size_t>(t - 1) * MD + (lane - 2 - AMD)] = quot;
    if (Mon == PfMon::Current && lane >= 2 && lane < 2 + MD) {
        sc.mean[lane - 2] = quot;
        if (rec)
            a.h_mean[static_cast<size_t>(t) * MD + (lane - 2)] = quot;
    }
    if (lane == 0) {
        if (!(S > 0) || !(ess > 0))
            sc.err |= DEV_ERR_NONFINITE;
        const int flag =
            ess < a.threshold * static_cast<double>(n) ? 1 : 0;
        if (rec) {
            a.h_ess[t] = ess;
            a.h_res[t] = flag;
        }
        sc.M = M1;
        sc.Mf = M;
        sc.S = S;
        sc.ess = ess;
        sc.resampled = flag;
        sc.gather = 0; // every block has read it; a resample sets it again
        sc.step = t + 1;
        sc.done = 0;
    }
}

template <class Model, bool First, PfMon Mon>
__global__ void __launch_bounds__(kPfBlock, 4) k_pf_step(
    const PfStepArgs a, const Model model)
{
    __shared__ PfStepSmem<Model, Mon> sh;
    __shared__ bool is_last;
    const uint32_t t = a.sc->step;
    const int resampled = First ? 1 : a.sc->resampled;
    const bool gather = First ? false : (a.sc->gather != 0);
    const float Mprev = First ? 0.0f : static_cast<float>(a.sc->M);
    pf_step_record<Model, First, Mon>(a, model, t, resampled, gather, Mprev,
        a.part + blockIdx.x, sh);
    if (threadIdx.x < 64)
        __threadfence();
    __syncthreads();
    if (threadIdx.x == 0)
        is_last = atomicAdd(&a.sc->done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!is_last)
        return;
    __threadfence();
    pf_step_combine<Model, First, Mon>(
        a, a.part, gridDim.x, *a.sc, true, t, resampled, sh);
}

// ------------------------------------------------------------ host launch

template <class Model, bool First, PfMon Mon>
inline int pf_step_occupancy()
{
    static int occ = 0;
    if (occ == 0) {
        int o = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                &o, k_pf_step<Model, First, Mon>, kPfBlock, 0) !=
                cudaSuccess ||
            o < 1)
            o = 1;
        occ = o;
    }
    return occ;
}

// Launch the fused step of `model` on the buffers of d (the next step of
// the filter d came from).  Returns a vsmc_cuda_status.
template <class Model>
inline int pf_step_launch(const vsmc_cuda_pf_step_desc &d, const Model &model)
{
    static_assert(Model::dim >= 1 && Model::dim <= kMaxFilterDim,
        "a model has 1 to 8 state components");
    static_assert(Model::monitor_dim >= 0 &&
            Model::monitor_dim <= kMaxMonitorDim &&
            Model::monitor_dim <= Model::dim,
        "monitor_dim is at most 4 and at most dim");
    if (d.dim != static_cast<size_t>(Model::dim) ||
        d.monitor_dim != static_cast<size_t>(Model::monitor_dim) ||
        d.state_in == nullptr || d.state_out == nullptr ||
        d.log_weight == nullptr || d.scalars == nullptr ||
        d.partials == nullptr || d.n == 0 || d.stride % 4 != 0)
        return VSMC_CUDA_ERR_ARG;
    PfStepArgs a;
    a.in = d.state_in;
    a.out = d.state_out;
    a.lw = d.log_weight;
    a.idx = d.index;
    a.srcs = d.sources;
    a.part = static_cast<PfPartial *>(d.partials);
    a.sc = static_cast<PfScalars *>(d.scalars);
    a.h_mean = d.hist_mean;
    a.h_ess = d.hist_ess;
    a.h_logz = d.hist_logz;
    a.h_res = d.hist_resampled;
    a.stride = d.stride;
    a.n = static_cast<uint32_t>(d.n);
    a.seed = d.seed;
    a.max_steps = static_cast<uint32_t>(d.max_steps);
    a.threshold = d.threshold;
    a.mon_prev = d.record_previous_mean;
    const bool first = d.step == 0;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) !=
            cudaSuccess)
        return VSMC_CUDA_ERR_CUDA;
    const bool prevmon = a.mon_prev != 0;
    const int occ = first
        ? (prevmon ? pf_step_occupancy<Model, true, PfMon::Previous>()
                   : pf_step_occupancy<Model, true, PfMon::Current>())
        : (prevmon ? pf_step_occupancy<Model, false, PfMon::Previous>()
                   : pf_step_occupancy<Model, false, PfMon::Current>());
    const size_t ntiles = (d.n + kPfTile - 1) / kPfTile;
    size_t grid = static_cast<size_t>(sms) * static_cast<size_t>(occ);
    if (grid > ntiles)
        grid = ntiles;
    if (grid > d.max_grid)
        grid = d.max_grid;
    if (grid < 1)
        return VSMC_CUDA_ERR_ARG;
    cudaStream_t st = static_cast<cudaStream_t>(d.stream);
    const unsigned g = static_cast<unsigned>(grid);
    if (first && prevmon)
        k_pf_step<Model, true, PfMon::Previous><<<g, kPfBlock, 0, st>>>(a,
            model);
    else if (first)
        k_pf_step<Model, true, PfMon::Current><<<g, kPfBlock, 0, st>>>(a,
            model);
    else if (prevmon)
        k_pf_step<Model, false, PfMon::Previous><<<g, kPfBlock, 0, st>>>(a,
            model);
    else
        k_pf_step<Model, false, PfMon::Current><<<g, kPfBlock, 0, st>>>(a,
            model);
    return cudaGetLastError() == cudaSuccess ? VSMC_CUDA_OK
                                             : VSMC_CUDA_ERR_CUDA;
}

} // namespace vsmc_cuda

#endif // VSMC_CUDA_FILTER_CUH
