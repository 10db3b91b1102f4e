// Batched FP32 bootstrap filters.
//
// Thousands of independent filters, each with its own particle count,
// horizon, model constants and seed, advance together: per global step one
// persistent kernel moves, weights and reduces the particles of every filter
// still running, and three kernels resample the filters whose ESS fell below
// the threshold, in equal units listed by the step kernel.  A whole run
// (every step of the longest horizon) is one CUDA graph.
//
// Filter f behaves exactly as a single precision-32 filter (pf.cu) with seed
// seeds[f]: the same particle streams (Philox4x32 key {step, seed}, counter
// {0, particle, 0, 0}), the same FP32 move / likelihood / log-weight
// arithmetic, the same resampling engine (key {0, seed}, counter {0, 0, 1, 0})
// and the same exact fixed-point counting, so its particles, counts and
// resampling decisions match; only the order of the FP64 block sums differs.
//
// Layout.  Filters are stored by horizon, longest first, so the filters still
// running at step t are a prefix and so are their tiles (a tile is
// kBlock * kPPT consecutive particles of one filter).  Particle arrays are the
// filters' segments concatenated, each starting on a multiple of 4 elements.
// Resampling indices are local to the filter's segment.
//
// The step and tile shapes (threads per block, particles per thread) are
// chosen by vsmc_cuda_batch_autotune from timed runs of the actual batch.
//
// No reference counterpart: the reference would run one Sampler<T> per
// filter (core/sampler.hpp:107-114) with the pf example's move
// (example/pf/include/pf.hpp:154-170).
#include "bearings.cuh"
#include "cv_sim.cuh"
#include "mlp.cuh"
#include "pf32_dev.cuh"
#include "pf_model.cuh"

#include <cuda_pipeline.h>

#include <algorithm>
#include <type_traits>
#include <cmath>
#include <cstring>
#include <new>
#include <vector>

using namespace vsmc_cuda;

namespace vsmc_cuda
{

// Static description of one filter (internal order).
struct BFilter {
    uint32_t n;        // particles
    uint32_t off;      // first particle in the concatenated arrays
    uint32_t tile0;    // first tile of the step kernel
    uint32_t ntiles;   // tiles of the step kernel
    uint32_t T;        // horizon: steps 0..T-1, step T records the last mean
    uint32_t obs_off;  // first observation pair (caller's filter order)
    uint32_t hist_off; // first history entry (caller's filter order)
    uint32_t seed;
    uint32_t shift;    // fixed-point K = 63 - ceil(log2 n)
    uint32_t rs_unit;  // particles of a resampling unit (a warp's)
    union {
        CvConst<float> c;   // position / Student-t model
        BearingsConst bc;   // bearings-only model
    };
};

// A block's record of the tiles of one filter: FP32 sums, as the block
// forms them (the single filter widens the same values to FP64).
struct TileRecord {
    float sx, sy, sw; // previous-step monitor sums
    float m, s, s2;   // new log-weights: max, sum exp, sum exp^2
};

// filter kinds
constexpr int kKindCv = 0;       // CV + Student-t positions, bootstrap
constexpr int kKindBearings = 1; // bearings-only, bootstrap
constexpr int kKindLearned = 2;  // bearings-only, learned proposal

struct BatchArgs {
    const BFilter *flt;
    PfScalars *st;               // dynamic state, one per filter
    const uint4 *segs;      // {first tile, tiles, filter, 0} of each segment
    const uint32_t *active; // [tmax + 1] segments of the filters with T >= t
    const float *ax, *ay, *avx, *avy; // state in
    float *bx, *by, *bvx, *bvy;       // state out
    float *lw;
    int32_t *rep, *idx;
    uint32_t *srcs;
    TileRecord *part; // per tile
    const float *obs; // the observations in FP32 (converted once per run)
    const float2 *obs_sc; // bearings kinds: (sin z, cos z) of each bearing
    double *h_mean, *h_ess, *h_logz;
    int *h_res;
    uint32_t *step; // global step counter
    // resampling list of the step: rs_list[rpar * rs_cap + v] = {filter,
    // unit}, rs_count[rpar] entries; per-entry totals of the passes, turned
    // into prefixes by the filter's last unit
    uint2 *rs_list;
    uint32_t *rs_count;
    uint32_t *work; // step kernel's segment counters, by step parity
    uint64_t *rs_q;  // CDF
    uint64_t *rs_ec; // copies (high half) and empty slots
    uint32_t rs_cap, rpar;
    const uint32_t *packed; // proposal network (learned kind)
    uint32_t nfilters, tmax;
    int scheme;
    double threshold;
};

// The FP32 per-particle body of the single filter (step_one in pf32.cuh),
// with the filter's constants and seed.
template <bool First>
__device__ __forceinline__ void batch_one(const CvConst<float> &c,
    uint32_t seed, uint32_t i, uint32_t t, float ox, float oy, int resampled,
    float Mprev, float &x, float &y, float &vx, float &vy, float &lw, float &m,
    float &s, float &s2, float &sx, float &sy, float &sw)
{
    const u32x4 w = particle_block(t, seed, i);
    float lw_old = 0.0f;
    if (First) {
        float z1, z2, z3, z4;
        normal_pair_f(w.x, w.y, z1, z2);
        normal_pair_f(w.z, w.w, z3, z4);
        x = c.sd_pos0 * z1;
        y = c.sd_pos0 * z2;
        vx = c.sd_vel0 * z3;
        vy = c.sd_vel0 * z4;
    } else {
        lw_old = resampled ? 0.0f : lw - Mprev;
        const float wo = resampled ? 1.0f : __expf(lw_old);
        sx += wo * x;
        sy += wo * y;
        sw += wo;
        float z1, z2;
        normal_pair_f(w.x, w.y, z1, z2);
        cv_move(c, c.sigma_a * z1, c.sigma_a * z2, x, y, vx, vy);
    }
    lw = lw_old + cv_loglik(c, ox, oy, x, y);
    lse_push(lw, m, s, s2);
}

__device__ __forceinline__ void load_run(const int32_t *p, int32_t (&v)[4])
{
    const int4 q = __ldcs(reinterpret_cast<const int4 *>(p));
    v[0] = q.x;
    v[1] = q.y;
    v[2] = q.z;
    v[3] = q.w;
}

__device__ __forceinline__ void load_run(const int32_t *p, int32_t (&v)[2])
{
    const int2 q = __ldcs(reinterpret_cast<const int2 *>(p));
    v[0] = q.x;
    v[1] = q.y;
}

__device__ __forceinline__ void load_run(const int32_t *p, int32_t (&v)[1])
{
    v[0] = __ldcs(p);
}

template <int kPPT>
__device__ __forceinline__ void load_run(const float *p, float (&v)[kPPT])
{
    if constexpr (kPPT == 4) {
        const float4 q = __ldcs(reinterpret_cast<const float4 *>(p));
        v[0] = q.x;
        v[1] = q.y;
        v[2] = q.z;
        v[3] = q.w;
    } else if constexpr (kPPT == 2) {
        const float2 q = __ldcs(reinterpret_cast<const float2 *>(p));
        v[0] = q.x;
        v[1] = q.y;
    } else {
        v[0] = __ldcs(p);
    }
}

template <int kPPT>
__device__ __forceinline__ void store_run(float *p, const float (&v)[kPPT])
{
    if constexpr (kPPT == 4) {
        __stcs(reinterpret_cast<float4 *>(p),
            make_float4(v[0], v[1], v[2], v[3]));
    } else if constexpr (kPPT == 2) {
        __stcs(reinterpret_cast<float2 *>(p), make_float2(v[0], v[1]));
    } else {
        __stcs(p, v[0]);
    }
}

// What a block needs to know of a segment (consecutive tiles of one filter),
// in shared memory: loaded while the block works on the segment before.
struct SegMeta {
    BFilter F;
    uint32_t tile, count, f; // count 0: no more segments
    int32_t resampled, gather;
    float Mf;
};

// The segment with number idx (>= nseg: none), by one warp, without waiting
// for it (cp.async; the caller waits and synchronizes).
__device__ __forceinline__ void seg_fetch(
    const BatchArgs &a, uint32_t idx, uint32_t nseg, SegMeta &m)
{
    const uint32_t lane = threadIdx.x & 31;
    if (idx >= nseg) {
        if (lane == 0)
            m.count = 0;
        return;
    }
    const uint4 seg = a.segs[idx];
    if (lane == 0) {
        m.tile = seg.x;
        m.count = seg.y;
        m.f = seg.z;
    }
    static_assert(sizeof(BFilter) % 4 == 0, "whole words");
    const uint32_t *src = reinterpret_cast<const uint32_t *>(a.flt + seg.z);
    uint32_t *dst = reinterpret_cast<uint32_t *>(&m.F);
    for (uint32_t w = lane; w < sizeof(BFilter) / 4; w += 32)
        __pipeline_memcpy_async(dst + w, src + w, 4);
    const PfScalars &S = a.st[seg.z];
    if (lane == 0)
        __pipeline_memcpy_async(&m.resampled, &S.resampled, 4);
    else if (lane == 1)
        __pipeline_memcpy_async(&m.gather, &S.gather, 4);
    else if (lane == 2)
        __pipeline_memcpy_async(&m.Mf, &S.Mf, 4);
    __pipeline_commit();
}

// a segment's sums of each warp
template <int kW>
struct SegSums {
    float v[6][kW]; // m, s, s2, sx, sy, sw
};

// the warp's sums over its lanes, left in sums
template <int kW>
__device__ __forceinline__ void seg_record_warp(SegSums<kW> &sums, float m,
    float s, float s2, float sx, float sy, float sw)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        const float om = __shfl_xor_sync(0xFFFFFFFFu, m, d);
        const float os = __shfl_xor_sync(0xFFFFFFFFu, s, d);
        const float os2 = __shfl_xor_sync(0xFFFFFFFFu, s2, d);
        sx += __shfl_xor_sync(0xFFFFFFFFu, sx, d);
        sy += __shfl_xor_sync(0xFFFFFFFFu, sy, d);
        sw += __shfl_xor_sync(0xFFFFFFFFu, sw, d);
        lse_merge_f(m, s, s2, om, os, os2);
    }
    if (lane == 0) {
        sums.v[0][wid] = m;
        sums.v[1][wid] = s;
        sums.v[2][wid] = s2;
        sums.v[3][wid] = sx;
        sums.v[4][wid] = sy;
        sums.v[5][wid] = sw;
    }
}

// The record of a segment from its warps' sums (FP32 within the segment,
// FP64 across), written at its first tile (its other tiles get empty
// records) and, when it completes the filter's last tile, the filter's FP64
// combination: ESS, log-evidence increment, resampling decision and
// histories (or, at t == T, the last weighted mean).  By one warp; the other
// warps of the block go on with the next segment.
template <int kW, bool First>
__device__ __forceinline__ void seg_finish(const BatchArgs &a,
    const SegMeta &meta, uint32_t t, bool mon, const SegSums<kW> &sums)
{
    const int lane = threadIdx.x & 31;
    const BFilter &F = meta.F;
    const uint32_t tile = meta.tile, count = meta.count, f = meta.f;
    PfScalars &S = a.st[f];
    {
        // merges the warps' records in FP32
        const bool in = lane < kW;
        float wm = in ? sums.v[0][lane] : -INFINITY;
        float ws = in ? sums.v[1][lane] : 0.0f;
        float ws2 = in ? sums.v[2][lane] : 0.0f;
        float wx = in ? sums.v[3][lane] : 0.0f;
        float wy = in ? sums.v[4][lane] : 0.0f;
        float ww = in ? sums.v[5][lane] : 0.0f;
#pragma unroll
        for (int d = kW / 2; d > 0; d >>= 1) {
            const float om = __shfl_xor_sync(0xFFFFFFFFu, wm, d);
            const float os = __shfl_xor_sync(0xFFFFFFFFu, ws, d);
            const float os2 = __shfl_xor_sync(0xFFFFFFFFu, ws2, d);
            wx += __shfl_xor_sync(0xFFFFFFFFu, wx, d);
            wy += __shfl_xor_sync(0xFFFFFFFFu, wy, d);
            ww += __shfl_xor_sync(0xFFFFFFFFu, ww, d);
            lse_merge_f(wm, ws, ws2, om, os, os2);
        }
        int last = 0;
        if (lane == 0) {
            const TileRecord p = {wx, wy, ww, wm, ws, ws2};
            a.part[tile] = p;
            const TileRecord empty = {0, 0, 0, -INFINITY, 0, 0};
            for (uint32_t k = 1; k < count; ++k)
                a.part[tile + k] = empty;
            __threadfence();
            last = atomicAdd(&S.done, count) == F.ntiles - count ? 1 : 0;
        }
        if (!__shfl_sync(0xFFFFFFFFu, last, 0))
            return;
    }
    __threadfence();
    // ---- the filter's last tile: its tile records in FP64
    float M = -INFINITY;
    for (uint32_t b = lane; b < F.ntiles; b += 32)
        M = fmaxf(M, __ldcg(&a.part[F.tile0 + b].m));
    M = warp_reduce(M, OpMax());
    // T1, T2, TX, TY, TW; the values are split over the lanes as they are
    // summed, and the quotients and logarithms taken in different lanes (an
    // FP64 instruction takes 19 cycles of the SM and 64 of latency)
    double v[5] = {};
    for (uint32_t b = lane; b < F.ntiles; b += 32) {
        const float2 *q =
            reinterpret_cast<const float2 *>(a.part + F.tile0 + b);
        const float2 q0 = __ldcg(q), q1 = __ldcg(q + 1), q2 = __ldcg(q + 2);
        const TileRecord p = {q0.x, q0.y, q1.x, q1.y, q2.x, q2.y};
        v[2] += p.sx;
        v[3] += p.sy;
        v[4] += p.sw;
        if (p.m > -INFINITY) {
            const double fct = __expf(p.m - M);
            v[0] += p.s * fct;
            v[1] += p.s2 * fct * fct;
        }
    }
    warp_sum_split(v);
    const double T1 = __shfl_sync(0xFFFFFFFFu, v[0], warp_sum_lane<5>(0));
    const double T2 = __shfl_sync(0xFFFFFFFFu, v[0], warp_sum_lane<5>(1));
    const double TX = __shfl_sync(0xFFFFFFFFu, v[0], warp_sum_lane<5>(2));
    const double TY = __shfl_sync(0xFFFFFFFFu, v[0], warp_sum_lane<5>(3));
    const double TW = __shfl_sync(0xFFFFFFFFu, v[0], warp_sum_lane<5>(4));
    // the previous weights' mass: their own normalizer (the single filter's
    // step kernel uses the same one)
    const double prev_mass =
        First || S.resampled ? static_cast<double>(F.n) : S.S;
    const double quot = (lane == 0 ? T1 * T1 : lane == 1 ? TX : TY) /
        (lane == 0 ? T2 : TW);
    const double lg = mon ? 0.0 : log(lane == 1 ? prev_mass : T1);
    const double mx = __shfl_sync(0xFFFFFFFFu, quot, 1);
    const double my = __shfl_sync(0xFFFFFFFFu, quot, 2);
    const double lg_prev = __shfl_sync(0xFFFFFFFFu, lg, 1);
    uint32_t rs_first = ~0u; // first list entry of the filter's units
    const uint32_t nu = (F.n + F.rs_unit - 1) / F.rs_unit;
    if (lane == 0) {
        if (mon) {
            a.h_mean[2 * (F.hist_off + F.T - 1) + 0] = mx;
            a.h_mean[2 * (F.hist_off + F.T - 1) + 1] = my;
            S.resampled = 0; // finished: nothing left to resample
            S.gather = 0;
        } else {
            if (!First) {
                a.h_mean[2 * (F.hist_off + t - 1) + 0] = mx;
                a.h_mean[2 * (F.hist_off + t - 1) + 1] = my;
            }
            const double ess = quot;
            const double M1 = static_cast<double>(M);
            S.logz += M1 + lg - lg_prev;
            if (!(T1 > 0) || !(ess > 0))
                S.err |= DEV_ERR_NONFINITE;
            const int flag =
                ess < a.threshold * static_cast<double>(F.n) ? 1 : 0;
            a.h_ess[F.hist_off + t] = ess;
            a.h_logz[F.hist_off + t] = S.logz;
            a.h_res[F.hist_off + t] = flag;
            S.M = M1;
            S.Mf = M;
            S.S = T1;
            S.ess = ess;
            S.resampled = flag;
            S.gather = 0;
            S.step = t + 1;
            if (flag) {
                const uint32_t v = atomicAdd(a.rs_count + a.rpar, nu);
                if (v + nu <= a.rs_cap)
                    rs_first = v;
                else
                    S.err |= DEV_ERR_INTERNAL;
            }
        }
        S.done = 0;
    }
    rs_first = __shfl_sync(0xFFFFFFFFu, rs_first, 0);
    if (rs_first != ~0u) {
        // list the filter's resampling units
        uint2 *list = a.rs_list + static_cast<size_t>(a.rpar) * a.rs_cap;
        for (uint32_t j = lane; j < nu; j += 32)
            list[rs_first + j] = make_uint2(f, j);
    }
}

// the sources, inside the filter, of kN slots with index entries I after a
// resample (bounds-checked); their loads are in flight together
template <int kN>
__device__ __forceinline__ void batch_sources(const BatchArgs &a,
    const BFilter &F, PfScalars &S, const int32_t (&I)[kN],
    uint32_t (&src)[kN])
{
    uint32_t most = 0;
#pragma unroll
    for (int k = 0; k < kN; ++k) {
        const uint32_t e = static_cast<uint32_t>(-(I[k] + 1));
        src[k] = I[k] >= 0 ? static_cast<uint32_t>(I[k])
                           : (e < F.n ? __ldcg(a.srcs + F.off + e) : F.n);
    }
#pragma unroll
    for (int k = 0; k < kN; ++k)
        most = max(most, src[k]);
    if (most >= F.n) {
        atomicOr(&S.err, DEV_ERR_INTERNAL);
#pragma unroll
        for (int k = 0; k < kN; ++k)
            src[k] = src[k] < F.n ? src[k] : 0;
    }
}

// bootstrap body of the bearings-only model (prior at t == 0)
template <bool First>
__device__ __forceinline__ void bearings_one(const BearingsConst &c,
    uint32_t seed, uint32_t i, uint32_t t, float z, int resampled,
    float Mprev, float &x, float &y, float &vx, float &vy, float &lw, float &m,
    float &s, float &s2, float &sx, float &sy, float &sw)
{
    float e[4];
    bearings_normals(t, seed, i, e);
    float lw_old = 0.0f;
    if (First) {
        bearings_prior(c, e, x, y, vx, vy);
    } else {
        lw_old = resampled ? 0.0f : lw - Mprev;
        const float wo = resampled ? 1.0f : __expf(lw_old);
        sx += wo * x;
        sy += wo * y;
        sw += wo;
        bearings_step(c, e, x, y, vx, vy);
    }
    lw = lw_old + bearings_loglik(c, z, x, y);
    lse_push(lw, m, s, s2);
}

// Tiles of a segment at most: one at the default 4 x 256 shape (1024
// particles, whose FP32 records then group the particles as the single
// filter's blocks do), 2048 particles' worth for smaller tiles (fewer
// records; 1024 took 231 ms per 4096-filter run, 2048 225 ms, 4096 227 ms).
constexpr uint32_t seg_tiles(uint32_t tile)
{
    return tile >= 1024 ? 1u : 2048u / tile;
}

// One global step of every running filter (bootstrap kinds).  A filter at
// t < T moves and weights its particles; at t == T it only records the
// weighted mean of its final particles.  A persistent block takes segments
// from a counter until none is left, so one whose segments are slower
// (gathered reads after a resample, many small filters) takes fewer.  The
// next segment's number and description are fetched while the current one
// is computed, and one warp (in turn) records a finished segment while the
// others start on the next: with three barriers and the chain counter, tile,
// filter, state in front of every segment's loads, a tile of 1024 particles
// took 10 us.  The registers bound the blocks of an SM: 512
// filters, 100 steps, took 10.62 ms with 64 registers (4 blocks of 256),
// 12.02 with 48 (5 blocks) and 10.91 with 80 (3 blocks).
template <int kBlock, int kPPT, bool First, int Kind>
__global__ void __launch_bounds__(kBlock, 1024 / kBlock) k_batch_step(
    const BatchArgs a)
{
    pdl_wait();
    constexpr uint32_t kTile = kBlock * kPPT;
    constexpr int kW = kBlock / 32;
    const uint32_t t = *a.step;
    const uint32_t nseg = t <= a.tmax ? a.active[t] : 0u;
    // a block's slots: a description is read by its segment's recorder until
    // the next segment's barrier, so three of them
    __shared__ SegMeta metas[3];
    __shared__ SegSums<kW> sums[2];
    const uint32_t lane = threadIdx.x & 31;
    const int wid = threadIdx.x >> 5;
    // the next step's counter was last used by the previous step's launch
    if (blockIdx.x == 0 && threadIdx.x == 0)
        a.work[(t + 1) & 1u] = 0;
    if (wid == kW - 1) {
        seg_fetch(a, blockIdx.x, nseg, metas[0]);
        __pipeline_wait_prior(0);
    }
    __syncthreads();
    uint32_t slot = 0;
    for (uint32_t it = 0;; ++it) {
        const SegMeta &meta = metas[slot];
        slot = slot == 2 ? 0 : slot + 1;
        if (meta.count == 0)
            break;
        uint32_t next = 0;
        if (wid == kW - 1 && lane == 0)
            next = gridDim.x + atomicAdd(a.work + (t & 1u), 1u);
        const BFilter &F = meta.F;
        const bool mon = !First && t == F.T;
        const int resampled = First ? 1 : meta.resampled;
        const bool gather = First ? false : (meta.gather != 0);
        const float Mprev = First ? 0.0f : meta.Mf;
        float ox = 0.0f, oy = 0.0f;
        if (!mon) {
            if (Kind == kKindCv) {
                ox = a.obs[2 * (F.obs_off + t) + 0];
                oy = a.obs[2 * (F.obs_off + t) + 1];
            } else {
                ox = a.obs[F.obs_off + t];
            }
        }
        float m = -INFINITY, s = 0, s2 = 0, sx = 0, sy = 0, sw = 0;
        const uint32_t end = meta.tile + meta.count;
        for (uint32_t tile = meta.tile; tile < end; ++tile) {
            const uint32_t i0 = (tile - F.tile0) * kTile + threadIdx.x * kPPT;
            const uint32_t g0 = F.off + i0;
            // one particle: weight its sums, move it and weight it, or (at
            // t == T) weight its sums alone
            auto body = [&](uint32_t i, float &x, float &y, float &vx,
                            float &vy, float &lw) {
                if (mon) {
                    const float wo = resampled ? 1.0f : __expf(lw - Mprev);
                    sx += wo * x;
                    sy += wo * y;
                    sw += wo;
                } else if (Kind == kKindCv) {
                    batch_one<First>(F.c, F.seed, i, t, ox, oy, resampled,
                        Mprev, x, y, vx, vy, lw, m, s, s2, sx, sy, sw);
                } else {
                    bearings_one<First>(F.bc, F.seed, i, t, ox, resampled,
                        Mprev, x, y, vx, vy, lw, m, s, s2, sx, sy, sw);
                }
            };
            const bool fetch = wid == kW - 1 && tile == meta.tile;
            if (i0 + kPPT <= F.n) {
                // a whole group: no test per particle, so its particles'
                // chains interleave
                float X[kPPT], Y[kPPT], VX[kPPT], VY[kPPT], LW[kPPT];
                if (First) {
#pragma unroll
                    for (int k = 0; k < kPPT; ++k)
                        X[k] = Y[k] = VX[k] = VY[k] = LW[k] = 0.0f;
                } else {
                    int32_t I[kPPT];
                    // after a resample, a group whose slots all keep their
                    // own particle reads like an unresampled one
                    bool own = true;
                    if (gather) {
                        load_run(a.idx + g0, I);
#pragma unroll
                        for (int k = 0; k < kPPT; ++k)
                            own = own && I[k] == static_cast<int>(i0) + k;
                    }
                    if (own) {
                        load_run<kPPT>(a.ax + g0, X);
                        load_run<kPPT>(a.ay + g0, Y);
                        load_run<kPPT>(a.avx + g0, VX);
                        load_run<kPPT>(a.avy + g0, VY);
                    } else {
                        uint32_t src[kPPT];
                        batch_sources<kPPT>(a, F, a.st[meta.f], I, src);
#pragma unroll
                        for (int k = 0; k < kPPT; ++k) {
                            X[k] = a.ax[F.off + src[k]];
                            Y[k] = a.ay[F.off + src[k]];
                            VX[k] = a.avx[F.off + src[k]];
                            VY[k] = a.avy[F.off + src[k]];
                        }
                    }
                    if (!resampled) {
                        load_run<kPPT>(a.lw + g0, LW);
                    } else {
#pragma unroll
                        for (int k = 0; k < kPPT; ++k)
                            LW[k] = 0.0f;
                    }
                }
#pragma unroll
                for (int k = 0; k < kPPT; ++k)
                    body(i0 + k, X[k], Y[k], VX[k], VY[k], LW[k]);
                if (!mon) {
                    store_run<kPPT>(a.bx + g0, X);
                    store_run<kPPT>(a.by + g0, Y);
                    store_run<kPPT>(a.bvx + g0, VX);
                    store_run<kPPT>(a.bvy + g0, VY);
                    store_run<kPPT>(a.lw + g0, LW);
                }
            } else {
#pragma unroll 1
                for (uint32_t i = i0; i < F.n && i < i0 + kPPT; ++i) {
                    const uint32_t g = F.off + i;
                    float x = 0, y = 0, vx = 0, vy = 0, lw = 0;
                    if (!First) {
                        uint32_t src[1] = {i};
                        if (gather) {
                            const int32_t I[1] = {a.idx[g]};
                            batch_sources<1>(a, F, a.st[meta.f], I, src);
                        }
                        x = a.ax[F.off + src[0]];
                        y = a.ay[F.off + src[0]];
                        vx = a.avx[F.off + src[0]];
                        vy = a.avy[F.off + src[0]];
                        if (!resampled)
                            lw = a.lw[g];
                    }
                    body(i, x, y, vx, vy, lw);
                    if (!mon) {
                        a.bx[g] = x;
                        a.by[g] = y;
                        a.bvx[g] = vx;
                        a.bvy[g] = vy;
                        a.lw[g] = lw;
                    }
                }
            }
            __syncwarp();
            if (fetch)
                seg_fetch(a, __shfl_sync(0xFFFFFFFFu, next, 0), nseg,
                    metas[slot]);
        }
        seg_record_warp(sums[it & 1], m, s, s2, sx, sy, sw);
        if (wid == kW - 1)
            __pipeline_wait_prior(0);
        __syncthreads();
        if (static_cast<uint32_t>(wid) == it % kW)
            seg_finish<kW, First>(a, meta, t, mon, sums[it & 1]);
    }
}

// A learned segment is up to 1024 particles: 8 tiles of 128, 32 particles a
// warp.  A block of 8 warps evaluates 2 tiles at a time, one of 4 warps one;
// then 4 warps take the sums, each lane over its particle of tile after tile.
constexpr uint32_t kLearnTile = 128;
constexpr uint32_t kLearnSeg = 1024u / kLearnTile; // tiles of a segment

// One global step of the learned-proposal filters.  A tile's evaluation is a
// chain of about 1560 instructions a warp: with four warps a segment, 64
// filters of 4096 particles (256 segments) left an SM 8 warps, each with
// eight evaluations in turn.  Two blocks of 8 warps, four tiles each,
// take the 50 steps (resampling included) from 3.06 to 2.45 ms; one block of
// 16 took 2.81, two of 16 (64 registers) 2.56.  With more segments than those
// blocks (two an SM) hold at once the SMs are full either way and four blocks
// of 4 warps lose less at the segments' ends: 20 steps of 128 filters of 4096
// take 1.43 ms against 1.56, of 1024 7.36 against 7.77; of 64 1.27 against
// 1.00 (step_shape).  Each warp evaluates the
// proposal network for 32 particles on the tensor cores (two 16-row tiles
// sharing the weight loads); lane 4g + q then moves particle g + 8q of the
// warp's 32.
template <bool First, int kBlock>
__global__ void __launch_bounds__(kBlock, 512 / kBlock) k_batch_step_learned(
    const BatchArgs a)
{
    pdl_wait();
    constexpr int kW = 4; // warps that take the sums
    constexpr int kLast = kBlock / 32 - 1;
    __shared__ __align__(16) uint32_t sp[kPackedWords];
    const uint32_t t = *a.step;
    const uint32_t nseg = t <= a.tmax ? a.active[t] : 0u;
    if (!First)
        load_packed(sp, a.packed);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int g = lane >> 2, q = lane & 3;
    __shared__ SegMeta metas[3];
    __shared__ SegSums<kW> sums[2];
    // a segment's particles: log-weight; previous weight and position
    __shared__ float s_lw[1024], s_wo[1024], s_x[1024], s_y[1024];
    // the next step's counter was last used by the previous step's launch
    if (blockIdx.x == 0 && threadIdx.x == 0)
        a.work[(t + 1) & 1u] = 0;
    if (wid == kLast) {
        seg_fetch(a, blockIdx.x, nseg, metas[0]);
        __pipeline_wait_prior(0);
    }
    __syncthreads();
    uint32_t slot = 0;
    for (uint32_t it = 0;; ++it) {
        const SegMeta &meta = metas[slot];
        slot = slot == 2 ? 0 : slot + 1;
        if (meta.count == 0)
            break;
        if (wid == kLast) { // the next segment
            uint32_t next = 0;
            if (lane == 0)
                next = gridDim.x + atomicAdd(a.work + (t & 1u), 1u);
            seg_fetch(
                a, __shfl_sync(0xFFFFFFFFu, next, 0), nseg, metas[slot]);
        }
        const BFilter F = meta.F; // in registers
        const BearingsConst &c = F.bc;
        const bool mon = !First && t == F.T;
        const int resampled = First ? 1 : meta.resampled;
        const bool gather = First ? false : (meta.gather != 0);
        const float Mprev = First ? 0.0f : meta.Mf;
        const float z = mon ? 0.0f : a.obs[F.obs_off + t];
        const uint32_t i00 = (meta.tile - F.tile0) * kLearnTile;
        bool written = false;
        for (uint32_t p = wid / kW; p < meta.count;
             p += kBlock / 128) {
            // slot of the segment: tile p, the lane's particle in it
            const uint32_t slot_i = p * kLearnTile + 32 * (wid % kW) + lane;
            const uint32_t i =
                i00 + p * kLearnTile + 32 * (wid % kW) + g + 8 * q;
            const bool mine = i < F.n;
            float wo = 0, x0 = 0, y0 = 0;
            float x = 0, y = 0, vx = 0, vy = 0, lw = 0;
            if (!First && mine) {
                uint32_t src[1] = {i};
                if (gather) {
                    const int32_t I[1] = {a.idx[F.off + i]};
                    batch_sources<1>(a, F, a.st[meta.f], I, src);
                }
                x = a.ax[F.off + src[0]];
                y = a.ay[F.off + src[0]];
                vx = a.avx[F.off + src[0]];
                vy = a.avy[F.off + src[0]];
                lw = resampled ? 0.0f : a.lw[F.off + i];
            }
            x0 = x;
            y0 = y;
            if (mon) {
                if (mine)
                    wo = resampled ? 1.0f : __expf(lw - Mprev);
            } else if (First) {
                if (mine) {
                    float e[4];
                    bearings_normals(t, F.seed, i, e);
                    bearings_prior(c, e, x, y, vx, vy);
                    lw = bearings_loglik(c, z, x, y);
                }
            } else {
                const float2 scz = a.obs_sc[F.obs_off + t];
                const float sz = scz.x, cz = scz.y;
                float fe[6];
                bearings_features(c, x, y, vx, vy, sz, cz, fe);
                uint32_t a0[4], b0[4];
                features_to_a2(fe, a0, b0);
                // one 16-row tile at a time keeps one tile's activations live
                float oa[4], ob[4];
#pragma unroll 1
                for (int h = 0; h < 2; ++h) {
                    uint32_t in[4];
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        in[r] = h ? b0[r] : a0[r];
                    float o[4];
                    mlp_forward_warp<false, true>(sp, in, o);
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        if (h)
                            ob[r] = o[r];
                        else
                            oa[r] = o[r];
                    }
                }
                float v[8];
                out_to_owner2(oa, ob, v);
                if (mine) {
                    const float lw_old = resampled ? 0.0f : lw - Mprev;
                    wo = resampled ? 1.0f : __expf(lw_old);
                    float e[4], fr[4], nu[4];
                    bearings_normals(t, F.seed, i, e);
                    float lq = 0;
#pragma unroll
                    for (int d = 0; d < 4; ++d) {
                        const float l = fminf(fmaxf(v[4 + d], c.lmin), c.lmax);
                        fr[d] = v[d] + __expf(0.5f * l) * e[d];
                        lq += 0.5f * (e[d] * e[d] - fr[d] * fr[d]) + 0.5f * l;
                    }
                    frame_to_axes(sz, cz, fr, nu); // the draw, bearing frame
                    bearings_step(c, nu, x, y, vx, vy);
                    lw = lw_old + bearings_loglik(c, z, x, y) + lq;
                }
            }
            if (!mon && mine) {
                const uint32_t gi = F.off + i;
                a.bx[gi] = x;
                a.by[gi] = y;
                a.bvx[gi] = vx;
                a.bvy[gi] = vy;
                a.lw[gi] = lw;
            }
            if (!written) { // the last segment's sums are taken
                __syncthreads();
                written = true;
            }
            s_lw[slot_i] = lw;
            s_wo[slot_i] = wo;
            s_x[slot_i] = x0;
            s_y[slot_i] = y0;
        }
        if (!written)
            __syncthreads();
        if (wid == kLast)
            __pipeline_wait_prior(0);
        __syncthreads();
        if (wid < kW) {
            float m = -INFINITY, s = 0, s2 = 0, sx = 0, sy = 0, sw = 0;
            for (uint32_t p = 0; p < meta.count; ++p) {
                const uint32_t slot_i = p * kLearnTile + 32 * wid + lane;
                if (i00 + p * kLearnTile + 32 * wid + g + 8 * q >= F.n)
                    continue;
                if (!First) {
                    const float wo = s_wo[slot_i];
                    sx += wo * s_x[slot_i];
                    sy += wo * s_y[slot_i];
                    sw += wo;
                }
                if (!mon)
                    lse_push(s_lw[slot_i], m, s, s2);
            }
            seg_record_warp(sums[it & 1], m, s, s2, sx, sy, sw);
            asm volatile("bar.sync 1, 128;" : : : "memory");
            if (static_cast<uint32_t>(wid) == it % kW)
                seg_finish<kW, First>(a, meta, t, mon, sums[it & 1]);
        }
    }
}

// ---------------------------------------------------------------- resampling
//
// The filters that resample at a step are resampled together by three
// kernels over the step's list of units: entry v of the list is unit k of
// filter f (its particles [k u, (k + 1) u) with u = F.rs_unit), and the units
// of a filter are consecutive entries, listed by the block that finished the
// filter's step (tile_finish).  A unit is one warp's work, and the passes are
// the single filter's over one warp range (qsum_range, count_range,
// assign_range), without a block barrier: a block per chunk of 4096 particles
// with block-wide scans took 34, 22 and 11 us a step at 512 filters, mostly
// barriers and, in filters below 4096 particles, idle warps; it is 37, 20
// and 15 us now with 6 million particles resampled in a step (early steps).
// Eight units a chunk took 10.62 ms for 100 steps, sixteen 11.21, four 11.57.
// The
// last unit of a filter to finish a pass (a ticket per filter, nothing
// waits) turns the units' totals into prefixes and records what the next
// pass needs.  Warps walk the list with a grid stride: the grids are fixed
// when a run is captured, and filters that do not resample cost nothing.

// one list entry, with its filter's sizes
struct RsUnit {
    uint32_t f, k;   // filter, unit of the filter
    uint32_t base;   // list entry of the filter's unit 0
    uint32_t nu;     // units of the filter
    uint32_t lo, hi; // particles of the unit
    Rs32Args r;      // the filter's arrays
};

__device__ __forceinline__ RsUnit rs_unit_at(const BatchArgs &a, uint32_t v)
{
    const uint2 e =
        __ldcg(a.rs_list + static_cast<size_t>(a.rpar) * a.rs_cap + v);
    const BFilter &F = a.flt[e.x];
    RsUnit c;
    c.f = e.x;
    c.k = e.y;
    c.base = v - e.y;
    c.nu = (F.n + F.rs_unit - 1) / F.rs_unit;
    c.lo = min(F.n, c.k * F.rs_unit);
    c.hi = min(F.n, c.lo + F.rs_unit);
    c.r = Rs32Args{};
    c.r.n = F.n;
    c.r.shift = F.shift;
    c.r.scheme = a.scheme;
    c.r.lw = a.lw + F.off;
    c.r.rep = a.rep + F.off;
    c.r.idx = a.idx + F.off;
    c.r.srcs = a.srcs + F.off;
    c.r.sc = a.st + e.x;
    return c;
}

// Whether the calling warp's unit is the last of its filter to get here
// (every lane gets the answer); its writes are ordered before.
__device__ __forceinline__ bool rs_last_unit(uint32_t *ticket, uint32_t nu)
{
    __threadfence();
    __syncwarp();
    int last = 0;
    if ((threadIdx.x & 31) == 0) {
        last = atomicAdd(ticket, 1u) == nu - 1 ? 1 : 0;
        if (last)
            *ticket = 0;
    }
    last = __shfl_sync(0xFFFFFFFFu, last, 0);
    if (last)
        __threadfence();
    return last != 0;
}

// v[0 .. nu) turned into exclusive prefixes by one warp; the total in every
// lane.  A filter has at most kMaxRsUnits units.
constexpr uint32_t kMaxRsUnits = 256;

__device__ __forceinline__ uint64_t rs_prefix(uint64_t *v, uint32_t nu)
{
    constexpr uint32_t kK = kMaxRsUnits / 32;
    const uint32_t lane = threadIdx.x & 31;
    uint64_t x[kK];
    uint64_t s = 0;
#pragma unroll
    for (uint32_t k = 0; k < kK; ++k) {
        const uint32_t j = lane * kK + k;
        x[k] = j < nu ? __ldcg(v + j) : 0ull;
        s += x[k];
    }
    const uint64_t incl = warp_inclusive_scan(s, OpAdd());
    uint64_t run = incl - s;
#pragma unroll
    for (uint32_t k = 0; k < kK; ++k) {
        const uint32_t j = lane * kK + k;
        if (j < nu)
            v[j] = run;
        run += x[k];
    }
    return __shfl_sync(0xFFFFFFFFu, incl, 31);
}

// warps of the grid and the calling one's number
#define RS_UNITS(a, v, count)                                                 \
    const uint32_t count = __ldcg((a).rs_count + (a).rpar);                   \
    for (uint32_t v = blockIdx.x * (kPfBlock / 32) + (threadIdx.x >> 5);      \
         v < count; v += gridDim.x * (kPfBlock / 32))

// pass 1: fixed-point total of each unit; the filter's last one sets the
// filter's counting constants.  Block 0 also advances the step counter
// (every step kernel block has read it) and empties the next step's list.
__global__ void __launch_bounds__(kPfBlock, 4) k_brs_qsum(const BatchArgs a)
{
    pdl_wait();
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        atomicAdd(a.step, 1u);
        a.rs_count[a.rpar ^ 1u] = 0;
    }
    RS_UNITS(a, v, count)
    {
        const RsUnit c = rs_unit_at(a, v);
        PfScalars &S = *c.r.sc;
        const uint64_t q = qsum_range(c.r, c.lo, c.hi, S.Mf);
        if ((threadIdx.x & 31) == 0)
            a.rs_q[v] = q;
        if (rs_last_unit(&S.done3, c.nu)) {
            const uint64_t Q = rs_prefix(a.rs_q + c.base, c.nu);
            uint32_t err = 0;
            cdf_constants(S, Q, c.r.n, a.scheme == VSMC_CUDA_SYSTEMATIC, err);
            if ((threadIdx.x & 31) == 0 && err)
                atomicOr(&S.err, err);
        }
    }
}

// pass 2: replication counts from the fixed-point CDF (count_range).  The
// filter's last unit records the resample: the empty count, the gather flag
// and the engine past the words the scheme consumed.  A zero total counts
// nothing: no resample.
template <bool Sys>
__global__ void __launch_bounds__(kPfBlock, 3) k_brs_count(const BatchArgs a)
{
    pdl_wait();
    __shared__ uint4 rows[Sys ? 1 : kPfBlock / 32][Sys ? 1 : kStratRow];
    RS_UNITS(a, v, count)
    {
        const RsUnit c = rs_unit_at(a, v);
        PfScalars &S = *c.r.sc;
        const CdfRcp p = load_cdf_rcp(S, c.r.n);
        uint32_t empties = 0, copies = 0;
        if (p.Q != 0) {
            EnginePos e = {};
            if (!Sys)
                e = engine_pos(S);
            uint4 *row = rows[Sys ? 0 : threadIdx.x >> 5];
            const uint64_t carry = __ldcg(a.rs_q + v);
            if (p.s != 0)
                count_range<Sys, true>(c.r, p, e, row, c.lo, c.hi, carry,
                    empties, copies);
            else
                count_range<Sys, false>(c.r, p, e, row, c.lo, c.hi, carry,
                    empties, copies);
            empties = __reduce_add_sync(0xFFFFFFFFu, empties);
            copies = __reduce_add_sync(0xFFFFFFFFu, copies);
        }
        if ((threadIdx.x & 31) == 0)
            a.rs_ec[v] = (static_cast<uint64_t>(copies) << 32) | empties;
        if (rs_last_unit(&S.done2, c.nu)) {
            const uint64_t ec = rs_prefix(a.rs_ec + c.base, c.nu);
            if ((threadIdx.x & 31) == 0) {
                S.nempty = static_cast<uint32_t>(ec);
                if (p.Q != 0) {
                    S.gather = 1;
                    if (static_cast<uint32_t>(ec >> 32) != c.r.n)
                        atomicOr(&S.err, DEV_ERR_INTERNAL);
                    scheme_words(c.r, S);
                }
            }
        }
    }
}

// pass 3: slot assignment (assign_range)
__global__ void __launch_bounds__(kPfBlock, 4) k_brs_assign(const BatchArgs a)
{
    pdl_wait();
    __shared__ __align__(16) uint32_t shm[kPfBlock / 32][kRunChunk];
    RS_UNITS(a, v, count)
    {
        const RsUnit c = rs_unit_at(a, v);
        const PfScalars &S = *c.r.sc;
        if (S.Q == 0)
            continue;
        const uint64_t ec = __ldcg(a.rs_ec + v);
        float macc[kMaxMonitorDim];
        assign_range<false>(c.r, c.lo, c.hi, static_cast<uint32_t>(ec >> 32),
            static_cast<uint32_t>(ec), S.nempty, shm[threadIdx.x >> 5], macc);
    }
}

// the run's observations in FP32, as the step kernels use them, and for
// the bearings kinds (sc != null) the sine and cosine of each FP32 bearing
__global__ void k_obs_f32(
    const double *obs, float *out, float2 *sc, uint32_t count)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count;
         i += gridDim.x * blockDim.x) {
        const float z = static_cast<float>(obs[i]);
        out[i] = z;
        if (sc)
            sc[i] = make_float2(sinf(z), cosf(z));
    }
}

__global__ void k_batch_reset(PfScalars *st, const BFilter *flt, uint32_t nf,
    uint32_t *step, uint32_t *rs_count)
{
    const uint32_t f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f == 0) {
        *step = 0;
        // list counts, then the step kernel's tile counters
        rs_count[0] = rs_count[1] = rs_count[2] = rs_count[3] = 0;
    }
    if (f >= nf)
        return;
    PfScalars z = {};
    z.resampled = 1;
    z.rindex = 4;
    z.rkey[0] = 0;
    z.rkey[1] = flt[f].seed;
    z.rctr[2] = 1;
    st[f] = z;
}

// each filter's observations from its own model and seed (one thread each)
__global__ void k_batch_simulate(const vsmc_cuda_cv_model *models,
    const uint32_t *seeds, const uint32_t *T, const uint32_t *obs_off,
    uint32_t nf, double *truth, double *obs)
{
    const uint32_t f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nf)
        return;
    const vsmc_cuda_cv_model m = models[f];
    cv_simulate_seq(seeds[f], T[f], m.dt, m.sigma_a, m.obs_scale, m.nu,
        m.sd_pos0, m.sd_vel0, truth ? truth + 4 * obs_off[f] : nullptr,
        obs + 2 * obs_off[f]);
}

// Bearings simulation of one filter on one thread: the FP64 draws of
// vsmc_cuda_bearings_simulate (CounterEngine(seed), NormalDistribution pairs,
// one NormalDistribution(0, sigma_z) for the bearing noise).
__global__ void k_batch_simulate_bearings(
    const vsmc_cuda_bearings_model *models, const uint32_t *seeds,
    const uint32_t *T, const uint32_t *obs_off, uint32_t nf, double *truth,
    double *obs)
{
    const uint32_t f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nf)
        return;
    bearings_simulate_seq(seeds[f], T[f], models[f],
        truth ? truth + 4 * obs_off[f] : nullptr, obs + obs_off[f]);
}

constexpr uint32_t kRsMinChunk = 4 * kPfTile; // resampling chunk: 4096 or more
constexpr uint32_t kMaxRsChunks = 32;          // chunks of one filter, at most
constexpr uint32_t kRsUnits = 8;               // warps' units of a chunk
static_assert(kMaxRsChunks * kRsUnits <= kMaxRsUnits, "units of a filter");
constexpr int kRsKernels = 3;
// the scan schedules the autotuner times: the smallest chunk of a filter
constexpr uint32_t kRsSchedules[] = {4096, 8192, 16384, 32768};
constexpr int kNumSchedules = 4;

// A filter's resampling chunk: min_chunk, doubled until the filter has at
// most kMaxRsChunks chunks.  Larger chunks mean fewer list entries (and
// fewer partial records to sum) but a longer last wave.
inline uint32_t rs_chunk_for(uint32_t n, uint32_t min_chunk)
{
    uint32_t c = min_chunk;
    while ((n + c - 1) / c > kMaxRsChunks)
        c *= 2;
    return c;
}

struct Shape {
    int ppt, block;
};
constexpr Shape kShapes[] = {
    {1, 128}, {2, 128}, {4, 128}, {1, 256}, {2, 256}, {4, 256}};
constexpr int kNumShapes = 6;

template <int kBlock, int kPPT, int Kind>
static cudaError_t launch_step_k(bool first, int grid, const BatchArgs &a,
    cudaStream_t st)
{
    if (first)
        launch_after(k_batch_step<kBlock, kPPT, true, Kind>, grid, kBlock, 0,
            st, a);
    else
        launch_after(k_batch_step<kBlock, kPPT, false, Kind>, grid, kBlock, 0,
            st, a);
    return cudaGetLastError();
}

template <int kBlock, int kPPT>
static cudaError_t launch_step_t(int kind, bool first, int grid,
    const BatchArgs &a, cudaStream_t st)
{
    return kind == kKindCv
        ? launch_step_k<kBlock, kPPT, kKindCv>(first, grid, a, st)
        : launch_step_k<kBlock, kPPT, kKindBearings>(first, grid, a, st);
}

template <int kBlock>
static cudaError_t launch_learned(
    bool first, int grid, const BatchArgs &a, cudaStream_t st)
{
    if (first)
        launch_after(k_batch_step_learned<true, kBlock>, grid, kBlock, 0, st,
            a);
    else
        launch_after(k_batch_step_learned<false, kBlock>, grid, kBlock, 0, st,
            a);
    return cudaGetLastError();
}

static cudaError_t launch_step(int kind, Shape s, bool first, int grid,
    const BatchArgs &a, cudaStream_t st)
{
    if (kind == kKindLearned)
        return s.block == 128 ? launch_learned<128>(first, grid, a, st)
                              : launch_learned<256>(first, grid, a, st);
    if (s.block == 128) {
        if (s.ppt == 1)
            return launch_step_t<128, 1>(kind, first, grid, a, st);
        if (s.ppt == 2)
            return launch_step_t<128, 2>(kind, first, grid, a, st);
        return launch_step_t<128, 4>(kind, first, grid, a, st);
    }
    if (s.ppt == 1)
        return launch_step_t<256, 1>(kind, first, grid, a, st);
    if (s.ppt == 2)
        return launch_step_t<256, 2>(kind, first, grid, a, st);
    return launch_step_t<256, 4>(kind, first, grid, a, st);
}

template <typename K>
static int occupancy_of(K kernel, int block)
{
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, block, 0) !=
            cudaSuccess ||
        occ < 1)
        occ = 2;
    return occ;
}

template <int kBlock, int kPPT>
static int occupancy_t(int kind)
{
    return kind == kKindCv
        ? occupancy_of(k_batch_step<kBlock, kPPT, false, kKindCv>, kBlock)
        : occupancy_of(
              k_batch_step<kBlock, kPPT, false, kKindBearings>, kBlock);
}

static int occupancy(int kind, Shape s)
{
    if (kind == kKindLearned)
        return s.block == 128
            ? occupancy_of(k_batch_step_learned<false, 128>, 128)
            : occupancy_of(k_batch_step_learned<false, 256>, 256);
    if (s.block == 128)
        return s.ppt == 1 ? occupancy_t<128, 1>(kind)
                          : (s.ppt == 2 ? occupancy_t<128, 2>(kind)
                                        : occupancy_t<128, 4>(kind));
    return s.ppt == 1 ? occupancy_t<256, 1>(kind)
                      : (s.ppt == 2 ? occupancy_t<256, 2>(kind)
                                    : occupancy_t<256, 4>(kind));
}

} // namespace vsmc_cuda

struct vsmc_cuda_batch {
    int kind = kKindCv;
    const uint32_t *packed = nullptr; // learned kind: proposal network
    std::vector<vsmc_cuda_bearings_model> bmodels;
    uint32_t nf = 0;
    uint32_t tmax = 0;
    int scheme = VSMC_CUDA_STRATIFIED;
    double threshold = 0.5;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    Shape shape = {4, 256};
    // caller order
    std::vector<uint32_t> n, T, seeds;
    std::vector<vsmc_cuda_cv_model> models;
    std::vector<uint32_t> obs_off; // prefix sums of T (caller order)
    size_t total_T = 0;
    // internal order: horizon descending
    std::vector<uint32_t> order;     // internal -> caller
    uint32_t rs_cap = 0;            // resampling chunks of all filters
    int rs_grid[kRsKernels] = {};   // persistent grids of the passes
    std::vector<BFilter> flt;        // internal order
    std::vector<uint32_t> active;
    std::vector<uint4> segs;
    size_t total_particles = 0; // with padding
    size_t max_tiles = 0;
    // device
    BFilter *d_flt = nullptr;
    PfScalars *d_st = nullptr;
    uint4 *d_segs = nullptr;
    uint32_t *d_active = nullptr, *d_step = nullptr;
    uint2 *d_rs_list = nullptr;
    uint32_t *d_rs_count = nullptr;
    uint64_t *d_rs_q = nullptr, *d_rs_ec = nullptr;
    float *d_state[2] = {nullptr, nullptr};
    float *d_lw = nullptr;
    int32_t *d_rep = nullptr, *d_idx = nullptr;
    uint32_t *d_srcs = nullptr;
    TileRecord *d_part = nullptr;
    float *d_obsf = nullptr; // the run's observations in FP32
    float2 *d_obs_sc = nullptr; // bearings kinds: sin, cos of each bearing
    double *d_obs = nullptr;
    double *d_mean = nullptr, *d_ess = nullptr, *d_logz = nullptr;
    int *d_res = nullptr;
    // run graph (for one observation pointer, shape and schedule)
    cudaGraphExec_t graph = nullptr;
    const double *graph_obs = nullptr;
    Shape graph_shape = {0, 0};
    uint32_t graph_chunk = 0;
    // scan schedule: the smallest resampling chunk of a filter (the list and
    // its buffers are sized for kRsMinChunk, the smallest allowed)
    uint32_t rs_min_chunk = 0;
};

namespace vsmc_cuda
{

template <typename T>
static int balloc(T **p, size_t count)
{
    void *q = nullptr;
    VSMC_CUDA_TRY(device_malloc(&q, sizeof(T) * (count ? count : 1)));
    *p = static_cast<T *>(q);
    return VSMC_CUDA_OK;
}

static void batch_free(vsmc_cuda_batch *b)
{
    if (b->graph)
        cudaGraphExecDestroy(b->graph);
    void *ptrs[] = {b->d_flt, b->d_st, b->d_segs, b->d_active,
        b->d_step, b->d_rs_list, b->d_rs_count, b->d_rs_q, b->d_rs_ec,
        b->d_state[0], b->d_state[1], b->d_lw,
        b->d_rep, b->d_idx, b->d_srcs, b->d_part, b->d_obs, b->d_obsf, b->d_obs_sc,
        b->d_mean, b->d_ess, b->d_logz, b->d_res};
    for (void *p : ptrs)
        if (p)
            cudaFree(p);
    if (b->own_stream && b->stream)
        cudaStreamDestroy(b->stream);
}

// tile tables for a shape (host + device)
static int batch_layout(vsmc_cuda_batch *b, Shape s)
{
    const uint32_t tile = b->kind == kKindLearned
        ? kLearnTile
        : static_cast<uint32_t>(s.ppt * s.block);
    const uint32_t most =
        b->kind == kKindLearned ? kLearnSeg : seg_tiles(tile);
    // a segment ends at its filter's last tile and at every `most` tiles
    b->segs.clear();
    std::vector<uint32_t> seg_end(b->nf); // segments up to each filter's
    uint32_t tiles = 0;
    for (uint32_t k = 0; k < b->nf; ++k) {
        BFilter &F = b->flt[k];
        F.tile0 = tiles;
        F.ntiles = (F.n + tile - 1) / tile;
        tiles += F.ntiles;
        for (uint32_t j = F.tile0; j < tiles;) {
            const uint32_t e = std::min(tiles, (j / most + 1) * most);
            b->segs.push_back(make_uint4(j, e - j, k, 0));
            j = e;
        }
        seg_end[k] = static_cast<uint32_t>(b->segs.size());
    }
    if (tiles > b->max_tiles)
        return VSMC_CUDA_ERR_INTERNAL;
    // filters are sorted by T descending: those with T >= t are a prefix
    b->active.assign(b->tmax + 1, 0);
    uint32_t k = b->nf;
    for (uint32_t t = 0; t <= b->tmax; ++t) {
        while (k > 0 && b->flt[k - 1].T < t)
            --k;
        b->active[t] = k == 0 ? 0 : seg_end[k - 1];
    }
    cudaStream_t st = b->stream;
    VSMC_CUDA_TRY(cudaMemcpyAsync(b->d_flt, b->flt.data(),
        sizeof(BFilter) * b->nf, cudaMemcpyHostToDevice, st));
    VSMC_CUDA_TRY(cudaMemcpyAsync(b->d_segs, b->segs.data(),
        sizeof(uint4) * b->segs.size(), cudaMemcpyHostToDevice, st));
    VSMC_CUDA_TRY(cudaMemcpyAsync(b->d_active, b->active.data(),
        sizeof(uint32_t) * b->active.size(), cudaMemcpyHostToDevice, st));
    VSMC_CUDA_TRY(cudaStreamSynchronize(st));
    b->shape = s;
    return VSMC_CUDA_OK;
}

// The step kernel's shape: the tiles', and for learned filters the block that
// suits their number of segments (see k_batch_step_learned).
static Shape step_shape(const vsmc_cuda_batch *b)
{
    Shape s = b->shape;
    if (b->kind == kKindLearned)
        s.block = b->segs.size() <= 2 * static_cast<size_t>(num_sms()) ? 256
                                                                       : 128;
    return s;
}

static BatchArgs batch_args(vsmc_cuda_batch *b, const double *obs, int cur)
{
    BatchArgs a = {};
    const size_t ld = b->total_particles;
    const float *A = b->d_state[cur];
    float *B = b->d_state[1 - cur];
    a.flt = b->d_flt;
    a.st = b->d_st;
    a.segs = b->d_segs;
    a.active = b->d_active;
    a.ax = A;
    a.ay = A + ld;
    a.avx = A + 2 * ld;
    a.avy = A + 3 * ld;
    a.bx = B;
    a.by = B + ld;
    a.bvx = B + 2 * ld;
    a.bvy = B + 3 * ld;
    a.lw = b->d_lw;
    a.rep = b->d_rep;
    a.idx = b->d_idx;
    a.srcs = b->d_srcs;
    a.part = b->d_part;
    a.obs = b->d_obsf;
    a.obs_sc = b->d_obs_sc;
    a.h_mean = b->d_mean;
    a.h_ess = b->d_ess;
    a.h_logz = b->d_logz;
    a.h_res = b->d_res;
    a.step = b->d_step;
    a.rs_list = b->d_rs_list;
    a.rs_count = b->d_rs_count;
    a.work = b->d_rs_count + 2;
    a.rs_q = b->d_rs_q;
    a.rs_ec = b->d_rs_ec;
    a.rs_cap = b->rs_cap;
    a.rpar = static_cast<uint32_t>(cur); // step parity, as the state buffers
    a.packed = b->packed;
    a.nfilters = b->nf;
    a.tmax = b->tmax;
    a.scheme = b->scheme;
    a.threshold = b->threshold;
    return a;
}

// enqueue a whole run (reset + steps 0..nsteps-1) on the batch's stream;
// grid = the step kernel's persistent grid for the current shape
static int enqueue_run(
    vsmc_cuda_batch *b, const double *obs, int nsteps, int grid)
{
    cudaStream_t st = b->stream;
    const uint32_t nobs = static_cast<uint32_t>(
        (b->kind == kKindCv ? 2 : 1) * b->total_T);
    k_obs_f32<<<grid_for(nobs, 256, 1, 4), 256, 0, st>>>(obs, b->d_obsf,
        b->kind == kKindCv ? nullptr : b->d_obs_sc, nobs);
    VSMC_CUDA_CHECK_LAUNCH();
    k_batch_reset<<<(b->nf + 255) / 256, 256, 0, st>>>(
        b->d_st, b->d_flt, b->nf, b->d_step, b->d_rs_count);
    VSMC_CUDA_CHECK_LAUNCH();
    for (int t = 0; t < nsteps; ++t) {
        const BatchArgs a = batch_args(b, obs, t & 1);
        VSMC_CUDA_TRY(launch_step(b->kind, step_shape(b), t == 0, grid, a, st));
        // the filters that resample, in the units the step listed
        const dim3 blk(kPfBlock);
        launch_after(k_brs_qsum, b->rs_grid[0], blk, 0, st, a);
        if (a.scheme == VSMC_CUDA_SYSTEMATIC)
            launch_after(k_brs_count<true>, b->rs_grid[1], blk, 0, st, a);
        else
            launch_after(k_brs_count<false>, b->rs_grid[1], blk, 0, st, a);
        launch_after(k_brs_assign, b->rs_grid[2], blk, 0, st, a);
        VSMC_CUDA_CHECK_LAUNCH();
    }
    return VSMC_CUDA_OK;
}

static int check_errors(vsmc_cuda_batch *b)
{
    std::vector<PfScalars> st(b->nf);
    VSMC_CUDA_TRY(cudaMemcpyAsync(st.data(), b->d_st,
        sizeof(PfScalars) * b->nf, cudaMemcpyDeviceToHost, b->stream));
    VSMC_CUDA_TRY(cudaStreamSynchronize(b->stream));
    uint32_t err = 0;
    for (const PfScalars &s : st)
        err |= s.err;
    if (err & DEV_ERR_NONFINITE)
        return VSMC_CUDA_ERR_NONFINITE;
    if (err)
        return VSMC_CUDA_ERR_INTERNAL;
    return VSMC_CUDA_OK;
}

} // namespace vsmc_cuda

extern "C" {

} // extern "C"

namespace vsmc_cuda
{

// Shared constructor of the three kinds: cv (position model) or bm
// (bearings model) per filter; packed: the proposal network (learned kind).
static int batch_create(vsmc_cuda_batch **out, int kind, size_t nfilters,
    const uint32_t *n, const uint32_t *T, const vsmc_cuda_cv_model *cv,
    const vsmc_cuda_bearings_model *bm, const uint32_t *seeds,
    const uint32_t *packed, int scheme, double threshold, void *stream)
{
    if (out == nullptr || n == nullptr || T == nullptr || seeds == nullptr ||
        std::isnan(threshold) ||
        (scheme != VSMC_CUDA_STRATIFIED && scheme != VSMC_CUDA_SYSTEMATIC))
        return VSMC_CUDA_ERR_ARG;
    *out = nullptr;
    if (nfilters < 1 || nfilters > (size_t(1) << 24))
        return VSMC_CUDA_ERR_SIZE;
    const uint32_t min_tile = kind == kKindLearned ? kLearnTile : 128u;
    size_t total = 0, totalT = 0, tiles = 0;
    uint32_t tmax = 0;
    for (size_t f = 0; f < nfilters; ++f) {
        if (kind == kKindCv ? !valid_cv_model(&cv[f])
                            : !valid_bearings_model(&bm[f]))
            return VSMC_CUDA_ERR_ARG;
        if (n[f] < 2 || n[f] > (1u << 30) || T[f] < 1 || T[f] > (1u << 24))
            return VSMC_CUDA_ERR_SIZE;
        total += (static_cast<size_t>(n[f]) + 3) / 4 * 4;
        totalT += T[f];
        tiles += (n[f] + min_tile - 1) / min_tile; // the smallest tile
        tmax = std::max(tmax, T[f]);
    }
    if (total >= (size_t(1) << 31) || totalT >= (size_t(1) << 31))
        return VSMC_CUDA_ERR_SIZE;
    vsmc_cuda_batch *b = new (std::nothrow) vsmc_cuda_batch;
    if (b == nullptr)
        return VSMC_CUDA_ERR_ALLOC;
    b->kind = kind;
    b->packed = packed;
    b->nf = static_cast<uint32_t>(nfilters);
    b->tmax = tmax;
    b->scheme = scheme;
    b->threshold = threshold;
    b->n.assign(n, n + nfilters);
    b->T.assign(T, T + nfilters);
    b->seeds.assign(seeds, seeds + nfilters);
    if (kind == kKindCv)
        b->models.assign(cv, cv + nfilters);
    else
        b->bmodels.assign(bm, bm + nfilters);
    b->total_T = totalT;
    b->total_particles = total;
    b->max_tiles = tiles;
    b->obs_off.resize(nfilters);
    size_t acc = 0;
    for (size_t f = 0; f < nfilters; ++f) {
        b->obs_off[f] = static_cast<uint32_t>(acc);
        acc += T[f];
    }
    b->order.resize(nfilters);
    for (uint32_t f = 0; f < nfilters; ++f)
        b->order[f] = f;
    std::stable_sort(b->order.begin(), b->order.end(),
        [&](uint32_t x, uint32_t y) { return T[x] > T[y]; });
    b->flt.resize(nfilters);
    b->rs_min_chunk = kRsMinChunk;
    size_t off = 0;
    for (uint32_t k = 0; k < nfilters; ++k) {
        const uint32_t f = b->order[k];
        BFilter &F = b->flt[k];
        F = BFilter{};
        F.n = n[f];
        F.off = static_cast<uint32_t>(off);
        off += (static_cast<size_t>(n[f]) + 3) / 4 * 4;
        F.T = T[f];
        F.obs_off = b->obs_off[f];
        F.hist_off = b->obs_off[f];
        F.seed = seeds[f];
        int lg = 0;
        while ((size_t(1) << lg) < n[f])
            ++lg;
        F.shift = static_cast<uint32_t>(63 - lg);
        F.rs_unit = rs_chunk_for(F.n, kRsMinChunk) / kRsUnits;
        b->rs_cap += (F.n + F.rs_unit - 1) / F.rs_unit;
        if (kind == kKindCv)
            F.c = make_cv_const<float>(cv[f]);
        else
            F.bc = make_bearings_const(bm[f]);
    }
    // the resampling passes walk the step's list with one full wave of
    // blocks each
    {
        const int sms = num_sms();
        const int occ[kRsKernels] = {occupancy_of(k_brs_qsum, kPfBlock),
            std::min(occupancy_of(k_brs_count<true>, kPfBlock),
                occupancy_of(k_brs_count<false>, kPfBlock)),
            occupancy_of(k_brs_assign, kPfBlock)};
        for (int k = 0; k < kRsKernels; ++k)
            b->rs_grid[k] = static_cast<int>(std::min<size_t>(
                static_cast<size_t>(sms) * occ[k],
                (b->rs_cap + kRsUnits - 1) / kRsUnits));
    }

    b->stream = as_stream(stream);
    if (b->stream == nullptr) {
        if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) !=
            cudaSuccess) {
            delete b;
            return VSMC_CUDA_ERR_CUDA;
        }
        b->own_stream = true;
    }
    int rc = VSMC_CUDA_OK;
#define B_TRY(x)                                                              \
    do {                                                                      \
        rc = (x);                                                             \
        if (rc != VSMC_CUDA_OK) {                                             \
            batch_free(b);                                                    \
            delete b;                                                         \
            return rc;                                                        \
        }                                                                     \
    } while (0)
    B_TRY(balloc(&b->d_flt, nfilters));
    B_TRY(balloc(&b->d_st, nfilters));
    B_TRY(balloc(&b->d_segs, tiles));
    B_TRY(balloc(&b->d_active, tmax + 1));
    B_TRY(balloc(&b->d_rs_list, 2 * static_cast<size_t>(b->rs_cap)));
    B_TRY(balloc(&b->d_rs_count, 4));
    B_TRY(balloc(&b->d_rs_q, b->rs_cap));
    B_TRY(balloc(&b->d_rs_ec, b->rs_cap));
    B_TRY(balloc(&b->d_step, 1));
    B_TRY(balloc(&b->d_state[0], 4 * total));
    B_TRY(balloc(&b->d_state[1], 4 * total));
    B_TRY(balloc(&b->d_lw, total));
    B_TRY(balloc(&b->d_rep, total));
    B_TRY(balloc(&b->d_idx, total));
    B_TRY(balloc(&b->d_srcs, total));
    B_TRY(balloc(&b->d_part, tiles));
    B_TRY(balloc(&b->d_obs, 2 * totalT));
    B_TRY(balloc(&b->d_obsf, 2 * totalT));
    if (kind != kKindCv)
        B_TRY(balloc(&b->d_obs_sc, totalT));
    B_TRY(balloc(&b->d_mean, 2 * totalT));
    B_TRY(balloc(&b->d_ess, totalT));
    B_TRY(balloc(&b->d_logz, totalT));
    B_TRY(balloc(&b->d_res, totalT));
    if (cudaMemsetAsync(b->d_mean, 0, sizeof(double) * 2 * totalT,
            b->stream) != cudaSuccess)
        B_TRY(VSMC_CUDA_ERR_CUDA);
    B_TRY(batch_layout(b, b->shape));
#undef B_TRY
    *out = b;
    return VSMC_CUDA_OK;
}

} // namespace vsmc_cuda

extern "C" {

int vsmc_cuda_batch_create(vsmc_cuda_batch **out, size_t nfilters,
    const uint32_t *n, const uint32_t *T, const vsmc_cuda_cv_model *models,
    const uint32_t *seeds, int scheme, double threshold, void *stream)
{
    if (models == nullptr)
        return VSMC_CUDA_ERR_ARG;
    return batch_create(out, kKindCv, nfilters, n, T, models, nullptr, seeds,
        nullptr, scheme, threshold, stream);
}

int vsmc_cuda_batch_create_bearings(vsmc_cuda_batch **out, size_t nfilters,
    const uint32_t *n, const uint32_t *T,
    const vsmc_cuda_bearings_model *models, const uint32_t *seeds,
    const uint32_t *packed, int scheme, double threshold, void *stream)
{
    if (models == nullptr)
        return VSMC_CUDA_ERR_ARG;
    return batch_create(out, packed ? kKindLearned : kKindBearings, nfilters,
        n, T, nullptr, models, seeds, packed, scheme, threshold, stream);
}

int vsmc_cuda_batch_destroy(vsmc_cuda_batch *b)
{
    if (b == nullptr)
        return VSMC_CUDA_OK;
    cudaStreamSynchronize(b->stream);
    batch_free(b);
    delete b;
    return VSMC_CUDA_OK;
}

int vsmc_cuda_batch_stream(vsmc_cuda_batch *b, void **stream)
{
    if (b == nullptr || stream == nullptr)
        return VSMC_CUDA_ERR_ARG;
    *stream = b->stream;
    return VSMC_CUDA_OK;
}

int vsmc_cuda_batch_simulate(vsmc_cuda_batch *b, double *truth_dev,
    double *obs_dev)
{
    if (b == nullptr || obs_dev == nullptr)
        return VSMC_CUDA_ERR_ARG;
    uint32_t *dseed = nullptr, *dT = nullptr, *doff = nullptr;
    cudaStream_t st = b->stream;
    Scratch scratch(st);
    void *dm = b->kind == kKindCv
        ? static_cast<void *>(scratch.get<vsmc_cuda_cv_model>(b->nf))
        : static_cast<void *>(scratch.get<vsmc_cuda_bearings_model>(b->nf));
    dseed = scratch.get<uint32_t>(b->nf);
    dT = scratch.get<uint32_t>(b->nf);
    doff = scratch.get<uint32_t>(b->nf);
    if (!dm || !dseed || !dT || !doff)
        return VSMC_CUDA_ERR_ALLOC;
    if (b->kind == kKindCv)
        VSMC_CUDA_TRY(cudaMemcpyAsync(dm, b->models.data(),
            sizeof(vsmc_cuda_cv_model) * b->nf, cudaMemcpyHostToDevice, st));
    else
        VSMC_CUDA_TRY(cudaMemcpyAsync(dm, b->bmodels.data(),
            sizeof(vsmc_cuda_bearings_model) * b->nf, cudaMemcpyHostToDevice,
            st));
    VSMC_CUDA_TRY(cudaMemcpyAsync(dseed, b->seeds.data(),
        sizeof(uint32_t) * b->nf, cudaMemcpyHostToDevice, st));
    VSMC_CUDA_TRY(cudaMemcpyAsync(dT, b->T.data(), sizeof(uint32_t) * b->nf,
        cudaMemcpyHostToDevice, st));
    VSMC_CUDA_TRY(cudaMemcpyAsync(doff, b->obs_off.data(),
        sizeof(uint32_t) * b->nf, cudaMemcpyHostToDevice, st));
    if (b->kind == kKindCv)
        k_batch_simulate<<<(b->nf + 63) / 64, 64, 0, st>>>(
            static_cast<const vsmc_cuda_cv_model *>(dm), dseed, dT, doff,
            b->nf, truth_dev, obs_dev);
    else
        k_batch_simulate_bearings<<<(b->nf + 63) / 64, 64, 0, st>>>(
            static_cast<const vsmc_cuda_bearings_model *>(dm), dseed, dT,
            doff, b->nf, truth_dev, obs_dev);
    VSMC_CUDA_CHECK_LAUNCH();
    VSMC_CUDA_TRY(cudaStreamSynchronize(st));
    return VSMC_CUDA_OK;
}

int vsmc_cuda_batch_run_device(vsmc_cuda_batch *b, const double *obs_dev)
{
    if (b == nullptr || obs_dev == nullptr)
        return VSMC_CUDA_ERR_ARG;
    const int nsteps = static_cast<int>(b->tmax) + 1;
    if (b->graph == nullptr || b->graph_obs != obs_dev ||
        b->graph_shape.ppt != b->shape.ppt ||
        b->graph_shape.block != b->shape.block ||
        b->graph_chunk != b->rs_min_chunk) {
        if (b->graph) {
            cudaGraphExecDestroy(b->graph);
            b->graph = nullptr;
        }
        const int grid = num_sms() * occupancy(b->kind, step_shape(b));
        VSMC_CUDA_TRY(cudaStreamBeginCapture(
            b->stream, cudaStreamCaptureModeThreadLocal));
        const int rc = enqueue_run(b, obs_dev, nsteps, grid);
        cudaGraph_t g = nullptr;
        const cudaError_t e = cudaStreamEndCapture(b->stream, &g);
        if (rc != VSMC_CUDA_OK) {
            if (g)
                cudaGraphDestroy(g);
            return rc;
        }
        VSMC_CUDA_TRY(e);
        const cudaError_t ei = cudaGraphInstantiate(&b->graph, g, 0);
        cudaGraphDestroy(g);
        VSMC_CUDA_TRY(ei);
        b->graph_obs = obs_dev;
        b->graph_shape = b->shape;
        b->graph_chunk = b->rs_min_chunk;
    }
    VSMC_CUDA_TRY(cudaGraphLaunch(b->graph, b->stream));
    return VSMC_CUDA_OK;
}

int vsmc_cuda_batch_history(vsmc_cuda_batch *b, double *mean_host,
    double *ess_host, int *resampled_host, double *logz_host)
{
    if (b == nullptr)
        return VSMC_CUDA_ERR_ARG;
    const int rc = check_errors(b);
    if (rc != VSMC_CUDA_OK)
        return rc;
    cudaStream_t st = b->stream;
    const size_t TT = b->total_T;
    if (mean_host)
        VSMC_CUDA_TRY(cudaMemcpyAsync(mean_host, b->d_mean,
            sizeof(double) * 2 * TT, cudaMemcpyDeviceToHost, st));
    if (ess_host)
        VSMC_CUDA_TRY(cudaMemcpyAsync(ess_host, b->d_ess, sizeof(double) * TT,
            cudaMemcpyDeviceToHost, st));
    if (resampled_host)
        VSMC_CUDA_TRY(cudaMemcpyAsync(resampled_host, b->d_res,
            sizeof(int) * TT, cudaMemcpyDeviceToHost, st));
    if (logz_host)
        VSMC_CUDA_TRY(cudaMemcpyAsync(logz_host, b->d_logz,
            sizeof(double) * TT, cudaMemcpyDeviceToHost, st));
    VSMC_CUDA_TRY(cudaStreamSynchronize(st));
    return VSMC_CUDA_OK;
}

int vsmc_cuda_batch_run(vsmc_cuda_batch *b, const double *obs_host,
    double *mean_host, double *ess_host, int *resampled_host,
    double *logz_host)
{
    if (b == nullptr || obs_host == nullptr)
        return VSMC_CUDA_ERR_ARG;
    const size_t obs_dim = b->kind == kKindCv ? 2 : 1;
    VSMC_CUDA_TRY(cudaMemcpyAsync(b->d_obs, obs_host,
        sizeof(double) * obs_dim * b->total_T, cudaMemcpyHostToDevice,
        b->stream));
    const int rc = vsmc_cuda_batch_run_device(b, b->d_obs);
    if (rc != VSMC_CUDA_OK)
        return rc;
    return vsmc_cuda_batch_history(
        b, mean_host, ess_host, resampled_host, logz_host);
}

int vsmc_cuda_batch_set_shape(vsmc_cuda_batch *b, int ppt, int block)
{
    if (b == nullptr || b->kind == kKindLearned)
        return VSMC_CUDA_ERR_ARG;
    for (int k = 0; k < kNumShapes; ++k)
        if (kShapes[k].ppt == ppt && kShapes[k].block == block)
            return batch_layout(b, kShapes[k]);
    return VSMC_CUDA_ERR_ARG;
}

int vsmc_cuda_batch_get_shape(vsmc_cuda_batch *b, int *ppt, int *block)
{
    if (b == nullptr || ppt == nullptr || block == nullptr)
        return VSMC_CUDA_ERR_ARG;
    *ppt = b->shape.ppt;
    *block = b->shape.block;
    return VSMC_CUDA_OK;
}

int vsmc_cuda_batch_set_schedule(vsmc_cuda_batch *b, uint32_t min_chunk)
{
    if (b == nullptr)
        return VSMC_CUDA_ERR_ARG;
    bool known = false;
    for (int k = 0; k < kNumSchedules; ++k)
        known = known || kRsSchedules[k] == min_chunk;
    if (!known)
        return VSMC_CUDA_ERR_ARG;
    for (uint32_t k = 0; k < b->nf; ++k) {
        BFilter &F = b->flt[k];
        F.rs_unit = rs_chunk_for(F.n, min_chunk) / kRsUnits;
    }
    b->rs_min_chunk = min_chunk;
    // re-uploads the filter descriptions (their chunks); the list keeps the
    // capacity of the smallest chunk, which bounds every schedule
    return batch_layout(b, b->shape);
}

int vsmc_cuda_batch_get_schedule(vsmc_cuda_batch *b, uint32_t *min_chunk)
{
    if (b == nullptr || min_chunk == nullptr)
        return VSMC_CUDA_ERR_ARG;
    *min_chunk = b->rs_min_chunk;
    return VSMC_CUDA_OK;
}

// time `nsteps` steps of the batch (one warm-up run first)
static int time_steps(vsmc_cuda_batch *b, const double *obs_dev, int nsteps,
    cudaEvent_t e0, cudaEvent_t e1, float *ms)
{
    const int grid = num_sms() * occupancy(b->kind, step_shape(b));
    int rc = enqueue_run(b, obs_dev, nsteps, grid); // warm-up
    if (rc != VSMC_CUDA_OK)
        return rc;
    VSMC_CUDA_TRY(cudaEventRecord(e0, b->stream));
    rc = enqueue_run(b, obs_dev, nsteps, grid);
    if (rc != VSMC_CUDA_OK)
        return rc;
    VSMC_CUDA_TRY(cudaEventRecord(e1, b->stream));
    VSMC_CUDA_TRY(cudaEventSynchronize(e1));
    VSMC_CUDA_TRY(cudaEventElapsedTime(ms, e0, e1));
    return VSMC_CUDA_OK;
}

int vsmc_cuda_batch_autotune_schedule(vsmc_cuda_batch *b,
    const double *obs_dev, int steps, float *ms_host)
{
    if (b == nullptr || obs_dev == nullptr || steps < 1)
        return VSMC_CUDA_ERR_ARG;
    const int nsteps = std::min(steps, static_cast<int>(b->tmax) + 1);
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    VSMC_CUDA_TRY(cudaEventCreate(&e0));
    if (cudaEventCreate(&e1) != cudaSuccess) {
        cudaEventDestroy(e0);
        return VSMC_CUDA_ERR_CUDA;
    }
    int best = -1;
    float best_ms = 0;
    int rc = VSMC_CUDA_OK;
    for (int k = 0; k < kNumSchedules && rc == VSMC_CUDA_OK; ++k) {
        rc = vsmc_cuda_batch_set_schedule(b, kRsSchedules[k]);
        float ms = 0;
        if (rc == VSMC_CUDA_OK)
            rc = time_steps(b, obs_dev, nsteps, e0, e1, &ms);
        if (rc != VSMC_CUDA_OK)
            break;
        if (ms_host)
            ms_host[k] = ms;
        if (best < 0 || ms < best_ms) {
            best = k;
            best_ms = ms;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc != VSMC_CUDA_OK)
        return rc;
    rc = check_errors(b);
    if (rc != VSMC_CUDA_OK)
        return rc;
    return vsmc_cuda_batch_set_schedule(b, kRsSchedules[best]);
}

int vsmc_cuda_batch_autotune(vsmc_cuda_batch *b, const double *obs_dev,
    int steps, float *ms_host)
{
    if (b == nullptr || obs_dev == nullptr || steps < 1 ||
        b->kind == kKindLearned)
        return VSMC_CUDA_ERR_ARG;
    const int nsteps = std::min(steps, static_cast<int>(b->tmax) + 1);
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    VSMC_CUDA_TRY(cudaEventCreate(&e0));
    if (cudaEventCreate(&e1) != cudaSuccess) {
        cudaEventDestroy(e0);
        return VSMC_CUDA_ERR_CUDA;
    }
    int best = -1;
    float best_ms = 0;
    int rc = VSMC_CUDA_OK;
    for (int k = 0; k < kNumShapes && rc == VSMC_CUDA_OK; ++k) {
        rc = batch_layout(b, kShapes[k]);
        if (rc != VSMC_CUDA_OK)
            break;
        const int grid = num_sms() * occupancy(b->kind, step_shape(b));
        rc = enqueue_run(b, obs_dev, nsteps, grid); // warm-up
        if (rc != VSMC_CUDA_OK)
            break;
        if (cudaEventRecord(e0, b->stream) != cudaSuccess) {
            rc = VSMC_CUDA_ERR_CUDA;
            break;
        }
        rc = enqueue_run(b, obs_dev, nsteps, grid);
        if (rc != VSMC_CUDA_OK)
            break;
        float ms = 0;
        if (cudaEventRecord(e1, b->stream) != cudaSuccess ||
            cudaEventSynchronize(e1) != cudaSuccess ||
            cudaEventElapsedTime(&ms, e0, e1) != cudaSuccess) {
            rc = VSMC_CUDA_ERR_CUDA;
            break;
        }
        if (ms_host)
            ms_host[k] = ms;
        if (best < 0 || ms < best_ms) {
            best = k;
            best_ms = ms;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc != VSMC_CUDA_OK)
        return rc;
    rc = check_errors(b);
    if (rc != VSMC_CUDA_OK)
        return rc;
    rc = batch_layout(b, kShapes[best]);
    if (rc != VSMC_CUDA_OK)
        return rc;
    // then the scan schedule (the resampling chunk) for that shape
    return vsmc_cuda_batch_autotune_schedule(b, obs_dev, steps, nullptr);
}

} // extern "C"
