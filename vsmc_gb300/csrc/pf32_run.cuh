// A whole run of the FP32 filter in one kernel, for filters whose blocks have
// one tile each.
//
// A step of the graph path is four dependent launches, three of which return
// at once when the step does not resample; at 1000 to 150000 particles their
// latencies are most of the step (20 to 25 us, against 2 to 8 us of work).
// Here the blocks stay resident for all steps and meet at a grid barrier:
// once a step (the records are there), and three times more in a resampling
// (range sums, counts, slots).  There is no last block: every block combines
// the records, and sums the ranges before its own, itself, on its own copy of
// the filter's scalars in shared memory, so nothing is broadcast and the
// copies stay equal.  The arithmetic, its order and the slots are those of
// k_pf_step and the k_rs32 passes (the same device functions over the same
// tiles), so results are bit-identical.
//
// Measured per step, launches against this kernel: n = 1000 19.6 -> 6.6 us
// (one block), 8192 20.7 -> 8.7 (one cluster of 8 blocks), 100003 22.0 -> 12.4
// (cooperative grid).  What is left is a chain: the tile, its warp and block
// sums, the FP64 quotient and logarithm, a grid barrier.
//
// It is taken up to a block an SM (155648 particles), where two runs are
// resident at once (kRunOcc): filters on streams of their own overlap then.
// 50 steps of 1, 2, 4, 8 and 16 filters of 155000 take 0.49, 0.59, 1.1, 2.2
// and 4.5 ms, 1.5, 1.6, 1.9, 2.4 and 4.3 by launches that returned at once
// without a resample.  A run of more blocks holds the chip while it waits at
// its barriers: filters of 300000 took 0.78, 1.5, 3.0, 6.1 and 12.1 ms, by
// the launches 1.6, 1.8, 2.1, 2.9 and 5.5 then, 1.1, 1.3, 1.7, 2.5 and 4.7
// now (figures at 320000).
#pragma once

#include "pf32.cuh"

#include <cooperative_groups.h>

namespace vsmc_cuda
{

// The grid barrier's counter and the arrivals it has to reach next.
struct RunBarrier {
    uint32_t *count;
    uint32_t target;
    uint32_t *err; // the filter's error word
};

__device__ __forceinline__ uint64_t run_clock()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// How the blocks of a run meet: one block; one cluster (the hardware's
// cluster barrier); a cooperative grid (a counter in memory, about 1.5 us).
enum class RunKind { Block, Cluster, Grid };

// Blocks an SM holds (registers), and those of them that one run may take
// (see the file comment).
constexpr int kRunOcc = 2;
constexpr int kRunShare = 1;

// Every block waits for every other; writes before it are visible after it.
// false, in every thread of the block, if the wait ran out (two seconds):
// the block then leaves the kernel.
template <RunKind Kind>
__device__ __forceinline__ bool run_barrier(RunBarrier &b)
{
    if (Kind == RunKind::Block) {
        __syncthreads();
        return true;
    }
    if (Kind == RunKind::Cluster) {
        cooperative_groups::this_cluster().sync();
        return true;
    }
    __shared__ bool ok;
    b.target += gridDim.x;
    __syncthreads();
    if (threadIdx.x == 0) {
        // the release orders the whole block's writes (the barrier above)
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;"
                     :
                     : "l"(b.count)
                     : "memory");
        const uint64_t t0 = run_clock();
        bool good = true;
        for (uint32_t k = 1;; ++k) {
            uint32_t v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];"
                         : "=r"(v)
                         : "l"(b.count)
                         : "memory");
            if (static_cast<int32_t>(v - b.target) >= 0)
                break;
            if (k % 256 == 0 && run_clock() - t0 > 2000000000ull) {
                good = false;
                atomicOr(b.err, DEV_ERR_TIMEOUT);
                break;
            }
        }
        ok = good;
    }
    __syncthreads();
    return ok;
}

// Sum of v[0 .. gridDim.x) before the block's own entry, and of all, in
// every thread (own: its entry).
template <RunKind Kind>
__device__ __forceinline__ void run_prefix(
    const uint64_t *v, uint64_t own, uint64_t &before, uint64_t &all)
{
    if (Kind == RunKind::Block) {
        before = 0;
        all = own;
        return;
    }
    constexpr int kW = kPfBlock / 32;
    __shared__ uint64_t sb[kW], sa[kW];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    before = 0;
    all = 0;
    for (uint32_t b = threadIdx.x; b < gridDim.x; b += kPfBlock) {
        const uint64_t x = __ldcg(v + b);
        all += x;
        before += b < blockIdx.x ? x : 0ull;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        before += __shfl_xor_sync(0xFFFFFFFFu, before, o);
        all += __shfl_xor_sync(0xFFFFFFFFu, all, o);
    }
    if (lane == 0) {
        sb[wid] = before;
        sa[wid] = all;
    }
    __syncthreads();
    before = 0;
    all = 0;
#pragma unroll
    for (int k = 0; k < kW; ++k) {
        before += sb[k];
        all += sa[k];
    }
    __syncthreads();
}

struct RunArgs {
    float *buf[2]; // state buffers
    int cur;       // the one that step t0 reads
    uint32_t t0, steps, tiles;
    PfScalars *sc; // the filter's scalars, before and after
    uint32_t *bar; // the barrier's counter (0)
};

// One resampling: qsum, count and assign of the block's tile.  r.sc is the
// block's copy of the scalars.  false if a wait ran out.
template <bool Sys, RunKind Kind>
__device__ __forceinline__ bool run_resample(
    const Rs32Args &r, PfScalars &sc, RunBarrier &bar)
{
    constexpr int kW = kPfBlock / 32;
    __shared__ uint64_t s_q[kW];
    __shared__ uint32_t s_e[kW], s_c[kW];
    __shared__ uint4 rows[Sys ? 1 : kRsWarps][Sys ? 1 : kStratRow];
    __shared__ __align__(16) uint32_t shm[kW][kRunChunk];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint64_t *qtot = r.qpart, *ectot = r.qpart + gridDim.x;
    uint32_t lo, hi, wlo, whi;
    chunk_range(r.n, r.chunk, lo, hi);
    warp_range(lo, hi, r.chunk, w, wlo, whi);
    {
        // a warp's range is 128 particles: one float4 per lane
        const float M = static_cast<float>(sc.M);
        const float4 v = load_lw4(r.lw, wlo + lane * 4, whi);
        uint64_t q = fixed_q(v.x, M, r.shift) + fixed_q(v.y, M, r.shift) +
            fixed_q(v.z, M, r.shift) + fixed_q(v.w, M, r.shift);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            q += __shfl_xor_sync(0xFFFFFFFFu, q, o);
        if (lane == 0)
            s_q[w] = q;
    }
    __syncthreads();
    uint64_t own = 0, carry = 0; // of the block, of its warps before
#pragma unroll
    for (int k = 0; k < kW; ++k) {
        if (static_cast<uint32_t>(k) == w)
            carry = own;
        own += s_q[k];
    }
    if (threadIdx.x == 0)
        qtot[blockIdx.x] = own;
    if (!run_barrier<Kind>(bar))
        return false;
    uint64_t before, all;
    run_prefix<Kind>(qtot, own, before, all);
    carry += before;
    if (w == 0) {
        uint32_t err = 0;
        cdf_constants(sc, all, r.n, Sys, err);
        if (lane == 0 && err)
            sc.err |= err;
    }
    __syncthreads();
    uint32_t empties = 0, copies = 0;
    {
        const CdfRcp p = load_cdf_rcp(sc, r.n);
        EnginePos e = {};
        if (!Sys)
            e = engine_pos(sc);
        uint4 *row = rows[Sys ? 0 : w];
        if (p.s != 0)
            count_range<Sys, true>(
                r, p, e, row, wlo, whi, carry, empties, copies);
        else
            count_range<Sys, false>(
                r, p, e, row, wlo, whi, carry, empties, copies);
    }
    empties = __reduce_add_sync(0xFFFFFFFFu, empties);
    copies = __reduce_add_sync(0xFFFFFFFFu, copies);
    if (lane == 0) {
        s_e[w] = empties;
        s_c[w] = copies;
    }
    __syncthreads();
    uint32_t eoff = 0, coff = 0, e = 0, c = 0;
#pragma unroll
    for (int k = 0; k < kW; ++k) {
        if (static_cast<uint32_t>(k) == w) {
            eoff = e;
            coff = c;
        }
        e += s_e[k];
        c += s_c[k];
    }
    own = (static_cast<uint64_t>(c) << 32) | e;
    if (threadIdx.x == 0)
        ectot[blockIdx.x] = own;
    if (!run_barrier<Kind>(bar))
        return false;
    run_prefix<Kind>(ectot, own, before, all);
    eoff += static_cast<uint32_t>(before);
    coff += static_cast<uint32_t>(before >> 32);
    const uint32_t etotal = static_cast<uint32_t>(all);
    float macc[kMaxMonitorDim] = {};
    assign_range<false>(r, wlo, whi, coff, eoff, etotal, shm[w], macc);
    if (threadIdx.x == kPfBlock - 1) {
        sc.nempty = etotal;
        if (static_cast<uint32_t>(all >> 32) != r.n)
            atomicOr(&sc.err, DEV_ERR_INTERNAL);
        sc.gather = 1;
        scheme_words(r, sc);
    }
    return run_barrier<Kind>(bar);
}

// Steps t0 .. t0 + steps - 1.  A block's tile is its resampling chunk too.
// The first `tiles` blocks have particles (a cluster may be larger).
template <class Model, bool Sys, RunKind Kind>
__global__ void __launch_bounds__(kPfBlock, Kind == RunKind::Grid ? kRunOcc : 1)
k_pf32_run(const PfStepArgs a0,
    const Rs32Args r0, const Model model, const RunArgs run)
{
    __shared__ PfStepSmem<Model, PfMon::Previous> sh;
    __shared__ PfScalars sc;
    __shared__ PfPartial own; // RunKind::Block: the step's record
    {
        const uint32_t *g = reinterpret_cast<const uint32_t *>(run.sc);
        uint32_t *l = reinterpret_cast<uint32_t *>(&sc);
        for (uint32_t i = threadIdx.x; i < sizeof(PfScalars) / 4; i += kPfBlock)
            l[i] = g[i];
    }
    __syncthreads();
    if (threadIdx.x == 0)
        sc.err = 0;
    RunBarrier bar = {run.bar, 0, &run.sc->err};
    PfStepArgs a = a0;
    a.sc = &sc;
    Rs32Args r = r0;
    r.sc = &sc;
    int cur = run.cur;
    __syncthreads();
    for (uint32_t k = 0; k < run.steps; ++k, cur ^= 1) {
        const uint32_t t = run.t0 + k;
        a.in = run.buf[cur];
        a.out = run.buf[cur ^ 1];
        // records by step parity: a block may be one barrier ahead
        constexpr bool kLocal = Kind == RunKind::Block;
        PfPartial *part =
            kLocal ? &own : a.part + (t & 1) * gridDim.x;
        PfPartial *mine = part + (kLocal ? 0u : blockIdx.x);
        const int resampled = t == 0 ? 1 : sc.resampled;
        if (t == 0)
            pf_step_record<Model, true, PfMon::Previous>(
                a, model, t, 1, false, 0.0f, mine, sh);
        else
            pf_step_record<Model, false, PfMon::Previous>(a, model, t,
                resampled, sc.gather != 0, static_cast<float>(sc.M), mine,
                sh);
        if (!run_barrier<Kind>(bar))
            return;
        if (t == 0)
            pf_step_combine<Model, true, PfMon::Previous, kLocal>(
                a, part, run.tiles, sc, blockIdx.x == 0, t, 1, sh);
        else
            pf_step_combine<Model, false, PfMon::Previous, kLocal>(
                a, part, run.tiles, sc, blockIdx.x == 0, t, resampled, sh);
        __syncthreads();
        if (sc.resampled && !run_resample<Sys, Kind>(r, sc, bar))
            return;
        __syncthreads();
    }
    if (threadIdx.x != 0)
        return;
    if (sc.err)
        atomicOr(&run.sc->err, sc.err);
    if (blockIdx.x == 0) {
        PfScalars &g = *run.sc;
        g.M = sc.M;
        g.Mf = sc.Mf;
        g.S = sc.S;
        g.logz = sc.logz;
        g.ess = sc.ess;
        g.Q = sc.Q;
        g.step = sc.step;
        g.resampled = sc.resampled;
        g.gather = sc.gather;
        g.nempty = sc.nempty;
        g.rindex = sc.rindex;
        for (int i = 0; i < 4; ++i)
            g.rctr[i] = sc.rctr[i];
    }
}

} // namespace vsmc_cuda
