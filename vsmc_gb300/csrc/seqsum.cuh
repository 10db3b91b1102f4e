// Left-to-right double summation, bit-identical to a sequential loop, in
// parallel.
//
// The reference accumulates its resampling CDF and its normalizing sums one
// element at a time (resample/transform.hpp:61-69, core/weight.hpp:224-229,
// resample/transform.hpp:164).  For non-negative terms the running sum s is
// non-decreasing, and while s_{i-1} and s_i stay in one binade [2^e, 2^(e+1))
// every partial sum is a multiple of u = 2^(e-52), so
//     s_i = fl(s_{i-1} + x_i) = s_{i-1} + rint(x_i / u) * u
// whenever x_i / u is not exactly half-way (a tie rounds to even, which
// depends on s_{i-1}).  The increment r_i = rint(x_i / u) is an exact integer
// that does not depend on s_{i-1}, and the sum's bit pattern grows by exactly
// r_i, so a run of such elements is an integer prefix sum.  What is left --
// elements whose running sum may cross a power of two, ties, and sums too
// small for the relative bounds -- is a short list of breakpoints, evaluated
// in order by one thread with real IEEE additions.
//
// Three passes over x, in tiles of 2048 elements.  Each pass is a grid of
// kSeqOcc blocks per SM; a block walks one range of consecutive tiles:
//   sums      approximate tile sums, as prefixes within the range; the last
//             block to finish (its ticket; nothing waits) turns the ranges'
//             totals into prefixes.  Together: P before every tile;
//   classify  a tile whose P and next P lie in one binade (with margin) has
//             one ulp for all its elements: its total increment is a sum of
//             integers.  Ties, and the few tiles that cross a binade (element
//             prefixes in FP64 there), list their breakpoints.  The last
//             block walks the breakpoints and leaves every range's exact
//             starting sum;
//   out       the increments again, as an integer prefix sum on top of the
//             tile's starting sum, handed to a functor (store, count).
// A caller that wants the total only stops after the second pass.
//
// P's margin is m = 4 n 2^-53 relative (at least 2^-40): |sequential - exact|
// is at most (n - 1) 2^-53 and |P - exact| below 2^-43.  Few elements lie
// that close to a power of two, so the serial walk (64 cycles of FP64 add
// latency and about as many around it per breakpoint) stays short: 50
// breakpoints at n = 2^24 instead of 180 at a fixed m = 2^-19.
//
// GB300 issues an FP64 instruction of a warp in 19 cycles of its SM (measured;
// an integer one in half a cycle), so nothing per element is FP64: tile sums
// add mantissas aligned to the warp's largest exponent (error below 2^-52 of
// that element each), and increments are shifts.
//
// At n = 2^24: sums 27 us (x read at 4.9 TB/s), classify 55 us (36 with the
// ALU pipe 60 % busy, then the last block's serial walk), out 52 us (5.1 TB/s),
// against
// 0.46 ms for two generic scans (FP64 prefixes, then 16-byte increment
// records) that moved 104 bytes per element.
#pragma once

#include "common.cuh"
#include "scan.cuh"

#include <cmath>
#include <cooperative_groups.h>
#include <type_traits>

namespace vsmc_cuda
{

constexpr int kSeqBlock = 256;
constexpr int kSeqWarps = kSeqBlock / 32;
constexpr int kSeqItems = 8; // elements of a thread
constexpr int kSeqTile = kSeqBlock * kSeqItems;
constexpr int kSeqMaxRanges = 1023;
// a warp's 256 staged elements, 16 bytes of padding after every eight
constexpr int kSeqRowBytes = 32 * 80;

struct SeqArgs {
    uint32_t n;      // elements
    uint32_t nt;     // tiles
    uint32_t tb;     // most tiles of a block's range
    uint32_t blocks; // ranges: range b is tiles [b nt / blocks, (b + 1) nt / blocks)
    uint64_t flo, fhi; // the margin's bounds on the fraction field
    // per range, blocks + 1 each
    double *P;    // approximate sums, then their exclusive prefixes
    uint64_t *R;  // increments
    uint32_t *F;  // breakpoints
    uint64_t *start; // bit pattern of the exact sum before each range
    // per tile, tb + 1 per range: the same within the range, before the tile
    double *tP;
    uint64_t *tR;
    uint32_t *tF;
    // breakpoint k of range b, from its first element's place on: the range's
    // increments through it, then its sum's bit pattern minus them; its
    // element; its sum's sign and exponent
    uint64_t *adj;
    uint32_t *pos;
    uint16_t *bex;
    double *total; // the sum (may be null)
    double *inv;   // its reciprocal (may be null)
    uint32_t *err;  // error word; the two words after it are the tickets
    int allow_inf;  // +inf terms are summed as a sequential loop would
};

// The margin tests on the fraction field f (units of 2^-52) of P, with
// flo = 2^53 m and fhi = 2^52 - 2^53 m:
//   P (1 - m) >= 2^e       holds when f >= flo > 2^52 m / (1 - m)
//   P (1 + m) <  2^(e + 1) holds when f <  fhi < 2^52 (1 - m) / (1 + m)
constexpr uint64_t kFracMask = (1ull << 52) - 1;
constexpr uint32_t kExpMin = 1023 - 1000; // running sums below 2^-1000 are breakpoints
constexpr uint64_t kInfBits = 0x7FF0000000000000ull;

__device__ __forceinline__ uint64_t dbits(double v)
{
    return static_cast<uint64_t>(__double_as_longlong(v));
}

__device__ __forceinline__ double from_dbits(uint64_t b)
{
    return __longlong_as_double(static_cast<long long>(b));
}

// whether running sums between approximate prefixes pa and pb stay in pa's
// binade
__device__ __forceinline__ bool seq_one_binade(
    const SeqArgs &a, uint64_t pa, uint64_t pb)
{
    const uint32_t ea = static_cast<uint32_t>(pa >> 52); // sign bit included
    return ea >= kExpMin && ea <= 2046u && (pa & kFracMask) >= a.flo &&
        static_cast<uint32_t>(pb >> 52) == ea && (pb & kFracMask) < a.fhi;
}

// Increment of x (bits xb) in ulps of the binade with biased exponent ea;
// regular is false for a tie, for x above the binade and for x that is not
// a finite non-negative number (r is 0 then).
__device__ __forceinline__ uint64_t seq_increment(
    uint64_t xb, uint32_t ea, bool &regular)
{
    const uint32_t xe = static_cast<uint32_t>(xb >> 52); // sign bit included
    const uint64_t xf = xb & kFracMask;
    const uint64_t mant = xe ? (xf | (1ull << 52)) : xf;
    // x / ulp = mant / 2^k
    const int k = static_cast<int>(ea) - static_cast<int>(xe ? xe : 1u);
    const int kk = k < 1 ? 1 : (k > 63 ? 63 : k);
    // rounded half up; exactly half leaves no remainder.  k >= 63: below
    // half a unit, and no tie
    const uint64_t t = mant + (1ull << (kk - 1));
    const uint64_t r = t >> kk;
    const bool exact_unit = k == 0;
    regular = ((k >= 1 && (r << kk) != t) || exact_unit) && xe < 0x7FFu;
    // -0 adds nothing
    if (xb == 0x8000000000000000ull) {
        regular = true;
        return 0;
    }
    return regular ? (exact_unit ? mant : r) : 0;
}

// seq_increment for x known to be below 2^e of the binade (so finite, not
// negative, and k >= 1) with ea >= 64 (a denormal x is far below half a
// unit): 16 integer instructions instead of about 25.
__device__ __forceinline__ uint64_t seq_increment_below(
    uint64_t xb, uint32_t ea, bool &tie)
{
    const uint32_t k = min(ea - static_cast<uint32_t>(xb >> 52), 63u);
    const uint64_t t = ((xb & kFracMask) | (1ull << 52)) + (1ull << (k - 1));
    const uint64_t r = t >> k;
    tie = (r << k) == t;
    return r;
}

// whether every value of the warp is below 2^e of the binade ea, ea >= 64
__device__ __forceinline__ bool seq_all_below(
    const double (&v)[kSeqItems], uint32_t ea)
{
    uint32_t top = 0;
#pragma unroll
    for (int k = 0; k < kSeqItems; ++k)
        top = max(top, static_cast<uint32_t>(__double2hiint(v[k])));
    return ea >= 64 &&
        __all_sync(0xFFFFFFFFu, top < (ea << 20));
}

// The increments of 8 values in a tile of one binade; false if one is not
// regular (its increment is 0).
__device__ __forceinline__ bool seq_increments(
    const double (&v)[kSeqItems], uint32_t ea, uint64_t (&r)[kSeqItems])
{
    bool ok = true;
    if (seq_all_below(v, ea)) {
#pragma unroll
        for (int k = 0; k < kSeqItems; ++k) {
            bool tie;
            r[k] = seq_increment_below(dbits(v[k]), ea, tie);
            if (tie)
                r[k] = 0;
            ok &= !tie;
        }
    } else {
#pragma unroll
        for (int k = 0; k < kSeqItems; ++k) {
            bool reg;
            r[k] = seq_increment(dbits(v[k]), ea, reg);
            ok &= reg;
        }
    }
    return ok;
}

// Sum of one 32-bit piece per lane over the warp, in every lane.
__device__ __forceinline__ uint32_t warp_add32(uint32_t v)
{
    return __reduce_add_sync(0xFFFFFFFFu, v);
}

// Sum over the warp of per-lane values below 2^56 whose total stays below
// 2^64, by three 32-bit reductions of 27-bit pieces.
__device__ __forceinline__ uint64_t warp_add56(uint64_t v)
{
    const uint32_t m = (1u << 27) - 1;
    const uint32_t a = warp_add32(static_cast<uint32_t>(v) & m);
    const uint32_t b = warp_add32(static_cast<uint32_t>(v >> 27) & m);
    const uint32_t c = warp_add32(static_cast<uint32_t>(v >> 54));
    return a + (static_cast<uint64_t>(b) << 27) +
        (static_cast<uint64_t>(c) << 54);
}

// Shared memory of one tile.
struct SeqSmem {
    alignas(16) unsigned char row[kSeqWarps][kSeqRowBytes];
    // warp results, one set per tile parity: a block walks its tiles with
    // one barrier each
    uint64_t w64[2][kSeqWarps];
    uint32_t w32[2][kSeqWarps];
    uint64_t rR; // the range's increments and breakpoints so far
    uint32_t rF;
    uint32_t last;
};

// The element index of slot k of the calling thread: striped (warp rows of
// 32 consecutive elements).
__device__ __forceinline__ uint32_t seq_striped(uint32_t tile, int k)
{
    return tile * kSeqTile + (threadIdx.x >> 5) * 256u +
        static_cast<uint32_t>(k) * 32u + (threadIdx.x & 31);
}

// A warp's striped values to blocked ones (lane l gets elements 8 l ..
// 8 l + 7 of the warp's 256) and back, through its row.
__device__ __forceinline__ void seq_to_blocked(
    unsigned char *row, const double (&v)[kSeqItems], double (&b)[kSeqItems])
{
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < kSeqItems; ++k) {
        const uint32_t e = static_cast<uint32_t>(k) * 32u + lane;
        *reinterpret_cast<double *>(row + (e >> 3) * 80 + (e & 7) * 8) = v[k];
    }
    __syncwarp();
    const double2 *q = reinterpret_cast<const double2 *>(row + lane * 80);
#pragma unroll
    for (int k = 0; k < kSeqItems / 2; ++k) {
        const double2 p = q[k];
        b[2 * k] = p.x;
        b[2 * k + 1] = p.y;
    }
    __syncwarp();
}

__device__ __forceinline__ void seq_to_striped(
    unsigned char *row, const double (&b)[kSeqItems], double (&v)[kSeqItems])
{
    const uint32_t lane = threadIdx.x & 31;
    __syncwarp();
    double2 *q = reinterpret_cast<double2 *>(row + lane * 80);
#pragma unroll
    for (int k = 0; k < kSeqItems / 2; ++k)
        q[k] = make_double2(b[2 * k], b[2 * k + 1]);
    __syncwarp();
#pragma unroll
    for (int k = 0; k < kSeqItems; ++k) {
        const uint32_t e = static_cast<uint32_t>(k) * 32u + lane;
        v[k] = *reinterpret_cast<const double *>(
            row + (e >> 3) * 80 + (e & 7) * 8);
    }
}

// The whole-block ticket of a pass: true in every thread of the block that
// finishes it last, whose thread 0 resets it.
__device__ __forceinline__ bool seq_last_block(uint32_t *ticket, SeqSmem &sh)
{
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const bool l = atomicAdd(ticket, 1u) == gridDim.x - 1;
        if (l)
            *ticket = 0;
        sh.last = l ? 1u : 0u;
    }
    __syncthreads();
    if (sh.last)
        __threadfence();
    return sh.last != 0;
}

// ------------------------------------------------------------- tile sums

// t 2^(E - 1075) as a double (E = 0xFFFF: infinite), by the exponent field
// where the result is a normal number
__device__ __forceinline__ double seq_scaled(uint64_t t, uint32_t E)
{
    if (E == 0xFFFFu)
        return from_dbits(kInfBits);
    const double d = __ull2double_rn(t);
    const int e = static_cast<int>(E) - 1075;
    if (t != 0 && E > 64 && E < 1983)
        return __hiloint2double(
            __double2hiint(d) + (e << 20), __double2loint(d));
    return ldexp(d, e);
}

// Approximate sum of the tile's values (v striped, 0 past the end), valid
// in thread 0.  Negative, NaN and (unless allowed) infinite values are
// reported and count as 0.
__device__ __forceinline__ double seq_tile_sum(const double (&v)[kSeqItems],
    int allow_inf, uint32_t *err, SeqSmem &sh, int par)
{
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t top = 0;
#pragma unroll
    for (int k = 0; k < kSeqItems; ++k)
        top = max(top, static_cast<uint32_t>(__double2hiint(v[k])));
    top = __reduce_max_sync(0xFFFFFFFFu, top);
    bool inf = false;
    uint64_t acc = 0;
    uint32_t E;
    if (top < 0x7FF00000u) {
        E = max(top >> 20, 1u);
#pragma unroll
        for (int k = 0; k < kSeqItems; ++k) {
            const uint64_t xb = dbits(v[k]);
            const uint32_t xe = static_cast<uint32_t>(xb >> 52);
            const uint64_t xf = xb & kFracMask;
            const uint64_t mant = xe ? (xf | (1ull << 52)) : xf;
            acc += mant >> min(E - max(xe, 1u), 63u);
        }
    } else { // a sign bit, an infinity or a NaN among them
        uint32_t hi = 0;
        bool bad = false;
#pragma unroll
        for (int k = 0; k < kSeqItems; ++k) {
            const uint64_t xb = dbits(v[k]);
            if (xb == kInfBits)
                inf = true;
            else if (xb > kInfBits && xb != 0x8000000000000000ull)
                bad = true;
            else if (xb < kInfBits)
                hi = max(hi, static_cast<uint32_t>(xb >> 32));
        }
        if ((bad || (inf && !allow_inf)) && err)
            atomicOr(err, DEV_ERR_NONFINITE);
        inf = __any_sync(0xFFFFFFFFu, inf) && allow_inf;
        hi = __reduce_max_sync(0xFFFFFFFFu, hi);
        E = max(hi >> 20, 1u);
#pragma unroll
        for (int k = 0; k < kSeqItems; ++k) {
            const uint64_t xb = dbits(v[k]);
            if (xb >= kInfBits)
                continue;
            const uint32_t xe = static_cast<uint32_t>(xb >> 52);
            const uint64_t xf = xb & kFracMask;
            const uint64_t mant = xe ? (xf | (1ull << 52)) : xf;
            acc += mant >> min(E - max(xe, 1u), 63u);
        }
    }
    acc = warp_add56(acc); // below 2^61: 256 values below 2^53
    if (lane == 0) {
        sh.w64[par][w] = acc;
        sh.w32[par][w] = inf ? 0xFFFFu : E;
    }
    __syncthreads();
    double s = 0;
    if (w == 0) {
        const uint32_t e = lane < kSeqWarps ? sh.w32[par][lane] : 1u;
        const uint32_t Em = __reduce_max_sync(0xFFFFFFFFu, e);
        uint64_t t = lane < kSeqWarps ? sh.w64[par][lane] >> min(Em - e, 63u) : 0;
#pragma unroll
        for (int o = kSeqWarps / 2; o > 0; o >>= 1)
            t += __shfl_xor_sync(0xFFFFFFFFu, t, o);
        if (lane == 0)
            s = seq_scaled(t, Em);
    }
    return s;
}

// P[0..m) replaced by its exclusive prefixes, P[m] the total, by one block
// of kB threads (m at most a few per thread).
template <int kB>
__device__ __forceinline__ void seq_scan_sums(double *P, uint32_t m)
{
    constexpr uint32_t kK = 4;
    const uint32_t per = (m + kB - 1) / kB;
    const uint32_t b0 = min(m, threadIdx.x * per);
    const uint32_t b1 = min(m, b0 + per);
    double s = 0;
    for (uint32_t i = b0; i < b1; i += kK) {
        double x[kK];
#pragma unroll
        for (uint32_t k = 0; k < kK; ++k)
            x[k] = i + k < b1 ? __ldcg(P + i + k) : 0.0;
#pragma unroll
        for (uint32_t k = 0; k < kK; ++k)
            if (i + k < b1)
                s += x[k];
    }
    double tot;
    double run = block_excl_any<double, OpAdd, kB>(s, OpAdd(), 0.0, &tot);
    for (uint32_t i = b0; i < b1; ++i) {
        const double x = __ldcg(P + i);
        P[i] = run;
        run += x;
    }
    if (threadIdx.x == 0)
        P[m] = tot;
}

// -------------------------------------------------------------- classify

// Increments and breakpoints of one tile: its total increment and breakpoint
// count in R and F (thread 0), its breakpoints appended to the range's list
// at l0 (sh.rR / sh.rF hold the range's increments and breakpoints before
// the tile).  v holds the values striped, 0 past the end; pa and pb are the
// approximate prefixes before and after the tile.
__device__ __forceinline__ void seq_classify_tile(const SeqArgs &a,
    uint32_t tile, size_t l0, const double (&v)[kSeqItems], double pa,
    double pb, SeqSmem &sh, int par, uint64_t &R, uint32_t &F)
{
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint64_t ba = dbits(pa), bb = dbits(pb);
    // no increments while the sum is infinite, or zero throughout
    const bool still = ba == kInfBits || bb == 0;
    const bool one = seq_one_binade(a, ba, bb);
    if (still) {
        R = 0;
        F = 0;
        __syncthreads(); // every tile has a barrier
        return;
    }
    if (one) {
        const uint32_t ea = static_cast<uint32_t>(ba >> 52);
        uint64_t ri[kSeqItems];
        const bool irregular = !seq_increments(v, ea, ri);
        uint64_t r = 0;
#pragma unroll
        for (int k = 0; k < kSeqItems; ++k)
            r += ri[k];
        r = warp_add56(r);
        if (lane == 0)
            sh.w64[par][w] = r;
        if (!__syncthreads_or(irregular)) {
            if (threadIdx.x == 0) {
                uint64_t t = 0;
#pragma unroll
                for (int k = 0; k < kSeqWarps; ++k)
                    t += sh.w64[par][k];
                R = t;
                F = 0;
            }
            return;
        }
    }
    // ---- the tile has breakpoints: element by element, in order
    double x[kSeqItems];
    seq_to_blocked(sh.row[w], v, x);
    const uint32_t first = tile * kSeqTile + threadIdx.x * kSeqItems;
    uint64_t r[kSeqItems];
    uint32_t f = 0; // breakpoint mask
    if (one) {
        const uint32_t ea = static_cast<uint32_t>(ba >> 52);
#pragma unroll
        for (int k = 0; k < kSeqItems; ++k) {
            bool reg;
            r[k] = seq_increment(dbits(x[k]), ea, reg);
            if (!reg)
                f |= 1u << k;
        }
    } else {
        // element prefixes in FP64 on top of the tile's
        double s = 0;
#pragma unroll
        for (int k = 0; k < kSeqItems; ++k)
            s += x[k];
        double tot;
        double run = pa +
            block_excl_any<double, OpAdd, kSeqBlock>(s, OpAdd(), 0.0, &tot);
        uint64_t p = dbits(run);
#pragma unroll
        for (int k = 0; k < kSeqItems; ++k) {
            run += x[k];
            const uint64_t q = dbits(run);
            bool reg = false;
            r[k] = 0;
            if (p == kInfBits || q == 0) {
                reg = true;
            } else if (seq_one_binade(a, p, q)) {
                r[k] = seq_increment(
                    dbits(x[k]), static_cast<uint32_t>(p >> 52), reg);
            }
            if (!reg)
                f |= 1u << k;
            p = q;
        }
    }
    uint64_t rs = 0;
    uint32_t fs = 0;
#pragma unroll
    for (int k = 0; k < kSeqItems; ++k) {
        if (first + k >= a.n) {
            r[k] = 0;
            f &= ~(1u << k);
        }
        rs += r[k];
    }
    fs = __popc(f);
    struct RF {
        uint64_t r;
        uint32_t f, pad;
    };
    struct OpRF {
        __device__ __forceinline__ RF operator()(
            const RF &x, const RF &y) const
        {
            return {x.r + y.r, x.f + y.f, 0u};
        }
    };
    RF tot;
    RF run = block_excl_any<RF, OpRF, kSeqBlock>(
        RF{rs, fs, 0u}, OpRF(), RF{0, 0, 0}, &tot);
#pragma unroll
    for (int k = 0; k < kSeqItems; ++k) {
        run.r += r[k];
        if (f & (1u << k)) {
            const size_t id = l0 + sh.rF + run.f;
            a.adj[id] = sh.rR + run.r;
            a.pos[id] = first + k;
            ++run.f;
        }
    }
    R = tot.r;
    F = tot.f;
    __syncthreads(); // rR and rF are read above, and change next
}

// first tile of range b
__device__ __forceinline__ uint32_t seq_first_tile(
    const SeqArgs &a, uint32_t b)
{
    return static_cast<uint32_t>(
        static_cast<uint64_t>(b) * a.nt / a.blocks);
}

// The largest b with F[b] <= g, for exclusive prefixes F[0..m] (F[0] = 0)
// and g < F[m]: the range that breakpoint g is in.
__device__ __forceinline__ uint32_t seq_range_of(
    const uint32_t *F, uint32_t m, uint32_t g)
{
    uint32_t lo = 0, hi = m; // F[lo] <= g < F[hi]
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (F[mid] <= g)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

// m breakpoints in order by one thread: x their elements, cr the increments
// through each, replaced by their sums' bit patterns; S the running sum's
// bit pattern and crprev the increments at the last breakpoint before.
__device__ __forceinline__ void seq_walk(const double *x, uint64_t *cr,
    uint32_t m, uint64_t &S, uint64_t &crprev, uint32_t *err)
{
    bool off = false;
    uint64_t c = cr[0];
    double v = x[0];
    for (uint32_t j = 0; j < m; ++j) {
        const uint32_t jn = j + 1 < m ? j + 1 : j;
        const uint64_t nc = cr[jn];
        const double nv = x[jn];
        // the regular elements since the last breakpoint stay in its binade
        const uint64_t q = S + (c - crprev);
        off |= (q >> 52) != (S >> 52);
        S = dbits(__dadd_rn(from_dbits(q), v));
        cr[j] = S;
        crprev = c;
        c = nc;
        v = nv;
    }
    if (off)
        atomicOr(err, DEV_ERR_BOUND);
}

// Walks the breakpoints of all ranges in order with real additions, by one
// block of kB threads after every tile was classified: exclusive prefixes
// of R and F, each range's exact starting sum, the breakpoints' sums and
// the total.  load(i) is element i.
template <int kB, class Load>
__device__ __forceinline__ void seq_fixup(const SeqArgs &a, const Load &load)
{
    __shared__ double s_x[kB];
    __shared__ uint64_t s_cr[kB];
    __shared__ uint64_t s_R[kSeqMaxRanges + 1];
    __shared__ uint32_t s_F[kSeqMaxRanges + 1];
    const uint32_t nr = a.blocks;
    struct RF {
        uint64_t r;
        uint32_t f, pad;
    };
    struct OpRF {
        __device__ __forceinline__ RF operator()(
            const RF &x, const RF &y) const
        {
            return {x.r + y.r, x.f + y.f, 0u};
        }
    };
    const uint32_t per = (nr + kB - 1) / kB;
    const uint32_t b0 = min(nr, threadIdx.x * per);
    const uint32_t b1 = min(nr, b0 + per);
    RF acc = {0, 0, 0};
    for (uint32_t i = b0; i < b1; ++i) {
        acc.r += __ldcg(a.R + i);
        acc.f += __ldcg(a.F + i);
    }
    RF tot;
    RF run = block_excl_any<RF, OpRF, kB>(acc, OpRF(), RF{0, 0, 0}, &tot);
    for (uint32_t i = b0; i < b1; ++i) {
        const uint64_t r = __ldcg(a.R + i);
        const uint32_t f = __ldcg(a.F + i);
        s_R[i] = run.r;
        s_F[i] = run.f;
        run.r += r;
        run.f += f;
    }
    if (threadIdx.x == 0) {
        s_R[nr] = tot.r;
        s_F[nr] = tot.f;
    }
    __syncthreads();
    auto list = [&](uint32_t b) {
        return static_cast<size_t>(seq_first_tile(a, b)) * kSeqTile;
    };
    const uint32_t nbk = tot.f;
    uint64_t S = 0; // the running sum's bit pattern at the last breakpoint
    uint64_t crprev = 0;
    for (uint32_t c0 = 0; c0 < nbk; c0 += kB) {
        const uint32_t g = c0 + threadIdx.x;
        size_t id = 0;
        uint64_t lr = 0;
        if (g < nbk) {
            const uint32_t b = seq_range_of(s_F, nr, g);
            id = list(b) + (g - s_F[b]);
            lr = __ldcg(a.adj + id);
            s_cr[threadIdx.x] = s_R[b] + lr;
            s_x[threadIdx.x] = load(__ldcg(a.pos + id));
        }
        __syncthreads();
        if (threadIdx.x == 0)
            seq_walk(s_x, s_cr, min(nbk - c0, static_cast<uint32_t>(kB)), S,
                crprev, a.err);
        __syncthreads();
        if (g < nbk) {
            const uint64_t s = s_cr[threadIdx.x];
            a.adj[id] = s - lr;
            a.bex[id] = static_cast<uint16_t>(s >> 52);
        }
        __syncthreads();
    }
    // every range's starting sum from the last breakpoint before it
    for (uint32_t b = threadIdx.x; b <= nr; b += kB) {
        const uint32_t g = s_F[b];
        uint64_t s = 0;
        if (g > 0) {
            const uint32_t q = seq_range_of(s_F, nr, g - 1);
            s = a.adj[list(q) + (g - 1 - s_F[q])] + (s_R[b] - s_R[q]);
        } else if (s_R[b] != 0) {
            atomicOr(a.err, DEV_ERR_INTERNAL); // a first sum is listed
        }
        a.start[b] = s;
        if (b == nr) {
            const double t = from_dbits(s);
            if (a.total)
                *a.total = t;
            if (a.inv)
                *a.inv = 1.0 / t;
        }
    }
}

// --------------------------------------------------------------- output

// The exact running sums of one tile (v: values striped, 0 past the end),
// handed to out(tile, i0, s, sprev, sh): s holds the sums of elements
// i0 .. i0 + 7 (blocked; i0 may reach past n), sprev the sum before i0.
// start, ea: the bit pattern before the tile, and the sign and exponent its
// increments are in; tR: the range's increments before the tile; the tile's
// nb breakpoints are at l0 of the lists.
template <class Out>
__device__ __forceinline__ void seq_out_tile(const SeqArgs &a, uint32_t tile,
    const double (&v)[kSeqItems], uint64_t start, uint32_t ea0, uint64_t tR,
    size_t l0, uint32_t nb, SeqSmem &sh, int par, const Out &out)
{
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t i0 = tile * kSeqTile + threadIdx.x * kSeqItems;
    double x[kSeqItems];
    seq_to_blocked(sh.row[w], v, x);
    uint64_t r[kSeqItems]; // increments, then bit patterns
    double s[kSeqItems];
    // increments of the tile before the thread's first element
    auto before = [&](uint64_t rs) {
        const uint64_t wincl = warp_incl_any(rs, OpAdd());
        if (lane == 31)
            sh.w64[par][w] = wincl;
        __syncthreads();
        uint64_t pre = wincl - rs;
#pragma unroll
        for (int k = 0; k < kSeqWarps; ++k)
            if (static_cast<uint32_t>(k) < w)
                pre += sh.w64[par][k];
        return pre;
    };
    if (nb == 0) {
        if (start == 0 || start == kInfBits) { // zero or infinite throughout
#pragma unroll
            for (int k = 0; k < kSeqItems; ++k)
                r[k] = 0;
        } else {
            seq_increments(x, ea0, r);
        }
        uint64_t rs = 0;
#pragma unroll
        for (int k = 0; k < kSeqItems; ++k)
            rs += r[k];
        uint64_t b = start + before(rs);
        const double sprev = from_dbits(b);
#pragma unroll
        for (int k = 0; k < kSeqItems; ++k) {
            b += r[k];
            s[k] = from_dbits(b);
        }
        // the tile's sums stay in the binade of its starting sum
        if ((b >> 52) != (start >> 52))
            atomicOr(a.err, DEV_ERR_BOUND);
        out(tile, i0, s, sprev, sh);
        return;
    }
    // breakpoint marks in the staging rows (one byte per element)
    __syncthreads();
    unsigned char *mark = &sh.row[0][0];
    *reinterpret_cast<uint64_t *>(mark + threadIdx.x * kSeqItems) = 0;
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < nb; j += kSeqBlock)
        mark[a.pos[l0 + j] - tile * kSeqTile] = 1;
    __syncthreads();
    const uint64_t m =
        *reinterpret_cast<uint64_t *>(mark + threadIdx.x * kSeqItems);
    uint32_t tot;
    uint32_t k0 = block_excl_any<uint32_t, OpAdd, kSeqBlock>(
        static_cast<uint32_t>(__popcll(m)), OpAdd(), 0u, &tot);
    uint64_t cur = start; // the bit pattern the tile's increments add to
    uint32_t ea = ea0;
    if (k0 > 0) {
        cur = a.adj[l0 + k0 - 1] + tR;
        ea = a.bex[l0 + k0 - 1];
    }
    const uint64_t first = cur;
    uint64_t base[kSeqItems];
    uint64_t rs = 0;
#pragma unroll
    for (int k = 0; k < kSeqItems; ++k) {
        const bool bp = (m >> (8 * k)) & 1;
        if (bp) {
            cur = a.adj[l0 + k0] + tR;
            ea = a.bex[l0 + k0];
            ++k0;
        }
        bool reg;
        r[k] = seq_increment(dbits(x[k]), ea, reg);
        // no increment of a breakpoint itself, nor while the sum is zero or
        // infinite
        if (bp || ea == 0x7FFu || (ea == 0 && cur == 0))
            r[k] = 0;
        base[k] = cur;
        rs += r[k];
    }
    uint64_t pre = before(rs);
    const double sprev = from_dbits(first + pre);
#pragma unroll
    for (int k = 0; k < kSeqItems; ++k) {
        pre += r[k];
        s[k] = from_dbits(base[k] + pre);
    }
    out(tile, i0, s, sprev, sh);
}

// ---------------------------------------------------------------- kernels

template <class Load>
__device__ __forceinline__ void seq_load(
    const Load &load, uint32_t tile, uint32_t n, double (&v)[kSeqItems])
{
#pragma unroll
    for (int k = 0; k < kSeqItems; ++k) {
        const uint32_t i = seq_striped(tile, k);
        v[k] = i < n ? load(i) : 0.0;
    }
}

// Blocks per SM of each pass.  The sums and classify passes load the next
// tile's values ahead of the current one's barrier (64 registers).
constexpr int kSeqOcc = 4;

__device__ __forceinline__ void seq_range(
    const SeqArgs &a, uint32_t &t0, uint32_t &t1)
{
    t0 = seq_first_tile(a, blockIdx.x);
    t1 = seq_first_tile(a, blockIdx.x + 1);
}

template <class Load>
__global__ void __launch_bounds__(kSeqBlock, kSeqOcc) k_seq_sums(
    const SeqArgs a, const Load load)
{
    pdl_begin();
    __shared__ SeqSmem sh;
    uint32_t t0, t1;
    seq_range(a, t0, t1);
    double v[kSeqItems], nv[kSeqItems];
    seq_load(load, t0, a.n, nv);
    double run = 0; // thread 0: the range's sum so far
    double *tP = a.tP + static_cast<size_t>(blockIdx.x) * (a.tb + 1);
    int par = 0;
    for (uint32_t t = t0; t < t1; ++t, par ^= 1) {
#pragma unroll
        for (int k = 0; k < kSeqItems; ++k)
            v[k] = nv[k];
        if (t + 1 < t1)
            seq_load(load, t + 1, a.n, nv);
        const double s = seq_tile_sum(v, a.allow_inf, a.err, sh, par);
        if (threadIdx.x == 0) {
            tP[t - t0] = run;
            run += s;
        }
    }
    if (threadIdx.x == 0) {
        tP[t1 - t0] = run;
        a.P[blockIdx.x] = run;
    }
    if (seq_last_block(a.err + 1, sh))
        seq_scan_sums<kSeqBlock>(a.P, a.blocks);
}

template <class Load>
__global__ void __launch_bounds__(kSeqBlock, kSeqOcc) k_seq_classify(
    const SeqArgs a, const Load load)
{
    pdl_begin();
    __shared__ SeqSmem sh;
    uint32_t t0, t1;
    seq_range(a, t0, t1);
    double v[kSeqItems], nv[kSeqItems];
    seq_load(load, t0, a.n, nv);
    const double P0 = a.P[blockIdx.x];
    const size_t tt = static_cast<size_t>(blockIdx.x) * (a.tb + 1);
    const size_t l0 = static_cast<size_t>(t0) * kSeqTile;
    double pb = P0 + a.tP[tt];
    if (threadIdx.x == 0) {
        sh.rR = 0;
        sh.rF = 0;
    }
    __syncthreads();
    int par = 0;
    for (uint32_t t = t0; t < t1; ++t, par ^= 1) {
#pragma unroll
        for (int k = 0; k < kSeqItems; ++k)
            v[k] = nv[k];
        const double pa = pb;
        pb = P0 + a.tP[tt + (t - t0) + 1];
        if (t + 1 < t1)
            seq_load(load, t + 1, a.n, nv);
        uint64_t R = 0;
        uint32_t F = 0;
        seq_classify_tile(a, t, l0, v, pa, pb, sh, par, R, F);
        if (threadIdx.x == 0) {
            a.tR[tt + (t - t0)] = sh.rR;
            a.tF[tt + (t - t0)] = sh.rF;
            sh.rR += R;
            sh.rF += F;
        }
    }
    if (threadIdx.x == 0) {
        a.tR[tt + (t1 - t0)] = sh.rR;
        a.tF[tt + (t1 - t0)] = sh.rF;
        a.R[blockIdx.x] = sh.rR;
        a.F[blockIdx.x] = sh.rF;
    }
    if (seq_last_block(a.err + 2, sh))
        seq_fixup<kSeqBlock>(a, load);
}

__device__ __forceinline__ void seq_prefetch(const void *p)
{
    asm volatile("prefetch.global.L2 [%0];" : : "l"(p));
}

template <class Load, class Out>
__global__ void __launch_bounds__(kSeqBlock, kSeqOcc) k_seq_out(
    const SeqArgs a, const Load load, const Out out)
{
    pdl_begin();
    __shared__ SeqSmem sh;
    uint32_t t0, t1;
    seq_range(a, t0, t1);
    const uint64_t start0 = a.start[blockIdx.x];
    const size_t tt = static_cast<size_t>(blockIdx.x) * (a.tb + 1);
    const size_t l0 = static_cast<size_t>(t0) * kSeqTile;
    double v[kSeqItems];
    int par = 0;
    for (uint32_t t = t0; t < t1; ++t, par ^= 1) {
        seq_load(load, t, a.n, v);
        const uint64_t tR = a.tR[tt + (t - t0)];
        const uint32_t f0 = a.tF[tt + (t - t0)];
        const uint32_t nb = a.tF[tt + (t - t0) + 1] - f0;
        // the last breakpoint before the tile, else the range's start
        const uint64_t start = (f0 ? a.adj[l0 + f0 - 1] : start0) + tR;
        // half the threads bring the next tile's lines to L2, half what out
        // reads for this one
        if (threadIdx.x < kSeqTile / 16) {
            const uint32_t i = (t + 1) * kSeqTile + threadIdx.x * 16;
            if (t + 1 < t1 && i < a.n)
                seq_prefetch(load.at(i));
        } else {
            out.prefetch(from_dbits(start), threadIdx.x - kSeqTile / 16);
        }
        seq_out_tile(a, t, v, start, static_cast<uint32_t>(start >> 52), tR,
            l0 + f0, nb, sh, par, out);
    }
}

// ------------------------------------------------------- one-cluster sums
//
// Up to kSeqSmall elements in one launch: a cluster of at most 8 blocks, a
// tile each, with the values in registers throughout and the partial results
// and breakpoint lists in (distributed) shared memory; hardware cluster
// barriers between the phases.  Three dependent launches with their tickets
// and lists in L2 made a systematic resampling call at n = 1000 83 us; it
// takes 41 us with this kernel.  Above 8 tiles (the portable cluster size)
// the passes above take over.

constexpr uint32_t kSeqSmallTiles = 8; // the portable cluster size
constexpr size_t kSeqSmall = static_cast<size_t>(kSeqSmallTiles) * kSeqTile;

struct SeqClusterSmem {
    SeqSmem t;
    double tsum, total, pa, pb;
    uint64_t R, start;
    uint32_t F;
    uint64_t s_R[kSeqSmallTiles + 1];
    uint32_t s_F[kSeqSmallTiles + 1];
    double s_x[kSeqBlock];
    uint64_t s_cr[kSeqBlock];
    uint64_t adj[kSeqTile];
    uint32_t pos[kSeqTile];
    uint16_t bex[kSeqTile];
};

// the block's dynamic shared memory, with a's lists in it
__device__ __forceinline__ SeqClusterSmem &seq_cluster_smem(SeqArgs &a)
{
    extern __shared__ __align__(16) unsigned char smem[];
    SeqClusterSmem &S = *reinterpret_cast<SeqClusterSmem *>(smem);
    a.adj = S.adj;
    a.pos = S.pos;
    a.bex = S.bex;
    return S;
}

// The exact left-to-right sum of the cluster's values (v: the block's tile,
// striped), in every thread; the tile's starting sum and breakpoints stay in
// S.  a.adj, a.pos and a.bex point at S's lists.
__device__ __forceinline__ double seq_cluster_total(
    const cooperative_groups::cluster_group &cl, const SeqArgs &a,
    const double (&v)[kSeqItems], SeqClusterSmem &S)
{
    const uint32_t tile = cl.block_rank(), nc = cl.num_blocks();
    const uint32_t lane = threadIdx.x & 31;
    const double ts = seq_tile_sum(v, a.allow_inf, a.err, S.t, 0);
    if (threadIdx.x == 0) {
        S.tsum = ts;
        S.t.rR = 0;
        S.t.rF = 0;
    }
    cl.sync();
    if (threadIdx.x < 32) {
        const double d = lane < nc ? cl.map_shared_rank(&S, lane)->tsum : 0.0;
        double run = 0;
        for (uint32_t q = 0; q <= tile; ++q) {
            if (q == tile && lane == 0)
                S.pa = run;
            run += __shfl_sync(0xFFFFFFFFu, d, q);
        }
        if (lane == 0)
            S.pb = run;
    }
    __syncthreads();
    uint64_t R = 0;
    uint32_t F = 0;
    seq_classify_tile(a, tile, 0, v, S.pa, S.pb, S.t, 0, R, F);
    if (threadIdx.x == 0) {
        S.R = R;
        S.F = F;
    }
    cl.sync();
    if (tile == 0) { // walk the breakpoints, as seq_fixup does
        if (threadIdx.x < 32) {
            const SeqClusterSmem *B = cl.map_shared_rank(&S, min(lane, nc - 1));
            const uint64_t r = warp_incl_any(lane < nc ? B->R : 0ull, OpAdd());
            const uint32_t f = warp_incl_any(lane < nc ? B->F : 0u, OpAdd());
            if (lane < nc) {
                S.s_R[lane + 1] = r;
                S.s_F[lane + 1] = f;
            }
            if (lane == 0) {
                S.s_R[0] = 0;
                S.s_F[0] = 0;
            }
        }
        __syncthreads();
        const uint32_t nbk = S.s_F[nc];
        uint64_t sum = 0, crprev = 0;
        for (uint32_t c0 = 0; c0 < nbk; c0 += kSeqBlock) {
            const uint32_t g = c0 + threadIdx.x;
            SeqClusterSmem *B = &S;
            uint32_t k = 0;
            uint64_t lr = 0;
            if (g < nbk) {
                const uint32_t b = seq_range_of(S.s_F, nc, g);
                B = cl.map_shared_rank(&S, b);
                k = g - S.s_F[b];
                lr = B->adj[k];
                S.s_cr[threadIdx.x] = S.s_R[b] + lr;
                // the element from the staging rows of its block
                const uint32_t e = B->pos[k] - b * kSeqTile;
                S.s_x[threadIdx.x] = *reinterpret_cast<const double *>(
                    B->t.row[e >> 8] + ((e & 255) >> 3) * 80 + (e & 7) * 8);
            }
            __syncthreads();
            if (threadIdx.x == 0)
                seq_walk(S.s_x, S.s_cr, min(nbk - c0, kSeqBlock + 0u), sum,
                    crprev, a.err);
            __syncthreads();
            if (g < nbk) {
                const uint64_t s = S.s_cr[threadIdx.x];
                B->adj[k] = s - lr;
                B->bex[k] = static_cast<uint16_t>(s >> 52);
            }
            __syncthreads();
        }
        if (threadIdx.x <= nc) {
            const uint32_t b = threadIdx.x, g = S.s_F[b];
            uint64_t s = 0;
            if (g > 0) {
                const uint32_t q = seq_range_of(S.s_F, nc, g - 1);
                s = cl.map_shared_rank(&S, q)->adj[g - 1 - S.s_F[q]] +
                    (S.s_R[b] - S.s_R[q]);
            } else if (S.s_R[b] != 0) {
                atomicOr(a.err, DEV_ERR_INTERNAL); // a first sum is listed
            }
            if (b < nc)
                cl.map_shared_rank(&S, b)->start = s;
            else
                for (uint32_t q = 0; q < nc; ++q)
                    cl.map_shared_rank(&S, q)->total = from_dbits(s);
        }
    }
    cl.sync();
    return S.total;
}

// sums of up to kSeqSmall elements: a.total and a.inv, and the running sums
// to out unless it is SeqNoOut
struct SeqNoOut {
};

template <class Load, class Out>
__global__ void __launch_bounds__(kSeqBlock) k_seq_small(
    SeqArgs a, const Load load, const Out out)
{
    pdl_begin();
    namespace cg = cooperative_groups;
    const cg::cluster_group cl = cg::this_cluster();
    SeqClusterSmem &S = seq_cluster_smem(a);
    const uint32_t tile = cl.block_rank();
    double v[kSeqItems];
    seq_load(load, tile, a.n, v);
    const double total = seq_cluster_total(cl, a, v, S);
    if (tile == 0 && threadIdx.x == 0) {
        if (a.total)
            *a.total = total;
        if (a.inv)
            *a.inv = 1.0 / total;
    }
    if constexpr (!std::is_same<Out, SeqNoOut>::value)
        seq_out_tile(a, tile, v, S.start,
            static_cast<uint32_t>(S.start >> 52), 0, 0, S.F, S.t, 1, out);
}

// ------------------------------------------------------------- functors

struct SeqLoad {
    const double *x;
    __device__ __forceinline__ double operator()(uint32_t i) const
    {
        return x[i];
    }
    __device__ __forceinline__ const double *at(uint32_t i) const
    {
        return x + i;
    }
};

// stores the prefix sums
struct SeqStore {
    double *p;
    uint32_t n;
    __device__ __forceinline__ void prefetch(double, uint32_t) const {}
    __device__ __forceinline__ void operator()(uint32_t tile, uint32_t,
        const double (&s)[kSeqItems], double, SeqSmem &sh) const
    {
        double v[kSeqItems];
        seq_to_striped(sh.row[threadIdx.x >> 5], s, v);
#pragma unroll
        for (int k = 0; k < kSeqItems; ++k) {
            const uint32_t i = seq_striped(tile, k);
            if (i < n)
                p[i] = v[k];
        }
    }
};

// ----------------------------------------------------------------- host

// A zeroed error word followed by the sums' two tickets (which every pass
// leaves zero) and words of the caller's, kErrWords in all; null on failure.
constexpr int kErrWords = 8;
uint32_t *new_err(Scratch &scratch, cudaStream_t st);

// The buffers for sums of n (1 <= n < 2^31) terms from one scratch
// allocation; err comes from new_err.
int seq_args(size_t n, uint32_t *err, bool allow_inf, Scratch &scratch,
    SeqArgs *a);

// A kernel of one cluster with a tile per block (a.n <= kSeqSmall).
template <class... Params, class... Args>
int seq_cluster_launch(void (*kernel)(SeqArgs, Params...), const SeqArgs &a,
    cudaStream_t st, const Args &...args)
{
    // the shared memory limit is a property of the kernel on each device
    VSMC_CUDA_TRY(cudaFuncSetAttribute(kernel,
        cudaFuncAttributeMaxDynamicSharedMemorySize,
        static_cast<int>(sizeof(SeqClusterSmem))));
    uint32_t c = 1;
    while (c < a.nt)
        c *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(c);
    cfg.blockDim = dim3(kSeqBlock);
    cfg.dynamicSmemBytes = sizeof(SeqClusterSmem);
    cfg.stream = st;
    cudaLaunchAttribute at[2] = {};
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = c;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1; // as launch_after
    cfg.attrs = at;
    cfg.numAttrs = 2;
    VSMC_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, a,
        static_cast<std::remove_cv_t<std::remove_reference_t<Params>>>(
            args)...));
    return VSMC_CUDA_OK;
}

template <class Load, class Out>
int seq_small(const SeqArgs &a, const Load &load, const Out &out,
    cudaStream_t st)
{
    return seq_cluster_launch(k_seq_small<Load, Out>, a, st, load, out);
}

// The sum by the large passes: sums sees every element once (it may compute
// and store them), load gives the same values afterwards.
template <class Sums, class Load>
int seq_total_large(const SeqArgs &a, const Sums &sums, const Load &load,
    cudaStream_t st)
{
    launch_after(k_seq_sums<Sums>, a.blocks, kSeqBlock, 0, st, a, sums);
    launch_after(k_seq_classify<Load>, a.blocks, kSeqBlock, 0, st, a, load);
    VSMC_CUDA_CHECK_LAUNCH();
    return VSMC_CUDA_OK;
}

// The sum of load(0 .. n - 1) into a.total / a.inv.
template <class Load>
int seq_total(const SeqArgs &a, const Load &load, cudaStream_t st)
{
    if (a.n <= kSeqSmall)
        return seq_small(a, load, SeqNoOut(), st);
    return seq_total_large(a, load, load, st);
}

// The same, and the running sums to out.
template <class Load, class Out>
int seq_scan(const SeqArgs &a, const Load &load, const Out &out,
    cudaStream_t st)
{
    if (a.n <= kSeqSmall)
        return seq_small(a, load, out, st);
    const int rc = seq_total(a, load, st);
    if (rc != VSMC_CUDA_OK)
        return rc;
    launch_after(k_seq_out<Load, Out>, a.blocks, kSeqBlock, 0, st, a, load,
        out);
    VSMC_CUDA_CHECK_LAUNCH();
    return VSMC_CUDA_OK;
}

// prefix (n doubles) and/or *total (device) of x[0..n), non-negative terms;
// allow_inf: +inf terms are summed as a sequential loop would (inf onward).
// Device error bits go to *err (DEV_ERR_NONFINITE for negative / NaN terms).
int seqsum_device(size_t n, const double *x, double *prefix, double *total,
    uint32_t *err, Scratch &scratch, cudaStream_t st, bool allow_inf = false);

// error bit: replication counts that do not sum to the slots
// (VSMC_CUDA_ERR_ARG)
enum : unsigned { DEV_ERR_COUNTS = 8u };

// status of a device error word
int err_status(uint32_t e);

// copy the device error word to the host (synchronizes) and map it to a
// status
int read_err(uint32_t *err_dev, cudaStream_t st, int *status);

} // namespace vsmc_cuda
