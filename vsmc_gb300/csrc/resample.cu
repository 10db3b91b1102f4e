// Resampling transforms, schemes, particle copy, weights and the monitor mean
// on the device, with the reference's arithmetic.
//
// Cumulative weights and normalizing sums are the reference's left-to-right
// sums bit for bit (seqsum.cu).  Counting uniforms against the CDF follows the
// two-pointer loop of resample/transform.hpp:43-71: after particle i the loop
// has consumed every uniform before the first one above cdf_i, so with the
// prefix maximum pm_j of the uniforms, F(cdf_i) = #{j : pm_j <= cdf_i} and
// rep_i = F(cdf_i) - F(cdf_{i-1}); the last particle takes the rest.
#include "common.cuh"
#include "explog64.cuh"
#include "rng_device.cuh"
#include "scan.cuh"
#include "seqsum.cuh"
#include "resample_internal.cuh"

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>

namespace vsmc_cuda
{

namespace
{

constexpr int kB = 256;

int grid1(size_t n) { return grid_for(n ? n : 1, kB, 4, 8); }

#define GRID_LOOP(i, n)                                                       \
    for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; \
         i < (n); i += static_cast<size_t>(gridDim.x) * blockDim.x)

// ------------------------------------------------------------ elementwise

__global__ void k_fill_i32(size_t n, int *p, int v)
{
    GRID_LOOP(i, n) p[i] = v;
}

// counts without uniforms to compare: v for every particle, plus integ
__global__ void k_rep_trivial(size_t m, int v, int *rep, const int *integ)
{
    GRID_LOOP(i, m) rep[i] = v + (integ ? integ[i] : 0);
}

// max-scan key: NaN compares as "above everything", as the reference's
// `u <= accw` test is false for NaN
__device__ __forceinline__ double key_of(double u)
{
    return isnan(u) ? INFINITY : u;
}

struct LoadKey {
    const double *u;
    __device__ double operator()(size_t i) const { return key_of(u[i]); }
};

struct StoreD {
    double *p;
    __device__ void operator()(size_t i, double v) const { p[i] = v; }
};

// #{i < m : s_i < x} (s non-decreasing): the first i with s_i >= x
__device__ __forceinline__ size_t lower_count(
    const double *s, size_t m, double x)
{
    size_t lo = 0, hi = m;
    while (lo < hi) {
        const size_t mid = lo + (hi - lo) / 2;
        if (s[mid] < x)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// Order-preserving integer key of a double, so the running maximum of the
// uniforms and the counting compare integers (GB300's FP64 rate is a small
// fraction of its integer rate): keys order as the doubles do, -0 equals +0,
// and a NaN uniform sits above everything, as the two-pointer test
// `u <= accw` is false for it.
__device__ __forceinline__ long long okey(double u)
{
    const long long b = __double_as_longlong(u);
    const unsigned long long a =
        static_cast<unsigned long long>(b) & 0x7FFFFFFFFFFFFFFFull;
    if (a == 0)
        return 0; // +0 and -0
    if (a > 0x7FF0000000000000ull)
        return LLONG_MAX; // NaN
    return b >= 0 ? b : (b ^ LLONG_MAX);
}

// the key a CDF value is compared with: a NaN CDF value counts no uniform
__device__ __forceinline__ long long okey_cdf(double x)
{
    const unsigned long long a =
        static_cast<unsigned long long>(__double_as_longlong(x)) &
        0x7FFFFFFFFFFFFFFFull;
    return a > 0x7FF0000000000000ull ? LLONG_MIN : okey(x);
}

struct LoadOKey {
    const double *u;
    __device__ long long operator()(size_t i) const { return okey(u[i]); }
};

struct StoreK {
    long long *p;
    __device__ void operator()(size_t i, long long v) const { p[i] = v; }
};

struct OpMaxK {
    __device__ __forceinline__ long long operator()(long long a,
        long long b) const
    {
        return a < b ? b : a;
    }
};

// Keys of the uniforms for counting: the running maximum's keys (KeysMax),
// or, for uniforms known to be non-decreasing, non-negative and free of NaN,
// each uniform's own key (KeysOwn; the running maximum is then the sequence
// itself).
struct KeysMax {
    const long long *pmk;
    __device__ __forceinline__ long long operator[](size_t j) const
    {
        return pmk[j];
    }
    __device__ __forceinline__ const void *at(size_t j) const
    {
        return pmk + j;
    }
};

struct KeysOwn {
    const double *u;
    __device__ __forceinline__ long long operator[](size_t j) const
    {
        // okey of a non-negative, non-NaN double is its bit pattern
        return __double_as_longlong(u[j]);
    }
    __device__ __forceinline__ const void *at(size_t j) const { return u + j; }
};

// The first index j >= lo with pmk_j > x (hi if none), given that every
// j < lo has pmk_j <= x and pmk_hi > x or hi == n.
template <class Keys>
__device__ __forceinline__ size_t first_above(
    const Keys &pmk, size_t lo, size_t hi, long long x)
{
    while (lo < hi) {
        const size_t mid = lo + (hi - lo) / 2;
        if (pmk[mid] <= x)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// #{j < n : pmk_j <= x} by exponential search from a guess g <= n.
template <class Keys>
__device__ __forceinline__ size_t count_from(
    const Keys &pmk, size_t n, long long x, size_t g)
{
    size_t lo, hi;
    size_t step = 1;
    if (g < n && pmk[g] <= x) { // the answer is above g
        lo = g + 1;
        hi = n;
        while (lo < n) {
            const size_t probe = lo + step - 1;
            if (probe >= n)
                break;
            if (pmk[probe] > x) {
                hi = probe;
                break;
            }
            lo = probe + 1;
            step <<= 1;
        }
    } else { // the answer is at most g
        lo = 0;
        hi = g;
        while (step <= hi) {
            const size_t probe = hi - step;
            if (pmk[probe] <= x) {
                lo = probe + 1;
                break;
            }
            hi = probe;
            step <<= 1;
        }
    }
    return first_above(pmk, lo, hi, x);
}

// floor(c n) for c in [0, 1) from the bits of c (integer operations; only a
// starting guess, so the low bits of c are dropped); n for c >= 1, 0 for a
// negative c
__device__ __forceinline__ size_t guess_cn(double c, size_t n)
{
    const unsigned long long b =
        static_cast<unsigned long long>(__double_as_longlong(c));
    if (b >> 63)
        return 0;
    const int e = static_cast<int>(b >> 52) - 1023;
    if (e >= 0)
        return n;
    const int sh = 31 - e; // c n = (mant >> 21) n 2^(e - 31)
    if (sh >= 64)
        return 0;
    const unsigned long long m32 = ((b & ((1ull << 52) - 1)) | (1ull << 52)) >> 21;
    const unsigned long long g = (m32 * static_cast<unsigned long long>(n)) >> sh;
    return g < n ? static_cast<size_t>(g) : n;
}

// guess_cn for c >= 0: the high product of c's top 32 significant bits and n
__device__ __forceinline__ uint32_t guess_below(double c, uint32_t n)
{
    const uint32_t h = static_cast<uint32_t>(__double2hiint(c));
    const uint32_t l = static_cast<uint32_t>(__double2loint(c));
    const uint32_t ef = h >> 20;
    const uint32_t m = __funnelshift_l(l, h, 11) | 0x80000000u;
    return ef < 1023u ? __umulhi(m, n) >> min(1022u - ef, 31u) : n;
}

// The first index j >= lo with pmk_j > x, given that every j < lo has
// pmk_j <= x: exponential search upwards.
template <class Keys>
__device__ __forceinline__ size_t count_ahead(
    const Keys &pmk, size_t n, long long x, size_t lo)
{
    size_t hi = n, step = 1;
    while (lo < n) {
        const size_t probe = lo + step - 1;
        if (probe >= n)
            break;
        if (pmk[probe] > x) {
            hi = probe;
            break;
        }
        lo = probe + 1;
        step <<= 1;
    }
    return first_above(pmk, lo, hi, x);
}

// Replication counts straight from the running sums of the weights (an
// output functor of the sequential sum, so the CDF is never stored): with
// F_i = #{j < n : pmk_j <= key(cdf_i)} (n for the last particle, whose CDF
// value the loop never compares), rep_i = F_i - F_{i-1}, plus integ_i where
// the integer parts are given.
//   Near: stratified and systematic uniforms, u_j in [j / n, (j + 1) / n] up
//   to rounding.  The answer is floor(n cdf) or one more: eight guesses of a
//   thread are loaded together, then the neighbours that confirm them; a
//   search runs only where one does not.  Striped elements (a warp's lanes
//   consecutive), so each load touches a few neighbouring lines; blocked
//   ones touched 16 and the pass took 123 us at 2^24.
//   else: blocked elements, the thread's first count by exponential search
//   from n cdf, each next one upwards from the one before (for sorted
//   uniforms n cdf is off by about sqrt(n), the previous count by a few).
template <class Keys, bool Near>
struct SeqCount {
    Keys pmk;
    uint32_t m, n;
    int *rep;
    const int *integ; // may be null
    uint32_t *tail;   // the uniforms left to the last particle

    // line l of the uniforms that a tile starting at CDF value c compares
    __device__ __forceinline__ void prefetch(double c, uint32_t l) const
    {
        const uint32_t j = guess_below(c, n) + 16 * l;
        if (j < n)
            seq_prefetch(pmk.at(j));
    }

    __device__ __forceinline__ uint32_t search(double c) const
    {
        return static_cast<uint32_t>(
            count_from(pmk, n, okey_cdf(c), guess_cn(c, n)));
    }

    __device__ __forceinline__ int one(
        uint32_t i, uint32_t F, uint32_t &Fl) const
    {
        const uint32_t Fk = i + 1 < m ? F : n;
        int r = static_cast<int>(Fk - Fl);
        Fl = Fk;
        if (i + 1 == m)
            *tail = static_cast<uint32_t>(r);
        if (integ && i < m)
            r += integ[i];
        return r;
    }

    __device__ __forceinline__ void operator()(uint32_t tile, uint32_t i0,
        const double (&s)[kSeqItems], double sprev, SeqSmem &sh) const
    {
        const uint32_t lane = threadIdx.x & 31;
        if (Near) {
            double c[kSeqItems];
            seq_to_striped(sh.row[threadIdx.x >> 5], s, c);
            long long x[kSeqItems]; // keys of non-negative sums: their bits
            uint32_t F[kSeqItems];
            bool at[kSeqItems];
#pragma unroll
            for (int k = 0; k < kSeqItems; ++k) {
                x[k] = __double_as_longlong(c[k]);
                F[k] = guess_below(c[k], n);
            }
#pragma unroll
            for (int k = 0; k < kSeqItems; ++k)
                at[k] = F[k] < n && pmk[F[k]] <= x[k];
#pragma unroll
            for (int k = 0; k < kSeqItems; ++k) {
                // confirms g + 1 (the next uniform is above) or g (the one
                // before is not)
                const uint32_t g = F[k];
                const bool ok = at[k] ? g + 1 == n || pmk[g + 1] > x[k]
                                      : g == 0 || pmk[g - 1] <= x[k];
                F[k] = ok ? g + (at[k] ? 1u : 0u)
                          : static_cast<uint32_t>(count_from(pmk, n, x[k], g));
            }
            // the counts before the warp's first element, then row by row
            uint32_t Fw = i0 == 0 && lane == 0 ? 0u : search(sprev);
            Fw = __shfl_sync(0xFFFFFFFFu, Fw, 0);
#pragma unroll
            for (int k = 0; k < kSeqItems; ++k) {
                uint32_t Fl = __shfl_up_sync(0xFFFFFFFFu, F[k], 1);
                if (lane == 0)
                    Fl = Fw;
                Fw = __shfl_sync(0xFFFFFFFFu, F[k], 31);
                const uint32_t i = seq_striped(tile, k);
                const int r = one(i, F[k], Fl);
                if (i < m)
                    rep[i] = r;
            }
            return;
        }
        uint32_t F[kSeqItems];
        F[0] = search(s[0]);
#pragma unroll
        for (int k = 1; k < kSeqItems; ++k)
            F[k] = static_cast<uint32_t>(
                count_ahead(pmk, n, okey_cdf(s[k]), F[k - 1]));
        uint32_t Fl = __shfl_up_sync(0xFFFFFFFFu, F[kSeqItems - 1], 1);
        if (lane == 0)
            Fl = i0 == 0 ? 0u : search(sprev);
#pragma unroll
        for (int k = 0; k < kSeqItems; ++k) {
            const int r = one(i0 + k, F[k], Fl);
            if (i0 + k < m)
                rep[i0 + k] = r;
        }
    }
};

// the weights of all particles but the last, whose CDF value is not formed
struct SeqLoadCdf {
    const double *w;
    uint32_t last;
    __device__ __forceinline__ double operator()(uint32_t i) const
    {
        return i < last ? w[i] : 0.0;
    }
    __device__ __forceinline__ const double *at(uint32_t i) const
    {
        return w + i;
    }
};

__global__ void k_index_from_cdf(size_t m, size_t n, const double *cdf,
    const double *pm, int *idx)
{
    GRID_LOOP(j, n)
    idx[j] = static_cast<int>(lower_count(cdf, m - 1, pm[j]));
}

// ---------------------------------------------- uniforms from the engine
// word k of the scalar stream of (key, ctr, index): gen(ctr + (index+k)/4)
struct EngineState {
    uint32_t k0, k1;
    uint32_t c[4];
    uint32_t index;
};

__device__ __forceinline__ uint32_t stream_word(const EngineState &e, size_t k)
{
    const uint64_t pos = static_cast<uint64_t>(e.index) + k;
    uint32_t c[4] = {e.c[0], e.c[1], e.c[2], e.c[3]};
    ctr32_add(c, pos / 4);
    const u32x4 b = philox4x32_10(c[0], c[1], c[2], c[3], e.k0, e.k1);
    const uint32_t i = static_cast<uint32_t>(pos % 4);
    return i == 0 ? b.x : (i == 1 ? b.y : (i == 2 ? b.z : b.w));
}

// x * 2^-e rounded to the nearest double, ties to even, for a result in the
// normal range: x normalized to 64 bits, its low 11 bits rounded away and
// the double assembled from its bits, about 17 integer instructions (the
// integer conversion takes 16 cycles of an SM per warp, twice as many).
__device__ __forceinline__ double rne_scaled(uint64_t x, int e)
{
    const int lz = __clzll(static_cast<long long>(x));
    const uint64_t y = x << (lz & 63);
    const uint32_t lo = static_cast<uint32_t>(y);
    const uint64_t up = (lo & 0x7FFu) + ((lo >> 11) & 1u) > 0x400u ? 1u : 0u;
    // the leading bit of y >> 11 (and a carry out of the rounding) adds one
    // to the exponent field
    const uint64_t field = static_cast<uint64_t>(63 - lz - e + 1022) << 52;
    return x == 0 ? 0.0
                  : __longlong_as_double(
                        static_cast<long long>(field + (y >> 11) + up));
}

// four consecutive doubles to a 32-byte aligned place in one store (four
// 8-byte stores of a warp write each 32-byte sector four times over)
__device__ __forceinline__ void store4(double *p, const double (&v)[4])
{
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};"
                 :
                 : "l"(p), "d"(v[0]), "d"(v[1]), "d"(v[2]), "d"(v[3])
                 : "memory");
}

// fl(v delta) for a 32-bit v with one FP64 instruction: 2^52 + v from its
// bits, times delta, minus 2^52 delta (exact), rounded once.
__device__ __forceinline__ double mul_u32(
    uint32_t v, double delta, double minus52delta)
{
    return __fma_rn(
        __hiloint2double(0x43300000, static_cast<int>(v)), delta, minus52delta);
}

// U01SequenceStratified: u_j = U_j * delta + j * delta.  Word j is at
// stream position index + j; one Philox block gives the four words of
// positions 4b .. 4b + 3.  For n = 2^k (log2n = k, else -1) delta is exact,
// both products are exact scalings of U_j = w 2^-32 and j, and the one
// rounding is that of the sum: u_j = RNE(j 2^32 + w) 2^-(32 + k), formed in
// integers (rne_scaled).  Otherwise the FP64 arithmetic of the reference in
// three instructions.
//
// What is stored is the running maximum.  For n = 2^k that is u_j itself (a
// non-decreasing integer sequence rounded to nearest).  Otherwise, with
// eps = 2^-53, u_i <= (i + 1) delta (1 + 3 eps) and u_j >= j delta (1 - eps),
// so u_j is below no uniform but possibly u_{j-1}, and below that one only
// if U_{j-1} - U_j >= 1 - 4 (j + 2) eps, that is word j below 2^34 (n + 2)
// eps <= 2^12: there word j - 1 is drawn again and the larger uniform kept.
// u - first is 32-byte aligned, so a block's four uniforms are one store.
__global__ void k_stratified_seq(EngineState e, size_t n, int log2n, double *u)
{
    pdl_begin();
    const double delta = 1.0 / static_cast<double>(n);
    const double d32 = delta * 0x1p-32;
    const double m52 = -0x1p52 * delta, m20 = -0x1p20 * delta;
    auto form = [&](uint32_t w, uint32_t j) {
        return __dadd_rn(mul_u32(w, d32, m20), mul_u32(j, delta, m52));
    };
    const uint64_t first = e.index;
    const uint64_t nblk = (first + n + 3) / 4;
    GRID_LOOP(b, nblk)
    {
        uint32_t c[4] = {e.c[0], e.c[1], e.c[2], e.c[3]};
        ctr32_add(c, b);
        const u32x4 w = philox4x32_10(c[0], c[1], c[2], c[3], e.k0, e.k1);
        const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
        double v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            // wraps before the first word, whose values are not stored
            const uint32_t j =
                static_cast<uint32_t>(4 * static_cast<uint64_t>(b) + k - first);
            if (log2n >= 0) {
                v[k] = rne_scaled((static_cast<uint64_t>(j) << 32) | ws[k],
                    32 + log2n);
            } else {
                v[k] = form(ws[k], j);
                if (ws[k] < (1u << 13) && j > 0 && j < n)
                    v[k] = fmax(v[k], form(stream_word(e, j - 1), j - 1));
            }
        }
        const uint64_t p0 = 4 * static_cast<uint64_t>(b);
        if (p0 >= first && p0 + 4 - first <= n) {
            store4(u + (p0 - first), v);
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (p0 + k >= first && p0 + k - first < n)
                    u[p0 + k - first] = v[k];
        }
    }
}

// U01SequenceSystematic: u0 = U * delta, u_j = u0 + j * delta (for n = 2^k
// the same integer rounding with one word for every j); non-decreasing, as
// every operation is monotone in j
__global__ void k_systematic_seq(EngineState e, size_t n, int log2n, double *u)
{
    pdl_begin();
    const uint32_t w0 = stream_word(e, 0);
    if (log2n >= 0) {
        GRID_LOOP(j, n)
        u[j] = rne_scaled((static_cast<uint64_t>(j) << 32) | w0, 32 + log2n);
        return;
    }
    const double delta = 1.0 / static_cast<double>(n);
    const double u0 = __dmul_rn(u01_co_d(w0), delta);
    const double m52 = -0x1p52 * delta;
    GRID_LOOP(j, n)
    u[j] = __dadd_rn(u0, mul_u32(static_cast<uint32_t>(j), delta, m52));
}

// U01SequenceSorted terms: -log(U_j) / (n - j), summed left to right below
// (a Philox block's four words, as in k_stratified_seq).
__global__ void k_sorted_terms(EngineState e, size_t n, double *t)
{
    pdl_begin();
    const uint64_t first = e.index;
    const uint64_t nblk = (first + n + 3) / 4;
    GRID_LOOP(b, nblk)
    {
        uint32_t c[4] = {e.c[0], e.c[1], e.c[2], e.c[3]};
        ctr32_add(c, b);
        const u32x4 w = philox4x32_10(c[0], c[1], c[2], c[3], e.k0, e.k1);
        const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
        const uint64_t p0 = 4 * static_cast<uint64_t>(b);
        double v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            // (past either end: not stored)
            const uint64_t j = p0 + k - first;
            const uint32_t d = j < n ? static_cast<uint32_t>(n - j) : 1u;
            v[k] = ws[k] == 0 ? CUDART_INF : n64_neg_log_over(ws[k], d);
        }
        if (p0 >= first && p0 + 4 - first <= n) {
            store4(t + (p0 - first), v);
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (p0 + k >= first && p0 + k - first < n)
                    t[p0 + k - first] = v[k];
        }
    }
}

__global__ void __launch_bounds__(kB64) k_sorted_terms_arr(
    size_t n, const double *u01, double *t)
{
    GRID_LOOP(j, n) t[j] = -(log(u01[j]) / static_cast<double>(n - j));
}

// The sorted uniforms u_j = 1 - exp(lmax_j), lmax_j = -s_j, from the running
// sums s; Max: their running maximum, which the counts compare (exp's last bit
// could turn two neighbours around).  The maximum is found where it is needed,
// by the predecessors within 2^-50 (n64_sorted_max): the expected number of
// such pairs is 4.5 n^2 2^-53, 0.1 at n = 2^24 and 2 at 2^26.  A flag and one
// block that then walked all of u took 17 ms of a call's 18 at 2^24 whenever
// one pair was that near.
template <bool Max>
__global__ void k_sorted_finish(size_t n, const double *s, double *u)
{
    pdl_begin();
    GRID_LOOP(j, n)
    {
        const SortedUniform form;
        u[j] = Max ? n64_sorted_max(s, j, form) : form(s[j]);
    }
}

__global__ void k_stratified_arr(size_t n, const double *u01, double *out)
{
    const double delta = 1.0 / static_cast<double>(n);
    GRID_LOOP(i, n)
    out[i] = __dadd_rn(__dmul_rn(u01[i], delta),
        __dmul_rn(static_cast<double>(i), delta));
}

__global__ void k_systematic_terms(size_t n, double u01, double *t)
{
    const double delta = 1.0 / static_cast<double>(n);
    GRID_LOOP(i, n) t[i] = i == 0 ? __dmul_rn(u01, delta) : delta;
}

// --------------------------------------------------------------- residual

// A NaN, infinite or negative weight is reported and split as zero, so the
// integer parts stay a valid count.
__global__ void k_residual_split(size_t m, size_t n, const double *w,
    double *resid, int *integ, uint32_t *err)
{
    const double coeff = static_cast<double>(n);
    GRID_LOOP(i, m)
    {
        const double wi = w[i];
        if (!(wi >= 0.0) || isinf(wi)) {
            atomicOr(err, DEV_ERR_NONFINITE);
            resid[i] = 0.0;
            integ[i] = 0;
            continue;
        }
        const double x = __dmul_rn(coeff, wi);
        const double ip = trunc(fmin(x, 2147483647.0));
        resid[i] = x - ip; // modf: exact
        integ[i] = static_cast<int>(ip);
    }
}

__global__ void k_scale(size_t m, const double *inv, double *v)
{
    const double c = *inv;
    GRID_LOOP(i, m) v[i] = __dmul_rn(c, v[i]);
}

// ------------------------------------------------------------ rep -> index

struct I2 {
    int32_t a, b;
};

struct OpI2 {
    __device__ __forceinline__ I2 operator()(const I2 &x, const I2 &y) const
    {
        return {x.a + y.a, x.b + y.b};
    }
};

struct OpMaxI {
    __device__ __forceinline__ int32_t operator()(int32_t x, int32_t y) const
    {
        return x < y ? y : x;
    }
};

// (rep, 0) for m != n
struct LoadES {
    const int *rep;
    __device__ I2 operator()(size_t i) const { return {rep[i], 0}; }
};

struct StoreI2 {
    I2 *p;
    __device__ void operator()(size_t i, I2 v) const { p[i] = v; }
};

// marks: the first output slot of p gets p + 1
__global__ void k_marks(size_t m, const int *rep, const I2 *incl, int *marks,
    size_t nmarks, uint32_t *err)
{
    GRID_LOOP(p, m)
    {
        const int r = rep[p];
        if (r < 0) {
            atomicOr(err, DEV_ERR_INTERNAL);
        } else if (r > 0) {
            const int first = incl[p].a - r;
            if (first >= 0 && static_cast<size_t>(first) < nmarks)
                marks[first] = static_cast<int>(p) + 1;
            else
                atomicOr(err, DEV_ERR_INTERNAL);
        }
    }
}

struct LoadI {
    const int *p;
    __device__ int32_t operator()(size_t i) const { return p[i]; }
};

struct StoreI {
    int *p;
    __device__ void operator()(size_t i, int32_t v) const { p[i] = v; }
};

// int entries widened to 64 bits (sums of up to 2^31 counts of up to 2^31)
struct LoadIW {
    const int *p;
    __device__ long long operator()(size_t i) const { return p[i]; }
};

// keeps only the last value of a scan (the total)
struct StoreLastW {
    long long *p;
    size_t last;
    __device__ void operator()(size_t i, long long v) const
    {
        if (i == last)
            *p = v;
    }
};

// ---- rep -> index for m == n (resample/transform.hpp:116-133): a parent
// keeps its slot, the e-th empty slot takes the e-th surplus copy in parent
// order.  Tiles of 2048 counts (8 consecutive ones per thread), a range of
// consecutive tiles per block:
//   count   empty slots and surplus copies of each range; the last block
//           (its ticket; nothing waits) scans the ranges and checks that the
//           totals agree;
//   assign  a block scan gives every slot its ranks: idx = the slot, or
//           -(rank + 1) for an empty one, and srcs[rank] = the parent of each
//           surplus copy (a run of more than 8 by its whole warp);
//   decode  empty slots read their parent.
// Up to 16384 counts one cluster does all of it in one launch.
struct SlotArgs {
    uint32_t n, nt, blocks;
    const int *rep;
    int *idx;
    uint32_t *srcs; // n
    uint64_t *S;    // blocks + 1: surplus copies of the ranges, then prefixes
    uint32_t *E;    // blocks + 1: empty slots
    uint32_t *err;
};

struct ES {
    uint64_t s;
    uint32_t e, pad;
};

struct OpES {
    __device__ __forceinline__ ES operator()(const ES &x, const ES &y) const
    {
        return {x.s + y.s, x.e + y.e, 0u};
    }
};

// the thread's eight counts of a tile (1 past the end: neither empty nor
// surplus) and their sum; negative ones are reported
__device__ __forceinline__ ES slot_load(
    const SlotArgs &a, uint32_t tile, int (&r)[kSeqItems])
{
    const uint32_t i0 = tile * kSeqTile + threadIdx.x * kSeqItems;
    if (i0 + kSeqItems <= a.n &&
        (reinterpret_cast<uintptr_t>(a.rep) & 15) == 0) {
        const int4 p = *reinterpret_cast<const int4 *>(a.rep + i0);
        const int4 q = *reinterpret_cast<const int4 *>(a.rep + i0 + 4);
        r[0] = p.x;
        r[1] = p.y;
        r[2] = p.z;
        r[3] = p.w;
        r[4] = q.x;
        r[5] = q.y;
        r[6] = q.z;
        r[7] = q.w;
    } else {
#pragma unroll
        for (int k = 0; k < kSeqItems; ++k)
            r[k] = i0 + k < a.n ? a.rep[i0 + k] : 1;
    }
    ES t = {0, 0, 0};
    bool neg = false;
#pragma unroll
    for (int k = 0; k < kSeqItems; ++k) {
        t.e += r[k] == 0 ? 1u : 0u;
        t.s += r[k] > 1 ? static_cast<uint32_t>(r[k]) - 1u : 0u;
        neg |= r[k] < 0;
    }
    if (neg)
        atomicOr(a.err, DEV_ERR_INTERNAL);
    return t;
}

// Places the thread's slots from the ranks before it.  out: what an empty
// slot of rank e gets until its source is known.
__device__ __forceinline__ void slot_place(const SlotArgs &a, uint32_t tile,
    const int (&r)[kSeqItems], ES at)
{
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t i0 = tile * kSeqTile + threadIdx.x * kSeqItems;
    uint32_t s = static_cast<uint32_t>(at.s);
    uint32_t e = at.e;
    int o[kSeqItems];
#pragma unroll
    for (int k = 0; k < kSeqItems; ++k) {
        const uint32_t i = i0 + k;
        o[k] = r[k] == 0 ? -static_cast<int>(e) - 1 : static_cast<int>(i);
        e += r[k] == 0 ? 1u : 0u;
        const uint32_t len = r[k] > 1 ? static_cast<uint32_t>(r[k]) - 1u : 0u;
        if (len <= 8)
            for (uint32_t q = 0; q < len; ++q)
                a.srcs[s + q] = i;
        unsigned big = __ballot_sync(0xFFFFFFFFu, len > 8);
        while (big) {
            const int who = __ffs(big) - 1;
            big &= big - 1;
            const uint32_t s1 = __shfl_sync(0xFFFFFFFFu, s, who);
            const uint32_t n1 = __shfl_sync(0xFFFFFFFFu, len, who);
            const uint32_t p1 = __shfl_sync(0xFFFFFFFFu, i, who);
            for (uint32_t q = lane; q < n1; q += 32)
                a.srcs[s1 + q] = p1;
        }
        s += len;
    }
    if (i0 + kSeqItems <= a.n &&
        (reinterpret_cast<uintptr_t>(a.idx) & 15) == 0) {
        int4 *q = reinterpret_cast<int4 *>(a.idx + i0);
        q[0] = make_int4(o[0], o[1], o[2], o[3]);
        q[1] = make_int4(o[4], o[5], o[6], o[7]);
    } else {
#pragma unroll
        for (int k = 0; k < kSeqItems; ++k)
            if (i0 + k < a.n)
                a.idx[i0 + k] = o[k];
    }
}

__device__ __forceinline__ void slot_range(
    const SlotArgs &a, uint32_t &t0, uint32_t &t1)
{
    const uint64_t b = blockIdx.x;
    t0 = static_cast<uint32_t>(b * a.nt / a.blocks);
    t1 = static_cast<uint32_t>((b + 1) * a.nt / a.blocks);
}

__global__ void __launch_bounds__(kSeqBlock) k_slots_count(const SlotArgs a)
{
    pdl_begin();
    uint32_t t0, t1;
    slot_range(a, t0, t1);
    ES acc = {0, 0, 0};
    for (uint32_t t = t0; t < t1; ++t) {
        int r[kSeqItems];
        acc = OpES()(acc, slot_load(a, t, r));
    }
    ES tot;
    block_excl_any<ES, OpES, kSeqBlock>(acc, OpES(), ES{0, 0, 0}, &tot);
    __shared__ bool last;
    if (threadIdx.x == 0) {
        a.S[blockIdx.x] = tot.s;
        a.E[blockIdx.x] = tot.e;
        __threadfence();
        last = atomicAdd(a.err + kErrTicket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last)
        return;
    __threadfence();
    const uint32_t per = (a.blocks + kSeqBlock - 1) / kSeqBlock;
    const uint32_t b0 = min(a.blocks, threadIdx.x * per);
    const uint32_t b1 = min(a.blocks, b0 + per);
    ES sum = {0, 0, 0};
    for (uint32_t i = b0; i < b1; ++i) {
        sum.s += __ldcg(a.S + i);
        sum.e += __ldcg(a.E + i);
    }
    ES run = block_excl_any<ES, OpES, kSeqBlock>(
        sum, OpES(), ES{0, 0, 0}, &tot);
    for (uint32_t i = b0; i < b1; ++i) {
        const uint64_t s = __ldcg(a.S + i);
        const uint32_t e = __ldcg(a.E + i);
        a.S[i] = run.s;
        a.E[i] = run.e;
        run.s += s;
        run.e += e;
    }
    if (threadIdx.x == 0) {
        a.err[kErrTicket] = 0;
        if (tot.s != tot.e)
            atomicOr(a.err, DEV_ERR_COUNTS);
    }
}

__global__ void __launch_bounds__(kSeqBlock) k_slots_assign(const SlotArgs a)
{
    pdl_begin();
    if (*a.err & DEV_ERR_COUNTS)
        return;
    uint32_t t0, t1;
    slot_range(a, t0, t1);
    ES before = {a.S[blockIdx.x], a.E[blockIdx.x], 0u};
    for (uint32_t t = t0; t < t1; ++t) {
        int r[kSeqItems];
        const ES mine = slot_load(a, t, r);
        ES tot;
        const ES ex = block_excl_any<ES, OpES, kSeqBlock>(
            mine, OpES(), ES{0, 0, 0}, &tot);
        slot_place(a, t, r, OpES()(before, ex));
        before = OpES()(before, tot);
    }
}

__global__ void __launch_bounds__(kB) k_slots_decode(const SlotArgs a)
{
    pdl_begin();
    if (*a.err & DEV_ERR_COUNTS)
        return;
    GRID_LOOP(i, a.n)
    {
        const int v = a.idx[i];
        if (v < 0)
            a.idx[i] = static_cast<int>(a.srcs[-v - 1]);
    }
}

// all of it by one cluster (a.n <= kSeqSmall)
__global__ void __launch_bounds__(kSeqBlock) k_slots_small(
    SeqArgs, const SlotArgs a)
{
    pdl_begin();
    namespace cg = cooperative_groups;
    const cg::cluster_group cl = cg::this_cluster();
    __shared__ ES s_tot;
    const uint32_t tile = cl.block_rank(), nc = cl.num_blocks();
    int r[kSeqItems];
    const ES mine = slot_load(a, tile, r);
    ES tot;
    ES at = block_excl_any<ES, OpES, kSeqBlock>(
        mine, OpES(), ES{0, 0, 0}, &tot);
    if (threadIdx.x == 0)
        s_tot = tot;
    cl.sync();
    ES all = {0, 0, 0};
    for (uint32_t q = 0; q < nc; ++q) {
        const ES o = *cl.map_shared_rank(&s_tot, q);
        if (q < tile)
            at = OpES()(at, o);
        all = OpES()(all, o);
    }
    if (all.s == all.e)
        slot_place(a, tile, r, at);
    else if (threadIdx.x == 0)
        atomicOr(a.err, DEV_ERR_COUNTS);
    cl.sync(); // srcs written; no block's totals are read any more
    if (all.s != all.e)
        return;
    const uint32_t i0 = tile * kSeqTile + threadIdx.x * kSeqItems;
#pragma unroll
    for (int k = 0; k < kSeqItems; ++k)
        if (r[k] == 0 && i0 + k < a.n)
            a.idx[i0 + k] = static_cast<int>(
                __ldcg(a.srcs + (-a.idx[i0 + k] - 1)));
}

__global__ void k_index_flat(size_t total, const int *src, int *idx)
{
    GRID_LOOP(d, total) idx[d] = src[d] - 1;
}

__global__ void k_hist(size_t m, size_t n, const int *idx, int *rep,
    uint32_t *err)
{
    GRID_LOOP(i, n)
    {
        const int p = idx[i];
        if (p < 0 || static_cast<size_t>(p) >= m)
            atomicOr(err, DEV_ERR_INTERNAL);
        else
            atomicAdd(rep + p, 1);
    }
}

// --------------------------------------------------------------- copying

__global__ void k_check_fixed_points(size_t n, const int *idx, uint32_t *err)
{
    pdl_begin();
    GRID_LOOP(d, n)
    {
        const int s = idx[d];
        if (s < 0 || static_cast<size_t>(s) >= n || idx[s] != s)
            atomicOr(err, DEV_ERR_INTERNAL);
    }
}

template <typename T>
__global__ void k_copy_state(size_t n, size_t dim, size_t ld, const int *idx,
    T *state, const uint32_t *err)
{
    pdl_begin();
    if (*err)
        return;
    GRID_LOOP(d, n)
    {
        const size_t s = static_cast<size_t>(idx[d]);
        if (s == d)
            continue;
        // four rows' loads in flight together
        size_t r = 0;
        for (; r + 4 <= dim; r += 4) {
            T *p = state + r * ld;
            const T v0 = p[s], v1 = p[ld + s], v2 = p[2 * ld + s],
                    v3 = p[3 * ld + s];
            p[d] = v0;
            p[ld + d] = v1;
            p[2 * ld + d] = v2;
            p[3 * ld + d] = v3;
        }
        for (; r < dim; ++r)
            state[r * ld + d] = state[r * ld + s];
    }
}

// ---------------------------------------------------------------- weights

struct OpMaxD {
    __device__ __forceinline__ double operator()(double a, double b) const
    {
        return a < b ? b : a;
    }
};

// The largest log-weight into *key (zero before).  Add: the log-weights are
// log(W) + l first (add_log, weight.hpp:168-173), stored in W.  64-thread
// blocks, one integer atomic each.
template <bool Add>
__global__ void __launch_bounds__(kB64) k_lw_max(
    size_t n, const double *l, double *W, unsigned long long *key)
{
    pdl_begin();
    unsigned long long m = 0;
    GRID_LOOP(i, n)
    {
        double v = l[i];
        if (Add) {
            v = __dadd_rn(log_of_fraction(W[i]), v);
            W[i] = v;
        }
        m = max(m, max_key(v));
    }
    __shared__ unsigned long long sh[kB64 / 32 + 1];
    m = block_reduce(m, OpMax(), 0ull, sh);
    if (threadIdx.x == 0)
        atomicMax(key, m);
}

// W = exp(lw - max)  (post_set_log -> normalize(true), weight.hpp:202-229)
__global__ void __launch_bounds__(kB64) k_exp_shift(
    size_t n, const double *lw, const unsigned long long *key, double *W)
{
    pdl_begin();
    const double m = from_max_key(*key);
    GRID_LOOP(i, n) W[i] = exp_of_negative(lw[i] - m);
}

// the normalized weights, stored, and their squares as the terms to sum
struct ScaleSquare {
    const double *v;
    const double *inv;
    double *W;
    __device__ __forceinline__ double operator()(uint32_t i) const
    {
        const double w = __dmul_rn(*inv, v[i]);
        W[i] = w;
        return __dmul_rn(w, w);
    }
};

struct SquareLoad {
    const double *W;
    __device__ __forceinline__ double operator()(uint32_t i) const
    {
        return __dmul_rn(W[i], W[i]);
    }
};

// Weight::normalize (weight.hpp:208-229) of up to kSeqSmall weights by one
// cluster: both left-to-right sums with the weights in registers.
__global__ void __launch_bounds__(kSeqBlock) k_normalize_small(
    SeqArgs a, const double *v, double *W, double *ess)
{
    pdl_begin();
    namespace cg = cooperative_groups;
    const cg::cluster_group cl = cg::this_cluster();
    SeqClusterSmem &S = seq_cluster_smem(a);
    __shared__ double s_inv;
    const uint32_t tile = cl.block_rank();
    double w[kSeqItems];
    seq_load(SeqLoad{v}, tile, a.n, w);
    const double total = seq_cluster_total(cl, a, w, S);
    if (threadIdx.x == 0)
        s_inv = 1.0 / total;
    __syncthreads();
    const double inv = s_inv;
#pragma unroll
    for (int k = 0; k < kSeqItems; ++k) {
        const uint32_t i = seq_striped(tile, k);
        w[k] = __dmul_rn(inv, w[k]);
        if (i < a.n)
            W[i] = w[k];
        w[k] = __dmul_rn(w[k], w[k]);
    }
    const double sq = seq_cluster_total(cl, a, w, S);
    if (ess && tile == 0 && threadIdx.x == 0)
        *ess = 1.0 / sq;
}

__global__ void k_fill_d(size_t n, double *p, double v)
{
    GRID_LOOP(i, n) p[i] = v;
}

// ---------------------------------------------------------------- monitor

// Weighted sums of dim rows: per-block partials, four rows to a pass over
// the weights, then a block for each row's partials (one thread adding 304
// partials at 64 cycles of FP64 latency each took 21 us).
template <typename T>
__global__ void __launch_bounds__(kB) k_wsum(size_t n, size_t dim, size_t ld,
    const T *state, const double *W, double *part)
{
    pdl_begin();
    constexpr int kD = 4;
    __shared__ double sh[kB / 32 + 1];
    for (size_t d0 = 0; d0 < dim; d0 += kD) {
        const int nd = dim - d0 < kD ? static_cast<int>(dim - d0) : kD;
        double s[kD] = {};
        GRID_LOOP(i, n)
        {
            const double w = W[i];
#pragma unroll
            for (int d = 0; d < kD; ++d)
                if (d < nd)
                    s[d] += w * static_cast<double>(state[(d0 + d) * ld + i]);
        }
#pragma unroll
        for (int d = 0; d < kD; ++d)
            if (d < nd) {
                const double t = block_reduce(s[d], OpAdd(), 0.0, sh);
                if (threadIdx.x == 0)
                    part[(d0 + d) * gridDim.x + blockIdx.x] = t;
            }
    }
}

__global__ void __launch_bounds__(kB) k_wsum_final(
    int nb, const double *part, double *out)
{
    pdl_begin();
    __shared__ double sh[kB / 32 + 1];
    double s = 0;
    for (int b = threadIdx.x; b < nb; b += kB)
        s += part[static_cast<size_t>(blockIdx.x) * nb + b];
    s = block_reduce(s, OpAdd(), 0.0, sh);
    if (threadIdx.x == 0)
        out[blockIdx.x] = s;
}

EngineState engine_state(const vsmc_cuda_rng &r)
{
    EngineState e;
    e.k0 = static_cast<uint32_t>(r.key[0]);
    e.k1 = static_cast<uint32_t>(r.key[1]);
    for (int i = 0; i < 4; ++i)
        e.c[i] = static_cast<uint32_t>(r.ctr[i]);
    e.index = r.index;
    return e;
}

// advance the host engine by k words of the scalar stream
void engine_advance_host(vsmc_cuda_rng &r, uint64_t k)
{
    if (k == 0)
        return;
    const uint64_t last = static_cast<uint64_t>(r.index) + k - 1;
    uint32_t c[4] = {static_cast<uint32_t>(r.ctr[0]),
        static_cast<uint32_t>(r.ctr[1]), static_cast<uint32_t>(r.ctr[2]),
        static_cast<uint32_t>(r.ctr[3])};
    ctr32_add(c, last / 4);
    for (int i = 0; i < 4; ++i)
        r.ctr[i] = c[i];
    r.index = static_cast<uint32_t>(last % 4) + 1;
}

bool size_ok(size_t n) { return n < (size_t(1) << 31); }

} // namespace

// ------------------------------------------------------- internal entries

// rep for m weights against n uniforms u (device); integ added if non-null.
// The uniforms left to the last particle go to err[kErrTail] (m >= 2, n > 0).
int u01_rep_device(size_t m, size_t n, const double *w, const double *u,
    UniformOrder order, int *rep, const int *integ, uint32_t *err,
    Scratch &scratch, cudaStream_t st)
{
    if (m == 0)
        return VSMC_CUDA_OK;
    if (m == 1 || n == 0) {
        k_rep_trivial<<<grid1(m), kB, 0, st>>>(
            m, m == 1 ? static_cast<int>(n) : 0, rep, integ);
        VSMC_CUDA_CHECK_LAUNCH();
        return VSMC_CUDA_OK;
    }
    SeqArgs a;
    int rc = seq_args(m, err, false, scratch, &a);
    if (rc != VSMC_CUDA_OK)
        return rc;
    const uint32_t m32 = static_cast<uint32_t>(m);
    const uint32_t n32 = static_cast<uint32_t>(n);
    const SeqLoadCdf load{w, m32 - 1};
    a.total = nullptr;
    a.inv = nullptr;
    uint32_t *tail = err + kErrTail;
    if (order == UniformOrder::Near)
        return seq_scan(a, load,
            SeqCount<KeysOwn, true>{KeysOwn{u}, m32, n32, rep, integ, tail},
            st);
    if (order == UniformOrder::Sorted)
        return seq_scan(a, load,
            SeqCount<KeysOwn, false>{KeysOwn{u}, m32, n32, rep, integ, tail},
            st);
    long long *pmk = scratch.get<long long>(n);
    long long *pp = scratch.get<long long>(scan_parts(n));
    if (!pmk || !pp)
        return VSMC_CUDA_ERR_ALLOC;
    rc = device_scan(
        n, LoadOKey{u}, StoreK{pmk}, OpMaxK(), LLONG_MIN, pp, st);
    if (rc != VSMC_CUDA_OK)
        return rc;
    return seq_scan(a, load,
        SeqCount<KeysMax, false>{KeysMax{pmk}, m32, n32, rep, integ, tail},
        st);
}

static int rep_index_square(size_t n, const int *rep, int *idx, uint32_t *err,
    Scratch &scratch, cudaStream_t st)
{
    SlotArgs a = {};
    a.n = static_cast<uint32_t>(n);
    a.nt = static_cast<uint32_t>((n + kSeqTile - 1) / kSeqTile);
    a.rep = rep;
    a.idx = idx;
    a.err = err;
    a.srcs = scratch.get<uint32_t>(n);
    if (a.srcs == nullptr)
        return VSMC_CUDA_ERR_ALLOC;
    if (n <= kSeqSmall) {
        SeqArgs q = {};
        q.n = a.n;
        q.nt = a.nt;
        return seq_cluster_launch(k_slots_small, q, st, a);
    }
    a.blocks = static_cast<uint32_t>(grid_for(a.nt, 1, 1, kSeqOcc));
    a.S = scratch.get<uint64_t>(a.blocks + 1);
    a.E = scratch.get<uint32_t>(a.blocks + 1);
    if (!a.S || !a.E)
        return VSMC_CUDA_ERR_ALLOC;
    launch_after(k_slots_count, a.blocks, kSeqBlock, 0, st, a);
    launch_after(k_slots_assign, a.blocks, kSeqBlock, 0, st, a);
    launch_after(k_slots_decode, grid1(n), kB, 0, st, a);
    VSMC_CUDA_CHECK_LAUNCH();
    return VSMC_CUDA_OK;
}

int rep_index_device(size_t m, size_t n, const int *rep, int *idx,
    uint32_t *err, Scratch &scratch, cudaStream_t st)
{
    if (m == 0 || n == 0)
        return VSMC_CUDA_OK;
    if (m == n)
        return rep_index_square(n, rep, idx, err, scratch, st);
    I2 *incl = scratch.get<I2>(m);
    I2 *pp = scratch.get<I2>(scan_parts(m));
    if (!incl || !pp)
        return VSMC_CUDA_ERR_ALLOC;
    int rc = device_scan(
        m, LoadES{rep}, StoreI2{incl}, OpI2(), I2{0, 0}, pp, st);
    if (rc != VSMC_CUDA_OK)
        return rc;
    // the number of slots is needed on the host to size the scan
    I2 tot;
    VSMC_CUDA_TRY(cudaMemcpyAsync(
        &tot, incl + (m - 1), sizeof(I2), cudaMemcpyDeviceToHost, st));
    VSMC_CUDA_TRY(cudaStreamSynchronize(st));
    if (tot.a < 0 || static_cast<size_t>(tot.a) > n)
        return VSMC_CUDA_ERR_ARG;
    const size_t nmarks = static_cast<size_t>(tot.a);
    if (nmarks == 0)
        return VSMC_CUDA_OK;
    int *marks = scratch.get<int>(nmarks);
    int *srcs = scratch.get<int>(nmarks);
    int *pm = scratch.get<int>(scan_parts(nmarks));
    if (!marks || !srcs || !pm)
        return VSMC_CUDA_ERR_ALLOC;
    VSMC_CUDA_TRY(cudaMemsetAsync(marks, 0, sizeof(int) * nmarks, st));
    k_marks<<<grid1(m), kB, 0, st>>>(m, rep, incl, marks, nmarks, err);
    VSMC_CUDA_CHECK_LAUNCH();
    rc = device_scan(nmarks, LoadI{marks}, StoreI{srcs}, OpMaxI(), 0, pm, st);
    if (rc != VSMC_CUDA_OK)
        return rc;
    k_index_flat<<<grid1(nmarks), kB, 0, st>>>(nmarks, srcs, idx);
    VSMC_CUDA_CHECK_LAUNCH();
    return VSMC_CUDA_OK;
}

// residual split; *R_dev receives n - sum(integ) (device size_t)
int residual_device(size_t m, size_t n, const double *w, double *resid,
    int *integ, size_t *R_host, uint32_t *err, Scratch &scratch,
    cudaStream_t st)
{
    if (m == 0) {
        *R_host = n;
        return VSMC_CUDA_OK;
    }
    k_residual_split<<<grid1(m), kB, 0, st>>>(m, n, w, resid, integ, err);
    VSMC_CUDA_CHECK_LAUNCH();
    long long *isum = scratch.get<long long>(1);
    long long *pp = scratch.get<long long>(scan_parts(m));
    if (!isum || !pp)
        return VSMC_CUDA_ERR_ALLOC;
    SeqArgs a;
    int rc = seq_args(m, err, false, scratch, &a);
    if (rc != VSMC_CUDA_OK)
        return rc;
    rc = seq_total(a, SeqLoad{resid}, st);
    if (rc != VSMC_CUDA_OK)
        return rc;
    k_scale<<<grid1(m), kB, 0, st>>>(m, a.inv, resid);
    VSMC_CUDA_CHECK_LAUNCH();
    // the integer parts summed in 64 bits: unnormalized weights can push
    // the sum past 2^31, and a wrapped 32-bit sum could land back in [0, n]
    rc = device_scan(m, LoadIW{integ}, StoreLastW{isum, m - 1}, OpAdd(),
        0LL, pp, st);
    if (rc != VSMC_CUDA_OK)
        return rc;
    long long R = 0;
    uint32_t e = 0;
    VSMC_CUDA_TRY(cudaMemcpyAsync(
        &R, isum, sizeof(R), cudaMemcpyDeviceToHost, st));
    VSMC_CUDA_TRY(
        cudaMemcpyAsync(&e, err, sizeof(e), cudaMemcpyDeviceToHost, st));
    VSMC_CUDA_TRY(cudaStreamSynchronize(st));
    if (e & DEV_ERR_NONFINITE)
        return VSMC_CUDA_ERR_NONFINITE;
    // normalised weights give integer parts summing to at most n
    if (R < 0 || static_cast<unsigned long long>(R) > n)
        return VSMC_CUDA_ERR_ARG;
    *R_host = n - static_cast<size_t>(R);
    return VSMC_CUDA_OK;
}

int scheme_enqueue(size_t m, size_t n, const vsmc_cuda_rng &rng,
    const double *w, int *rep, int scheme, uint32_t *err, size_t *N_out,
    Scratch &scratch, cudaStream_t st)
{
    const bool residual = scheme >= VSMC_CUDA_RESIDUAL;
    const int base = residual ? scheme - VSMC_CUDA_RESIDUAL : scheme;
    const double *wt = w;
    int *integ = nullptr;
    size_t N = n;
    int rc;
    if (residual) {
        double *resid = scratch.get<double>(m);
        integ = scratch.get<int>(m);
        if (!resid || !integ)
            return VSMC_CUDA_ERR_ALLOC;
        rc = residual_device(m, n, w, resid, integ, &N, err, scratch, st);
        if (rc != VSMC_CUDA_OK)
            return rc;
        wt = resid;
    }
    *N_out = N;
    const EngineState es = engine_state(rng);
    double *u = scratch.get<double>(N + 4);
    if (u == nullptr)
        return VSMC_CUDA_ERR_ALLOC;
    u += es.index % 4; // the engine's blocks of four words 32-byte aligned
    // N = 2^k: the uniforms are formed in integers (exact, no FP64)
    int log2n = -1;
    if (N > 0 && (N & (N - 1)) == 0 && N <= (size_t(1) << 31)) {
        log2n = 0;
        while ((size_t(1) << log2n) < N)
            ++log2n;
    }
    UniformOrder order = UniformOrder::Near;
    if (N > 0) {
        if (base == VSMC_CUDA_STRATIFIED) {
            launch_after(k_stratified_seq, grid1(N), kB, 0, st, es, N, log2n,
                u);
        } else if (base == VSMC_CUDA_SYSTEMATIC) {
            launch_after(k_systematic_seq, grid1(N), kB, 0, st, es, N, log2n,
                u);
        } else {
            order = UniformOrder::Sorted;
            double *t = scratch.get<double>(N + 4);
            if (t == nullptr)
                return VSMC_CUDA_ERR_ALLOC;
            t += es.index % 4; // as u
            launch_after(k_sorted_terms, grid1(N), kB, 0, st, es, N, t);
            rc = seqsum_device(N, t, t, nullptr, err, scratch, st, true);
            if (rc != VSMC_CUDA_OK)
                return rc;
            launch_after(k_sorted_finish<true>, grid1(N), kB, 0, st, N, t, u);
        }
        VSMC_CUDA_CHECK_LAUNCH();
    }
    return u01_rep_device(m, N, wt, u, order, rep, integ, err, scratch, st);
}

void scheme_advance(
    vsmc_cuda_rng &rng, size_t m, size_t N, int scheme, uint32_t tail)
{
    // systematic: the sequence constructor draws once; the others draw
    // lazily, up to the first uniform above the second-to-last CDF value
    uint64_t words = 0;
    if (scheme == VSMC_CUDA_SYSTEMATIC ||
        scheme == VSMC_CUDA_RESIDUAL_SYSTEMATIC)
        words = 1;
    else if (m >= 2 && N > 0)
        words = std::min<uint64_t>(N - tail + 1, N);
    engine_advance_host(rng, words);
}

int scheme_device(size_t m, size_t n, vsmc_cuda_rng *rng, const double *w,
    int *rep, int scheme, Scratch &scratch, cudaStream_t st)
{
    uint32_t *err = new_err(scratch, st);
    if (err == nullptr)
        return VSMC_CUDA_ERR_ALLOC;
    size_t N = 0;
    const int rc =
        scheme_enqueue(m, n, *rng, w, rep, scheme, err, &N, scratch, st);
    if (rc != VSMC_CUDA_OK)
        return rc;
    uint32_t word[kErrWords] = {};
    VSMC_CUDA_TRY(cudaMemcpyAsync(
        word, err, sizeof(word), cudaMemcpyDeviceToHost, st));
    VSMC_CUDA_TRY(cudaStreamSynchronize(st));
    const int status = err_status(word[0]);
    if (status != VSMC_CUDA_OK)
        return status;
    scheme_advance(*rng, m, N, scheme, word[kErrTail]);
    return VSMC_CUDA_OK;
}

// Both sums of more than kSeqSmall weights: W = v / sum(v), *ess (may be
// null); a.total gets the first.
int weight_sums(SeqArgs a, const double *v, double *W, double *ess,
    cudaStream_t st)
{
    const int rc = seq_total(a, SeqLoad{v}, st);
    if (rc != VSMC_CUDA_OK)
        return rc;
    const ScaleSquare scale{v, a.inv, W};
    a.total = nullptr;
    a.inv = ess;
    return seq_total_large(a, scale, SquareLoad{W}, st);
}

// Weight::normalize: W = v / sum(v), ESS (weight.hpp:208-229); v may be W
int weight_normalize_device(size_t n, const double *v, double *W,
    double *ess_dev, uint32_t *err, Scratch &scratch, cudaStream_t st)
{
    SeqArgs a;
    int rc = seq_args(n, err, false, scratch, &a);
    if (rc != VSMC_CUDA_OK)
        return rc;
    if (n <= kSeqSmall)
        return seq_cluster_launch(k_normalize_small, a, st, v, W, ess_dev);
    return weight_sums(a, v, W, ess_dev, st);
}

// the running maximum's key, two words of new_err's
unsigned long long *max_word(uint32_t *err)
{
    return reinterpret_cast<unsigned long long *>(err + kErrMax);
}

int weight_set_log_device(size_t n, const double *lw, double *W,
    double *ess_dev, uint32_t *err, Scratch &scratch, cudaStream_t st)
{
    launch_after(k_lw_max<false>, grid64(n), kB64, 0, st, n, lw, nullptr,
        max_word(err));
    launch_after(k_exp_shift, grid64(n), kB64, 0, st, n, lw, max_word(err), W);
    VSMC_CUDA_CHECK_LAUNCH();
    return weight_normalize_device(n, W, W, ess_dev, err, scratch, st);
}

int weight_set_equal_device(size_t n, double *W, double *ess_dev,
    uint32_t *err, Scratch &scratch, cudaStream_t st)
{
    k_fill_d<<<grid1(n), kB, 0, st>>>(n, W, 1.0 / static_cast<double>(n));
    VSMC_CUDA_CHECK_LAUNCH();
    return weight_normalize_device(n, W, W, ess_dev, err, scratch, st);
}

int weight_add_log_device(size_t n, const double *l, double *W,
    double *ess_dev, uint32_t *err, Scratch &scratch, cudaStream_t st)
{
    launch_after(k_lw_max<true>, grid64(n), kB64, 0, st, n, l, W,
        max_word(err));
    launch_after(k_exp_shift, grid64(n), kB64, 0, st, n, W, max_word(err), W);
    VSMC_CUDA_CHECK_LAUNCH();
    return weight_normalize_device(n, W, W, ess_dev, err, scratch, st);
}

template <typename T>
int monitor_mean_device(size_t n, size_t dim, size_t ld, const T *state,
    const double *W, double *out, Scratch &scratch, cudaStream_t st)
{
    const int nb = grid_for(n, kB, 2, 2);
    double *part = scratch.get<double>(dim * nb);
    if (part == nullptr)
        return VSMC_CUDA_ERR_ALLOC;
    launch_after(k_wsum<T>, nb, kB, 0, st, n, dim, ld, state, W, part);
    if (dim)
        launch_after(k_wsum_final, static_cast<unsigned>(dim), kB, 0, st, nb,
            part, out);
    VSMC_CUDA_CHECK_LAUNCH();
    return VSMC_CUDA_OK;
}

template int monitor_mean_device<float>(size_t, size_t, size_t, const float *,
    const double *, double *, Scratch &, cudaStream_t);
template int monitor_mean_device<double>(size_t, size_t, size_t,
    const double *, const double *, double *, Scratch &, cudaStream_t);

template <typename T>
int state_copy_device(size_t n, size_t dim, size_t ld, const int *idx,
    T *state, uint32_t *err, cudaStream_t st)
{
    launch_after(k_check_fixed_points, grid1(n), kB, 0, st, n, idx, err);
    launch_after(k_copy_state<T>, grid1(n), kB, 0, st, n, dim, ld, idx, state,
        err);
    VSMC_CUDA_CHECK_LAUNCH();
    return VSMC_CUDA_OK;
}

template int state_copy_device<float>(
    size_t, size_t, size_t, const int *, float *, uint32_t *, cudaStream_t);
template int state_copy_device<double>(
    size_t, size_t, size_t, const int *, double *, uint32_t *, cudaStream_t);

} // namespace vsmc_cuda

using namespace vsmc_cuda;

namespace
{

// run `body(err, scratch)` with a fresh error word, then report it
template <typename F>
int with_err(void *stream, F body)
{
    cudaStream_t st = as_stream(stream);
    Scratch scratch(st);
    uint32_t *err = new_err(scratch, st);
    if (err == nullptr)
        return VSMC_CUDA_ERR_ALLOC;
    int rc = body(err, scratch, st);
    if (rc != VSMC_CUDA_OK)
        return rc;
    int status = VSMC_CUDA_OK;
    rc = read_err(err, st, &status);
    return rc != VSMC_CUDA_OK ? rc : status;
}

bool valid_philox(const vsmc_cuda_rng *r)
{
    return r != nullptr && r->kind == VSMC_CUDA_PHILOX4X32 && r->index >= 1 &&
        r->index <= 4;
}

} // namespace

extern "C" {

int vsmc_cuda_u01_sorted(size_t n, const double *u01, double *u01seq,
    void *stream)
{
    if ((u01 == nullptr || u01seq == nullptr) && n)
        return VSMC_CUDA_ERR_ARG;
    if (!size_ok(n))
        return VSMC_CUDA_ERR_SIZE;
    if (n == 0)
        return VSMC_CUDA_OK;
    return with_err(stream, [&](uint32_t *err, Scratch &sc, cudaStream_t st) -> int {
        double *t = sc.get<double>(n);
        if (t == nullptr)
            return static_cast<int>(VSMC_CUDA_ERR_ALLOC);
        k_sorted_terms_arr<<<grid64(n), kB64, 0, st>>>(n, u01, t);
        VSMC_CUDA_CHECK_LAUNCH();
        int rc = seqsum_device(n, t, t, nullptr, err, sc, st, true);
        if (rc != VSMC_CUDA_OK)
            return rc;
        launch_after(
            k_sorted_finish<false>, grid1(n), kB, 0, st, n, t, u01seq);
        VSMC_CUDA_CHECK_LAUNCH();
        return static_cast<int>(VSMC_CUDA_OK);
    });
}

int vsmc_cuda_u01_stratified(size_t n, const double *u01, double *u01seq,
    void *stream)
{
    if ((u01 == nullptr || u01seq == nullptr) && n)
        return VSMC_CUDA_ERR_ARG;
    if (!size_ok(n))
        return VSMC_CUDA_ERR_SIZE;
    if (n == 0)
        return VSMC_CUDA_OK;
    k_stratified_arr<<<grid1(n), kB, 0, as_stream(stream)>>>(n, u01, u01seq);
    VSMC_CUDA_CHECK_LAUNCH();
    return VSMC_CUDA_OK;
}

int vsmc_cuda_u01_systematic(size_t n, double u01, double *u01seq,
    void *stream)
{
    if (u01seq == nullptr && n)
        return VSMC_CUDA_ERR_ARG;
    if (!size_ok(n))
        return VSMC_CUDA_ERR_SIZE;
    if (n == 0)
        return VSMC_CUDA_OK;
    return with_err(stream, [&](uint32_t *err, Scratch &sc, cudaStream_t st) -> int {
        double *t = sc.get<double>(n);
        if (t == nullptr)
            return static_cast<int>(VSMC_CUDA_ERR_ALLOC);
        k_systematic_terms<<<grid1(n), kB, 0, st>>>(n, u01, t);
        VSMC_CUDA_CHECK_LAUNCH();
        return seqsum_device(n, t, u01seq, nullptr, err, sc, st);
    });
}

int vsmc_cuda_resample_trans_u01_rep(size_t m, size_t n, const double *weight,
    const double *u01, int *replication, void *stream)
{
    if ((m && (weight == nullptr || replication == nullptr)) ||
        (n && m > 1 && u01 == nullptr))
        return VSMC_CUDA_ERR_ARG;
    if (!size_ok(m) || !size_ok(n))
        return VSMC_CUDA_ERR_SIZE;
    return with_err(stream, [&](uint32_t *err, Scratch &sc, cudaStream_t st) -> int {
        return u01_rep_device(m, n, weight, u01, UniformOrder::Any,
            replication, nullptr, err, sc, st);
    });
}

int vsmc_cuda_resample_trans_u01_index(size_t m, size_t n,
    const double *weight, const double *u01, int *index, void *stream)
{
    if (m == 0 || n == 0)
        return VSMC_CUDA_OK;
    if (weight == nullptr || u01 == nullptr || index == nullptr)
        return VSMC_CUDA_ERR_ARG;
    if (!size_ok(m) || !size_ok(n))
        return VSMC_CUDA_ERR_SIZE;
    return with_err(stream, [&](uint32_t *err, Scratch &sc, cudaStream_t st) -> int {
        if (m == 1) {
            k_fill_i32<<<grid1(n), kB, 0, st>>>(n, index, 0);
            VSMC_CUDA_CHECK_LAUNCH();
            return static_cast<int>(VSMC_CUDA_OK);
        }
        double *cdf = sc.get<double>(m - 1);
        double *pm = sc.get<double>(n);
        double *pp = sc.get<double>(scan_parts(n));
        if (!cdf || !pm || !pp)
            return static_cast<int>(VSMC_CUDA_ERR_ALLOC);
        int rc = seqsum_device(m - 1, weight, cdf, nullptr, err, sc, st);
        if (rc != VSMC_CUDA_OK)
            return rc;
        rc = device_scan(
            n, LoadKey{u01}, StoreD{pm}, OpMaxD(), -static_cast<double>(INFINITY), pp, st);
        if (rc != VSMC_CUDA_OK)
            return rc;
        k_index_from_cdf<<<grid1(n), kB, 0, st>>>(m, n, cdf, pm, index);
        VSMC_CUDA_CHECK_LAUNCH();
        return static_cast<int>(VSMC_CUDA_OK);
    });
}

int vsmc_cuda_resample_trans_rep_index(size_t m, size_t n,
    const int *replication, int *index, void *stream)
{
    if (m == 0 || n == 0)
        return VSMC_CUDA_OK;
    if (replication == nullptr || index == nullptr)
        return VSMC_CUDA_ERR_ARG;
    if (!size_ok(m) || !size_ok(n))
        return VSMC_CUDA_ERR_SIZE;
    return with_err(stream, [&](uint32_t *err, Scratch &sc, cudaStream_t st) -> int {
        return rep_index_device(m, n, replication, index, err, sc, st);
    });
}

int vsmc_cuda_resample_trans_index_rep(size_t m, size_t n, const int *index,
    int *replication, void *stream)
{
    if (m == 0 || n == 0)
        return VSMC_CUDA_OK;
    if (replication == nullptr || index == nullptr)
        return VSMC_CUDA_ERR_ARG;
    if (!size_ok(m) || !size_ok(n))
        return VSMC_CUDA_ERR_SIZE;
    return with_err(stream, [&](uint32_t *err, Scratch &sc, cudaStream_t st) -> int {
        (void)sc;
        VSMC_CUDA_TRY(cudaMemsetAsync(replication, 0, sizeof(int) * m, st));
        k_hist<<<grid1(n), kB, 0, st>>>(m, n, index, replication, err);
        VSMC_CUDA_CHECK_LAUNCH();
        return static_cast<int>(VSMC_CUDA_OK);
    });
}

int vsmc_cuda_resample_trans_residual(size_t m, size_t n,
    const double *weight, double *resid, int *integ, size_t *r_host,
    void *stream)
{
    if (r_host == nullptr ||
        (m && (weight == nullptr || resid == nullptr || integ == nullptr)))
        return VSMC_CUDA_ERR_ARG;
    if (!size_ok(m) || !size_ok(n))
        return VSMC_CUDA_ERR_SIZE;
    return with_err(stream, [&](uint32_t *err, Scratch &sc, cudaStream_t st) -> int {
        return residual_device(m, n, weight, resid, integ, r_host, err, sc, st);
    });
}

int vsmc_cuda_resample(size_t m, size_t n, vsmc_cuda_rng *rng,
    const double *weight, int *replication, int scheme, void *stream)
{
    if (!valid_philox(rng) || scheme < VSMC_CUDA_MULTINOMIAL ||
        scheme > VSMC_CUDA_RESIDUAL_SYSTEMATIC ||
        (m && (weight == nullptr || replication == nullptr)))
        return VSMC_CUDA_ERR_ARG;
    if (!size_ok(m) || !size_ok(n))
        return VSMC_CUDA_ERR_SIZE;
    cudaStream_t st = as_stream(stream);
    Scratch scratch(st);
    return scheme_device(m, n, rng, weight, replication, scheme, scratch, st);
}

#define VSMC_CUDA_SCHEME_ENTRY(name, id)                                      \
    int vsmc_cuda_resample_##name(size_t m, size_t n, vsmc_cuda_rng *rng,     \
        const double *weight, int *replication, void *stream)                 \
    {                                                                         \
        return vsmc_cuda_resample(m, n, rng, weight, replication, id, stream); \
    }

VSMC_CUDA_SCHEME_ENTRY(multinomial, VSMC_CUDA_MULTINOMIAL)
VSMC_CUDA_SCHEME_ENTRY(stratified, VSMC_CUDA_STRATIFIED)
VSMC_CUDA_SCHEME_ENTRY(systematic, VSMC_CUDA_SYSTEMATIC)
VSMC_CUDA_SCHEME_ENTRY(residual, VSMC_CUDA_RESIDUAL)
VSMC_CUDA_SCHEME_ENTRY(residual_stratified, VSMC_CUDA_RESIDUAL_STRATIFIED)
VSMC_CUDA_SCHEME_ENTRY(residual_systematic, VSMC_CUDA_RESIDUAL_SYSTEMATIC)

int vsmc_cuda_state_copy_f32(size_t n, size_t dim, const int *index,
    float *state, void *stream)
{
    if (n && (index == nullptr || state == nullptr))
        return VSMC_CUDA_ERR_ARG;
    if (!size_ok(n))
        return VSMC_CUDA_ERR_SIZE;
    if (n == 0 || dim == 0)
        return VSMC_CUDA_OK;
    const int rc = with_err(stream, [&](uint32_t *err, Scratch &, cudaStream_t st) -> int {
        return state_copy_device<float>(n, dim, n, index, state, err, st);
    });
    return rc == VSMC_CUDA_ERR_INTERNAL ? VSMC_CUDA_ERR_ARG : rc;
}

int vsmc_cuda_state_copy_f64(size_t n, size_t dim, const int *index,
    double *state, void *stream)
{
    if (n && (index == nullptr || state == nullptr))
        return VSMC_CUDA_ERR_ARG;
    if (!size_ok(n))
        return VSMC_CUDA_ERR_SIZE;
    if (n == 0 || dim == 0)
        return VSMC_CUDA_OK;
    const int rc = with_err(stream, [&](uint32_t *err, Scratch &, cudaStream_t st) -> int {
        return state_copy_device<double>(n, dim, n, index, state, err, st);
    });
    return rc == VSMC_CUDA_ERR_INTERNAL ? VSMC_CUDA_ERR_ARG : rc;
}

int vsmc_cuda_weight_set(size_t n, const double *w, double *W,
    double *ess_dev, void *stream)
{
    if (n == 0)
        return VSMC_CUDA_OK;
    if (w == nullptr || W == nullptr)
        return VSMC_CUDA_ERR_ARG;
    if (!size_ok(n))
        return VSMC_CUDA_ERR_SIZE;
    return with_err(stream, [&](uint32_t *err, Scratch &sc, cudaStream_t st) -> int {
        return weight_normalize_device(n, w, W, ess_dev, err, sc, st);
    });
}

int vsmc_cuda_weight_set_log(size_t n, const double *lw, double *W,
    double *ess_dev, void *stream)
{
    if (n == 0)
        return VSMC_CUDA_OK;
    if (lw == nullptr || W == nullptr)
        return VSMC_CUDA_ERR_ARG;
    if (!size_ok(n))
        return VSMC_CUDA_ERR_SIZE;
    return with_err(stream, [&](uint32_t *err, Scratch &sc, cudaStream_t st) -> int {
        return weight_set_log_device(n, lw, W, ess_dev, err, sc, st);
    });
}

int vsmc_cuda_weight_add_log(size_t n, const double *l, double *W,
    double *ess_dev, void *stream)
{
    if (n == 0)
        return VSMC_CUDA_OK;
    if (l == nullptr || W == nullptr)
        return VSMC_CUDA_ERR_ARG;
    if (!size_ok(n))
        return VSMC_CUDA_ERR_SIZE;
    return with_err(stream, [&](uint32_t *err, Scratch &sc, cudaStream_t st) -> int {
        return weight_add_log_device(n, l, W, ess_dev, err, sc, st);
    });
}

int vsmc_cuda_weight_set_equal(size_t n, double *W, double *ess_dev,
    void *stream)
{
    if (n == 0)
        return VSMC_CUDA_OK;
    if (W == nullptr)
        return VSMC_CUDA_ERR_ARG;
    if (!size_ok(n))
        return VSMC_CUDA_ERR_SIZE;
    return with_err(stream, [&](uint32_t *err, Scratch &sc, cudaStream_t st) -> int {
        return weight_set_equal_device(n, W, ess_dev, err, sc, st);
    });
}

int vsmc_cuda_monitor_mean_f64(size_t n, size_t dim, const double *state,
    const double *W, double *out_dev, void *stream)
{
    if (state == nullptr || W == nullptr || out_dev == nullptr || dim > 32)
        return VSMC_CUDA_ERR_ARG;
    if (!size_ok(n) || n == 0)
        return VSMC_CUDA_ERR_SIZE;
    cudaStream_t st = as_stream(stream);
    Scratch sc(st);
    return monitor_mean_device<double>(n, dim, n, state, W, out_dev, sc, st);
}

int vsmc_cuda_monitor_mean_f32(size_t n, size_t dim, const float *state,
    const double *W, double *out_dev, void *stream)
{
    if (state == nullptr || W == nullptr || out_dev == nullptr || dim > 32)
        return VSMC_CUDA_ERR_ARG;
    if (!size_ok(n) || n == 0)
        return VSMC_CUDA_ERR_SIZE;
    cudaStream_t st = as_stream(stream);
    Scratch sc(st);
    return monitor_mean_device<float>(n, dim, n, state, W, out_dev, sc, st);
}

} // extern "C"
