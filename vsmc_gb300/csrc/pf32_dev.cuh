// Device helpers of the FP32 filters (single and batched): log-sum-exp
// accumulation, the resampling engine's word stream, and exact counting of
// systematic / stratified uniforms against a 64-bit fixed-point CDF.
#pragma once

#include "common.cuh"
#include "pf32_types.cuh"

namespace vsmc_cuda
{

// ------------------------------------------------------- small utilities

// Both without branches, as LseMon's: the side with the larger max keeps its
// sums, the other's are scaled by e; what carries no weight adds nothing.
__device__ __forceinline__ void lse_push(float v, float &m, float &s, float &s2)
{
    const bool up = v > m;
    // -inf and NaN carry no weight
    const float e = v > -INFINITY ? __expf(up ? m - v : v - m) : 0.0f;
    s = fmaf(up ? s : 1.0f, e, up ? 1.0f : s);
    s2 = fmaf((up ? s2 : 1.0f) * e, e, up ? 1.0f : s2);
    m = up ? v : m;
}

// merge (m2, t, t2) into (m, s, s2): max, sum exp(v - m), sum exp(2(v - m))
__device__ __forceinline__ void lse_merge_f(
    float &m, float &s, float &s2, float m2, float t, float t2)
{
    const bool up = m2 > m;
    const float lo = up ? m : m2, hi = up ? m2 : m;
    const float e = lo > -INFINITY ? __expf(lo - hi) : 0.0f;
    s = fmaf(up ? s : t, e, up ? t : s);
    s2 = fmaf((up ? s2 : t2) * e, e, up ? t2 : s2);
    m = hi;
}

// 64 x 64 -> 128 bit product, compared as (hi, lo)
struct U128 {
    uint64_t hi, lo;
};

__device__ __forceinline__ U128 mul_u64(uint64_t a, uint64_t b)
{
    return {__umul64hi(a, b), a * b};
}

__device__ __forceinline__ bool le_u128(const U128 &a, const U128 &b)
{
    return a.hi < b.hi || (a.hi == b.hi && a.lo <= b.lo);
}

// word k (k >= 0) of the scalar stream of an engine at (key, ctr, index):
// gen(ctr + (index + k) / 4)[(index + k) % 4]
__device__ __forceinline__ uint32_t engine_word(const PfScalars &sc, uint64_t k)
{
    const uint64_t pos = static_cast<uint64_t>(sc.rindex) + k;
    uint32_t c[4] = {sc.rctr[0], sc.rctr[1], sc.rctr[2], sc.rctr[3]};
    ctr32_add(c, pos / 4);
    const u32x4 b = philox4x32_10(c[0], c[1], c[2], c[3], sc.rkey[0], sc.rkey[1]);
    const uint32_t i = static_cast<uint32_t>(pos % 4);
    return i == 0 ? b.x : (i == 1 ? b.y : (i == 2 ? b.z : b.w));
}

// advance the engine by k >= 1 words
__device__ __forceinline__ void engine_advance(PfScalars &sc, uint64_t k)
{
    if (k == 0)
        return;
    const uint64_t last = static_cast<uint64_t>(sc.rindex) + k - 1;
    uint32_t c[4] = {sc.rctr[0], sc.rctr[1], sc.rctr[2], sc.rctr[3]};
    ctr32_add(c, last / 4);
    for (int i = 0; i < 4; ++i)
        sc.rctr[i] = c[i];
    sc.rindex = static_cast<uint32_t>(last % 4) + 1;
}

// Counting uniforms against the fixed-point CDF.
//
// Uniform j is u_j = (j + a_j 2^-32) / N with a 32-bit word a_j.  With the
// integer CDF C_i and total Q, u_j <= C / Q  <=>  (j 2^32 + a_j) Q <= C N 2^32
// <=>  j Q + G_j <= C N  with G_j = ceil(a_j Q / 2^32) <= Q, since both sides
// are integers.  The counts follow from one exact floor((C N - G) / Q) per
// CDF value (below).
__device__ __forceinline__ uint64_t ceil_aq(uint32_t a, uint64_t Q)
{
    const uint64_t hi = __umul64hi(static_cast<uint64_t>(a), Q); // < 2^32
    const uint64_t lo = static_cast<uint64_t>(a) * Q;
    return ((hi << 32) | (lo >> 32)) + ((lo & 0xFFFFFFFFull) != 0 ? 1 : 0);
}

__device__ __forceinline__ U128 sub_u128(const U128 &a, const U128 &b)
{
    return {a.hi - b.hi - (a.lo < b.lo ? 1ull : 0ull), a.lo - b.lo};
}

// floor((hi 2^64 + lo) / d) for 0 < d, hi < d (the quotient fits 64 bits).
// Two estimates from below, each followed by the exact 128-bit remainder.
// The first is in FP64: y = y0 (2 - d y0) from the FP32 reciprocal y0, whose
// relative error e0 (below 2^-22.4) makes y low by e0^2, so with a factor
// 1 - 2^-50 for the roundings the estimate is never above the quotient and
// leaves a remainder below 2^20 d.  The second is in FP32, low by less than
// 2^-20 relative, and leaves less than 3 d; then unit steps (bounded;
// DEV_ERR_BOUND if ever exceeded).  FP64 latency is 64 cycles an operation:
// two FP64 divisions took 2000 cycles, this takes about 700.
__device__ __forceinline__ uint64_t div_u128_u64(
    uint64_t hi, uint64_t lo, uint64_t d, uint32_t &err)
{
    const float fd = __ull2float_rn(d);
    const float f0 = 1.0f / fd;
    const double y0 = static_cast<double>(f0);
    const double y =
        fma(y0, fma(-static_cast<double>(d), y0, 1.0), y0) * (1.0 - 0x1p-50);
    const double e =
        fma(static_cast<double>(hi), 0x1p64, static_cast<double>(lo)) * y;
    const uint64_t t = e < 0x1p64 ? static_cast<uint64_t>(e) : 0ull;
    U128 R = sub_u128(U128{hi, lo}, mul_u64(t, d));
    uint64_t quo = t;
    const float r =
        fmaf(__ull2float_rn(R.hi), 0x1p64f, __ull2float_rn(R.lo));
    const uint64_t t2 = static_cast<uint64_t>(
        __float2uint_rz(r * f0 * (1.0f - 0x1p-21f)));
    R = sub_u128(R, mul_u64(t2, d));
    quo += t2;
    for (int s = 0; s < 4 && (R.hi != 0 || R.lo >= d); ++s) {
        R = sub_u128(R, U128{0, d});
        ++quo;
    }
    if (R.hi != 0 || R.lo >= d)
        err |= DEV_ERR_BOUND;
    return quo;
}

// Counting by a fixed-point reciprocal (no division per particle).
//
// Usual case (qs > 0, totals Q >= 2^20 n): with s fraction bits chosen so
// that 2^s n < Q <= 2^(s+1) n (s at most 32), m = floor(2^(64+s) n / Q) and
// gs = floor(2^s G / Q).  H, the high half of C m from three 32 x 32-bit
// products (the low x low product and the carries of the dropped halves
// left out), is 0 to 3 below C m / 2^64, and C m / 2^64 is within 0.5 below
// 2^s C n / Q (C < 2^63); so B = H - gs lies in (V - 4.5, V + 1) for
// V = 2^s (C n - G) / Q.  floor((C n - G) / Q) is then B >> s unless B's low
// s bits are below 2 or within 6 of 2^s; there one exact test settles it.
//
// Any other total: z = clz(Q), rcp = floor((2^128 - 1) / (Q << z)) - 2^64,
// gam = floor(2^64 G / Q) (2^64 - 1 when G = Q).  For C < Q, with
// C' = C << z, H = C' + umulhi(C', rcp) lies in (T - 2, T] for
// T = 2^64 C / Q, so B = n H - gam lies in (V - 2n, V + 1] for
// V = 2^64 (C n - G) / Q, and floor(V / 2^64) is B's high word unless B's
// low word is 0 or within 4n + 8 of 2^64.
//
// G = ceil(a Q / 2^32) for the systematic word a; stratified: G = 0.  The
// exact test for a candidate m is m Q + G <= C n in 128 bits.
struct CdfRcp {
    uint64_t Q, G;
    uint64_t m, gs; // usual case
    uint64_t rcp, gam;
    uint64_t wlim; // 2^64 - (4 n + 8): low words at or above it are checked
    uint32_t s, fmask, z, n; // fmask = 2^s - 1 (32 bits)
};

__device__ __forceinline__ CdfRcp load_cdf_rcp(const PfScalars &sc, uint32_t n)
{
    CdfRcp p;
    p.Q = sc.Q;
    p.G = sc.qG;
    p.m = sc.qm;
    p.gs = sc.qgs;
    p.s = sc.qs;
    p.fmask = static_cast<uint32_t>((1ull << sc.qs) - 1ull);
    p.rcp = sc.qrcp;
    p.gam = sc.qgam;
    p.z = sc.qz;
    p.n = n;
    p.wlim = 0ull - (4ull * n + 8ull);
    return p;
}

// floor((C n - G) / Q) when the estimate k may be one off: low means the
// answer is k or k - 1, otherwise k or k + 1
static __device__ __noinline__ int64_t cdf_floor_near(
    uint64_t C, int64_t k, bool low, uint64_t Q, uint64_t G, uint32_t n)
{
    const int64_t m = low ? k : k + 1;
    bool ok = true; // m <= floor((C n - G) / Q), i.e. m Q + G <= C n
    if (m >= 0) {
        const U128 cn = mul_u64(C, static_cast<uint64_t>(n));
        U128 mq = mul_u64(static_cast<uint64_t>(m), Q);
        const uint64_t l = mq.lo + G;
        mq.hi += l < mq.lo ? 1ull : 0ull;
        mq.lo = l;
        ok = le_u128(mq, cn);
    }
    if (low)
        return ok ? k : k - 1;
    return ok ? k + 1 : k;
}

// B of the usual case: the truncated high product minus gs (two's
// complement: -2^s <= B < 2^63)
__device__ __forceinline__ uint64_t rcp_product(uint64_t C, const CdfRcp &p)
{
    const uint32_t c1 = static_cast<uint32_t>(C >> 32);
    const uint32_t c0 = static_cast<uint32_t>(C);
    const uint32_t m1 = static_cast<uint32_t>(p.m >> 32);
    const uint32_t m0 = static_cast<uint32_t>(p.m);
    const uint64_t H = static_cast<uint64_t>(c1) * m1 + __umulhi(c1, m0) +
        __umulhi(c0, m1);
    return H - p.gs;
}

// floor((C n - G) / Q) for C < Q (at least -1, below n).  Usual: the
// usual case's reciprocal (p.s > 0) is known to apply, so the loop that
// calls this holds one path only (the choice is made once per pass).
template <bool Usual>
__device__ __forceinline__ int64_t cdf_floor(uint64_t C, const CdfRcp &p)
{
    if (Usual) {
        const uint64_t B = rcp_product(C, p);
        const uint32_t bl = static_cast<uint32_t>(B);
        // B >> s (20 <= s <= 32): its low 32 bits are the signed answer
        const int32_t k = static_cast<int32_t>(
            __funnelshift_rc(bl, static_cast<uint32_t>(B >> 32), p.s));
        if (((bl + 6u) & p.fmask) < 8u)
            return cdf_floor_near(C, k, (bl & p.fmask) < 2u, p.Q, p.G, p.n);
        return k;
    }
    const uint64_t Cs = C << p.z;
    const uint64_t H = Cs + __umul64hi(Cs, p.rcp);
    const uint64_t al = H * static_cast<uint64_t>(p.n);
    const uint64_t ah = __umul64hi(H, static_cast<uint64_t>(p.n));
    const uint64_t f = al - p.gam;
    int64_t k = static_cast<int64_t>(ah - (al < p.gam ? 1ull : 0ull));
    if (f == 0 || f >= p.wlim)
        k = cdf_floor_near(C, k, f == 0, p.Q, p.G, p.n);
    return k;
}

// F(C): the systematic uniforms at or below C / Q, clamped to n
template <bool Usual>
__device__ __forceinline__ uint32_t sys_F(uint64_t C, const CdfRcp &p)
{
    if (C >= p.Q)
        return p.n;
    const int64_t F = cdf_floor<Usual>(C, p) + 1;
    return F < static_cast<int64_t>(p.n) ? static_cast<uint32_t>(F) : p.n;
}

// The resampling engine's position (the words the stratified uniforms use).
struct EnginePos {
    uint32_t key[2], ctr[4], index;
};

__device__ __forceinline__ EnginePos engine_pos(const PfScalars &sc)
{
    return {{sc.rkey[0], sc.rkey[1]},
        {sc.rctr[0], sc.rctr[1], sc.rctr[2], sc.rctr[3]}, sc.rindex};
}

// Philox block b of the engine's stream (word rindex + j is in block
// (rindex + j) / 4)
__device__ __forceinline__ uint4 engine_block(const EnginePos &e, uint32_t b)
{
    uint32_t c[4] = {e.ctr[0], e.ctr[1], e.ctr[2], e.ctr[3]};
    ctr32_add(c, b);
    const u32x4 v = philox4x32_10(c[0], c[1], c[2], c[3], e.key[0], e.key[1]);
    return make_uint4(v.x, v.y, v.z, v.w);
}

// the rare block past a warp's row (not inlined: off the common path's
// register budget)
static __device__ __noinline__ uint4 engine_block_far(
    const EnginePos &e, uint32_t b)
{
    return engine_block(e, b);
}

// Stratified: uniform j lies in [j / n, (j + 1) / n), so the uniforms at or
// below C / Q are every j < j* = floor(C n / Q), and j* itself when its own
// word passes: a_{j*} 2^-32 <= V - j*, V = C n / Q.  In the usual case the
// reciprocal's B gives both: j* = B >> s, and 2^s (V - j*) lies within -1 to
// 4.5 of B's low s bits, so the word's top s bits decide unless they are
// within a few units of them (StratPos::near; about 6 words in 2^s).  There,
// and in the general case, the exact test: G_{j*} = ceil(a_{j*} Q / 2^32) <=
// r = C n - j* Q (r < Q, so 64-bit wrapping arithmetic gives it exactly).
// The exact remainder and product took 30 instructions of every particle.
struct StratPos {
    uint32_t j;    // j*, n when C >= Q
    uint32_t frac; // usual case: B's low s bits; all ones when not usable
    bool near;     // usual case: frac does not decide alone
};

template <bool Usual>
__device__ __forceinline__ StratPos strat_pos(uint64_t C, const CdfRcp &p)
{
    StratPos q = {p.n, 0, true};
    if (C >= p.Q)
        return q;
    if (Usual) {
        const uint64_t B = rcp_product(C, p);
        const uint32_t bl = static_cast<uint32_t>(B);
        int32_t k = static_cast<int32_t>(
            __funnelshift_rc(bl, static_cast<uint32_t>(B >> 32), p.s));
        q.near = ((bl + 6u) & p.fmask) < 8u;
        if (q.near)
            k = static_cast<int32_t>(cdf_floor_near(
                C, k, (bl & p.fmask) < 2u, p.Q, p.G, p.n));
        q.frac = bl & p.fmask;
        q.j = static_cast<uint32_t>(k);
        return q;
    }
    q.j = static_cast<uint32_t>(cdf_floor<false>(C, p));
    return q;
}

// the exact test of word a for j < n (rare: off the common path's registers)
static __device__ __noinline__ bool strat_exact(
    uint64_t C, uint32_t j, uint32_t a, uint64_t Q, uint32_t n)
{
    const uint64_t r =
        C * static_cast<uint64_t>(n) - static_cast<uint64_t>(j) * Q;
    return ceil_aq(a, Q) <= r;
}

// F(C) from its position and word j* (for j < n)
template <bool Usual>
__device__ __forceinline__ uint32_t strat_count(
    uint64_t C, const StratPos &q, uint32_t a, const CdfRcp &p)
{
    if (!Usual)
        return q.j + (strat_exact(C, q.j, a, p.Q, p.n) ? 1u : 0u);
    const uint32_t as = a >> (32u - p.s); // p.s is 20 to 32
    bool pass = as <= q.frac - 2u; // frac is 2 or more unless near
    // frac - as from -4 to 1, or frac itself next to a whole number
    if (q.near || q.frac - as + 4u <= 5u)
        pass = strat_exact(C, q.j, a, p.Q, p.n);
    return q.j + (pass ? 1u : 0u);
}

// A warp's window of the engine's Philox blocks: blocks [lo, hi) of the
// stream are at row[b % kStratRow].  Blocks are generated 32 at a time, a
// lane each, ahead of their use: a group of 128 particles needs 33 or so
// blocks, and generating each group's own took two rounds of which the
// second had one or two lanes.
constexpr uint32_t kStratRow = 64; // blocks of a row (256 words)

struct StratWindow {
    uint32_t lo, hi;
};

// Blocks [b0, bl] into the window as far as it reaches (from b0 on).
__device__ __forceinline__ void strat_fill(const EnginePos &e, uint4 *row,
    StratWindow &w, uint32_t b0, uint32_t bl)
{
    const uint32_t lane = threadIdx.x & 31;
    if (b0 < w.lo || b0 > w.hi) { // not where the window ends: start anew
        w.lo = b0;
        w.hi = b0;
    }
    __syncwarp(); // the row's last readers
    while (w.hi <= bl && w.hi + 32 - b0 <= kStratRow) {
        const uint32_t b = w.hi + lane;
        row[b % kStratRow] = engine_block(e, b);
        w.hi += 32;
    }
    if (w.hi - w.lo > kStratRow)
        w.lo = w.hi - kStratRow;
    __syncwarp();
}

// word j of the uniforms, from the window or generated when outside it
__device__ __forceinline__ uint32_t strat_word(uint32_t j, const EnginePos &e,
    const uint4 *row, const StratWindow &w)
{
    const uint32_t pos = e.index + j;
    const uint32_t b = pos >> 2;
    uint32_t a;
    if (b - w.lo < w.hi - w.lo) {
        a = reinterpret_cast<const uint32_t *>(row)[pos % (4 * kStratRow)];
    } else {
        const uint4 v = engine_block_far(e, b);
        const uint32_t k = pos & 3u;
        a = k == 0 ? v.x : (k == 1 ? v.y : (k == 2 ? v.z : v.w));
    }
    return a;
}

// The per-event constants above, from the total Q (the same in every lane),
// by one warp: lane 0 divides for the reciprocal, lane 1 for the systematic
// word's term (one thread did both in turn), and lane 0 writes sc and has
// err.  A total of 0 or of 2^63 and more is not a valid integer CDF:
// DEV_ERR_NONFINITE, with constants that keep every later pass in range.
__device__ __forceinline__ void cdf_constants(
    PfScalars &sc, uint64_t Q, uint32_t n, bool sys, uint32_t &err)
{
    const uint32_t lane = threadIdx.x & 31;
    const bool bad = Q == 0 || (Q >> 63) != 0;
    const uint64_t G =
        sys && !bad ? ceil_aq(engine_word(sc, 0), Q) : 0ull;
    // the usual case's s: the largest s <= 32 with 2^s n < Q, if s >= 20;
    // the general reciprocal otherwise
    uint32_t s = 0;
    if (!bad) {
        // 2^s n < Q holds for s up to the difference of the bit lengths, or
        // one less
        const int up = __clz(static_cast<int>(n)) + 32 -
            __clzll(static_cast<long long>(Q));
        s = static_cast<uint32_t>(up < 0 ? 0 : (up > 32 ? 32 : up));
        if (s > 0 && (static_cast<uint64_t>(n) << s) >= Q)
            --s;
    }
    const bool usual = s >= 20;
    const uint32_t z = bad
        ? 0u
        : static_cast<uint32_t>(__clzll(static_cast<long long>(Q)));
    const uint64_t Qs = Q << z;
    uint64_t quo = 0;
    if (!bad && lane < 2) {
        uint64_t hi, lo, d;
        if (usual) {
            hi = lane == 0 ? static_cast<uint64_t>(n) << s : G >> (64 - s);
            lo = lane == 0 ? 0 : G << s;
            d = Q;
        } else {
            hi = lane == 0 ? ~Qs : G;
            lo = lane == 0 ? ~0ull : 0;
            d = lane == 0 ? Qs : Q;
        }
        if (hi < d) // G = Q in the general case: all ones below
            quo = div_u128_u64(hi, lo, d, err);
        else
            quo = ~0ull;
    }
    const uint64_t quo1 = __shfl_sync(0xFFFFFFFFu, quo, 1);
    err |= __shfl_sync(0xFFFFFFFFu, err, 1);
    if (bad)
        err |= DEV_ERR_NONFINITE;
    if (lane != 0)
        return;
    sc.Q = Q;
    sc.qG = G;
    sc.qs = usual ? s : 0;
    sc.qm = usual ? quo : 0;
    sc.qgs = usual ? quo1 : 0;
    sc.qz = usual || bad ? 0 : z;
    sc.qrcp = usual || bad ? 0 : quo;
    sc.qgam = usual || bad ? 0 : quo1;
}

// floor(w * 2^shift) for w = exp(lw - M) in [0, 1] and shift <= 63, in two
// 32-bit halves by float operations that are all exact: x = w 2^shift is
// w with its exponent moved; h = trunc(x 2^-32) is the high half; and
// x - h 2^32 (one fma) is the low half exactly, because it is x mod 2^32,
// which keeps at most x's 24 significant bits (or is x itself, below 2^32).
// Both halves then convert by truncation.  -inf and NaN give 0.
__device__ __forceinline__ uint64_t fixed_q(float lw, float M, uint32_t shift)
{
    const float w = fminf(__expf(lw - M), 1.0f);
    const float x = w * __uint_as_float((127u + shift) << 23);
    const float h = truncf(x * 0x1p-32f);
    const uint32_t hi = __float2uint_rz(h);
    const uint32_t lo = __float2uint_rz(fmaf(-h, 0x1p32f, x));
    const uint64_t q = (static_cast<uint64_t>(hi) << 32) | lo;
    return lw > -INFINITY ? q : 0ull;
}

// counts of slots i0..i0+3 below hi (-1 past hi)
__device__ __forceinline__ int4 load_rep4(
    const int32_t *rep, uint32_t i0, uint32_t hi)
{
    if (i0 + 3 < hi)
        return __ldcg(reinterpret_cast<const int4 *>(rep + i0));
    int4 v;
    v.x = i0 + 0 < hi ? rep[i0 + 0] : -1;
    v.y = i0 + 1 < hi ? rep[i0 + 1] : -1;
    v.z = i0 + 2 < hi ? rep[i0 + 2] : -1;
    v.w = i0 + 3 < hi ? rep[i0 + 3] : -1;
    return v;
}

// row values i0..i0+3 below hi (0 past hi); i0 is a multiple of 4
__device__ __forceinline__ float4 load_row4(
    const float *row, uint32_t i0, uint32_t hi)
{
    if (i0 + 3 < hi)
        return __ldcs(reinterpret_cast<const float4 *>(row + i0));
    float4 v;
    v.x = i0 + 0 < hi ? row[i0 + 0] : 0.0f;
    v.y = i0 + 1 < hi ? row[i0 + 1] : 0.0f;
    v.z = i0 + 2 < hi ? row[i0 + 2] : 0.0f;
    v.w = i0 + 3 < hi ? row[i0 + 3] : 0.0f;
    return v;
}

// Surplus runs of one warp's 128 particles.  A parent with r >= 2 copies
// keeps one in its own slot and its other r - 1 fill the next r - 1 empty
// slots in order, so the warp's parents own consecutive runs that together
// cover the warp's surplus ranks [W0, W0 + S) exactly.  The sources
// srcs[W0 .. W0 + S) are written in order from position p:
//   * when more than a chunk (kRunChunk ranks) is left and the run holding p
//     goes on for at least a chunk, the warp stores its parent up to the
//     run's end directly (32 consecutive ranks per store), so a parent with
//     a huge copy count costs its ranks' stores and nothing more;
//   * otherwise each parent marks the first rank of its run inside the
//     chunk [p, p + kRunChunk) in the warp's shared-memory row, a warp
//     max-scan over the chunk gives every rank its parent, and the warp
//     stores the chunk (coalesced).
// Warp-synchronous: called by every lane with warp-uniform W0 and S; rs / rl:
// the lane's runs (start rank, length; 0 for none).
constexpr uint32_t kRunChunk = 128;

__device__ __forceinline__ void write_surplus_runs(uint32_t *srcs,
    const uint32_t (&rs)[4], const uint32_t (&rl)[4], uint32_t i0,
    uint32_t W0, uint32_t S, uint32_t *shm, uint32_t &err)
{
    const uint32_t lane = threadIdx.x & 31;
    uint32_t p0 = 0;
    while (p0 < S) {
        // a run can cover a whole chunk only when more than a chunk is left
        // (the usual group, whose ranks fit one chunk, skips the search)
        if (S - p0 > kRunChunk) {
            // the run holding p0 (exactly one lane has it)
            uint32_t own_end = 0, own_par = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t b0 = rs[k] - W0;
                if (rl[k] != 0 && b0 <= p0 && p0 < b0 + rl[k]) {
                    own_end = b0 + rl[k];
                    own_par = i0 + k;
                }
            }
            const unsigned who = __ballot_sync(0xFFFFFFFFu, own_end != 0);
            if (who == 0) {
                err |= DEV_ERR_INTERNAL; // a rank no run covers
                return;
            }
            const int src = __ffs(who) - 1;
            const uint32_t end = __shfl_sync(0xFFFFFFFFu, own_end, src);
            const uint32_t par = __shfl_sync(0xFFFFFFFFu, own_par, src);
            const uint32_t stop = end < S ? end : S;
            if (stop - p0 >= kRunChunk) {
                for (uint32_t q = p0 + lane; q < stop; q += 32)
                    srcs[W0 + q] = par;
                p0 = stop;
                continue;
            }
        }
        reinterpret_cast<uint4 *>(shm)[lane] = make_uint4(0, 0, 0, 0);
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (rl[k] == 0)
                continue;
            const uint32_t b0 = rs[k] - W0, b1 = b0 + rl[k];
            if (b1 > p0 && b0 < p0 + kRunChunk)
                shm[(b0 > p0 ? b0 : p0) - p0] = i0 + k + 1;
        }
        __syncwarp();
        const uint4 m = reinterpret_cast<const uint4 *>(shm)[lane];
        uint32_t run[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
        for (int j = 1; j < 4; ++j)
            run[j] = max(run[j], run[j - 1]);
        uint32_t incl = run[3];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= static_cast<uint32_t>(o))
                incl = max(incl, y);
        }
        uint32_t before = __shfl_up_sync(0xFFFFFFFFu, incl, 1);
        if (lane == 0)
            before = 0;
        const uint32_t lim = S - p0 < kRunChunk ? S - p0 : kRunChunk;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t pos = 4 * lane + j;
            if (pos < lim) {
                const uint32_t o = max(run[j], before);
                if (o == 0)
                    err |= DEV_ERR_INTERNAL; // a rank no run covers
                srcs[W0 + p0 + pos] = o - 1;
            }
        }
        __syncwarp(); // the row is reused by the next chunk
        p0 += kRunChunk;
    }
}

// ------------------------------------------- the passes over one warp range

__device__ __forceinline__ uint64_t q_at(
    const Rs32Args &a, uint32_t i, float M)
{
    return a.q ? a.q[i] : fixed_q(a.lw[i], M, a.shift);
}

// log-weights i..i+3 (i a multiple of 4) below hi, -inf past it
__device__ __forceinline__ float4 load_lw4(
    const float *lw, uint32_t i, uint32_t hi)
{
    if (i + 3 < hi)
        return __ldcg(reinterpret_cast<const float4 *>(lw + i));
    float4 v = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
    if (i < hi)
        v.x = lw[i];
    if (i + 1 < hi)
        v.y = lw[i + 1];
    if (i + 2 < hi)
        v.z = lw[i + 2];
    return v;
}

// sum of q over [wlo, whi), in every lane of the warp
__device__ __forceinline__ uint64_t qsum_range(
    const Rs32Args &a, uint32_t wlo, uint32_t whi, float M)
{
    const uint32_t lane = threadIdx.x & 31;
    uint64_t acc = 0;
    constexpr int kG = 4;
    constexpr uint32_t kSpan = kG * 128;
    if (a.q == nullptr) {
        // groups of kG float4 per lane; the next group's loads are issued
        // before this group's weights, and a float4 past the range reads as
        // -inf (weight 0), so the range's last group needs no other path
        float4 v[kG], nv[kG];
#pragma unroll
        for (int h = 0; h < kG; ++h)
            v[h] = load_lw4(a.lw, wlo + h * 128 + lane * 4, whi);
        for (uint32_t base = wlo; base < whi; base += kSpan) {
#pragma unroll
            for (int h = 0; h < kG; ++h)
                nv[h] = load_lw4(a.lw, base + kSpan + h * 128 + lane * 4, whi);
#pragma unroll
            for (int h = 0; h < kG; ++h)
                acc += fixed_q(v[h].x, M, a.shift) +
                    fixed_q(v[h].y, M, a.shift) +
                    fixed_q(v[h].z, M, a.shift) + fixed_q(v[h].w, M, a.shift);
#pragma unroll
            for (int h = 0; h < kG; ++h)
                v[h] = nv[h];
        }
    } else {
        for (uint32_t base = wlo; base < whi; base += kSpan)
            for (int h = 0; h < kG; ++h) {
                const uint32_t i0 = base + h * 128 + lane * 4;
                for (uint32_t i = i0; i < whi && i < i0 + 4; ++i)
                    acc += a.q[i];
            }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        acc += __shfl_xor_sync(0xFFFFFFFFu, acc, o);
    return acc;
}

// Replication counts, one warp per warp range, no block barrier.  Particle
// i's count is F(C_i) - F(C_{i-1}) for the CDF C_i: exact 64-bit prefix sums
// (the range's offset from qsum, a warp scan per group of 128 particles).
// F(C), the uniforms at or below C / Q, comes from the fixed-point
// reciprocal of Q (cdf_floor): no division and no position carried from
// particle to particle.  Stratified also reads each particle's word a_{j*}
// from the warp's window of Philox blocks.  The range's empty slots and
// copies are added to empties and copies (per lane).

// One warp's range, carry the CDF before it; Usual picks the reciprocal's
// case for the whole pass.
template <bool Sys, bool Usual>
__device__ __forceinline__ void count_range(const Rs32Args &a,
    const CdfRcp &p, const EnginePos &e, uint4 *row, uint32_t wlo,
    uint32_t whi, uint64_t carry, uint32_t &empties, uint32_t &copies)
{
    const uint32_t lane = threadIdx.x & 31;
    const float M = static_cast<float>(a.sc->M);
    const bool checked = a.q != nullptr;
    const uint32_t n = a.n;
    uint32_t Fprev = 0;
    StratWindow win = {0, 0};
    if (wlo != 0 && wlo < whi) {
        if (Sys) {
            Fprev = sys_F<Usual>(carry, p);
        } else {
            const StratPos q = strat_pos<Usual>(carry, p);
            const uint32_t b = (e.index + q.j) >> 2;
            Fprev = n;
            if (q.j < n) { // the same in every lane
                strat_fill(e, row, win, b, b);
                Fprev = strat_count<Usual>(
                    carry, q, strat_word(q.j, e, row, win), p);
            }
        }
    }
    float4 nxt = make_float4(0, 0, 0, 0);
    if (!checked && wlo + lane * 4 + 3 < whi)
        nxt = __ldcg(reinterpret_cast<const float4 *>(a.lw + wlo + lane * 4));
    for (uint32_t base = wlo; base < whi; base += 128) {
        const uint32_t i0 = base + lane * 4;
        const float4 v = nxt;
        if (!checked && i0 + 128 + 3 < whi)
            nxt = __ldcg(reinterpret_cast<const float4 *>(a.lw + i0 + 128));
        uint64_t q[4];
        if (i0 + 3 < whi && !checked) {
            q[0] = fixed_q(v.x, M, a.shift);
            q[1] = fixed_q(v.y, M, a.shift);
            q[2] = fixed_q(v.z, M, a.shift);
            q[3] = fixed_q(v.w, M, a.shift);
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                q[k] = (i0 + k < whi) ? q_at(a, i0 + k, M) : 0;
        }
        uint64_t s[4];
        s[0] = q[0];
        s[1] = s[0] + q[1];
        s[2] = s[1] + q[2];
        s[3] = s[2] + q[3];
        const uint64_t incl = warp_inclusive_scan(s[3], OpAdd());
        const uint64_t tot = __shfl_sync(0xFFFFFFFFu, incl, 31);
        const uint64_t cb = carry + (incl - s[3]);
        uint32_t F[4];
        if (Sys) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                F[k] = i0 + k + 1 >= n ? n : sys_F<Usual>(cb + s[k], p);
        } else {
            StratPos sp[4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                sp[k] = strat_pos<Usual>(cb + s[k], p);
            // the group's words: j of lane 0's first .. of lane 31's last
            // (j = n needs none)
            uint32_t jv = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (sp[k].j < n)
                    jv = sp[k].j;
            const uint32_t jl = __reduce_min_sync(0xFFFFFFFFu, sp[0].j);
            const uint32_t jh = __reduce_max_sync(0xFFFFFFFFu, jv);
            if (jl < n)
                strat_fill(e, row, win, (e.index + jl) >> 2,
                    (e.index + (jh > jl ? jh : jl)) >> 2);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                F[k] = n;
                if (i0 + k + 1 < n && sp[k].j < n)
                    F[k] = strat_count<Usual>(cb + s[k], sp[k],
                        strat_word(sp[k].j, e, row, win), p);
            }
        }
        uint32_t Fl = __shfl_up_sync(0xFFFFFFFFu, F[3], 1);
        if (lane == 0)
            Fl = Fprev;
        int32_t r[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            r[k] = static_cast<int32_t>(F[k] - Fl);
            Fl = F[k];
        }
        if (i0 + 3 < whi) {
            *reinterpret_cast<int4 *>(a.rep + i0) =
                make_int4(r[0], r[1], r[2], r[3]);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                empties += r[k] == 0 ? 1u : 0u;
                copies += static_cast<uint32_t>(r[k]);
            }
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (i0 + k < whi) {
                    a.rep[i0 + k] = r[k];
                    empties += r[k] == 0 ? 1u : 0u;
                    copies += static_cast<uint32_t>(r[k]);
                }
        }
        carry += tot;
        Fprev = __shfl_sync(0xFFFFFFFFu, F[3], 31);
    }
}

// Slot assignment, one warp per warp range (no block barrier).  With
// c = copies before slot i and e = empty slots before i, the first surplus
// rank of i is c - (i - e) (every non-empty slot before i keeps one of its
// copies).  idx[i] = i for a parent (it keeps its slot), idx[i] = -(e + 1)
// for the e-th empty slot, and srcs[first surplus rank .. + r - 1) = i for a
// parent with r >= 2 copies: the reference's layout
// (resample/transform.hpp:116-133) in one pass over the counts.  Each range
// starts from its offsets (c, e) that the counting pass left in cpart /
// epart, and a warp scan of (copies, empties) carries them through its
// 128-particle groups.
// One warp's range from its offsets (copies and empty slots before it); row:
// kRunChunk words of the warp's; macc: the monitor's sums when asked for.
template <bool Mon>
__device__ __forceinline__ void assign_range(const Rs32Args &a, uint32_t wlo,
    uint32_t whi, uint32_t coff, uint32_t eoff, uint32_t etotal,
    uint32_t *row, float (&macc)[kMaxMonitorDim])
{
    const uint32_t lane = threadIdx.x & 31;
    // monitor of the resampled particles, sum_i rep_i x_{d,i}, when the
    // host asks for it right after resampling (mon_dim > 0); the rows, like
    // the counts, are loaded one group ahead
    const uint32_t md = Mon ? a.mon_dim : 0u;
    float4 mrow[kMaxMonitorDim], mnxt[kMaxMonitorDim];
#pragma unroll
    for (int d = 0; d < kMaxMonitorDim; ++d)
        mnxt[d] = static_cast<uint32_t>(d) < md
            ? load_row4(a.mon_state + d * a.stride, wlo + lane * 4, whi)
            : make_float4(0, 0, 0, 0);
    uint32_t err = 0;
    int4 nxt = load_rep4(a.rep, wlo + lane * 4, whi);
    for (uint32_t base = wlo; base < whi; base += 128) {
        const uint32_t i0 = base + lane * 4;
        const int4 cur = nxt;
        if (base + 128 < whi)
            nxt = load_rep4(a.rep, i0 + 128, whi);
#pragma unroll
        for (int d = 0; d < kMaxMonitorDim; ++d) {
            mrow[d] = mnxt[d];
            if (static_cast<uint32_t>(d) < md && base + 128 < whi)
                mnxt[d] = load_row4(a.mon_state + d * a.stride, i0 + 128, whi);
        }
        const int32_t r[4] = {cur.x, cur.y, cur.z, cur.w};
#pragma unroll
        for (int d = 0; d < kMaxMonitorDim; ++d)
            if (static_cast<uint32_t>(d) < md)
                macc[d] += static_cast<float>(max(r[0], 0)) * mrow[d].x +
                    static_cast<float>(max(r[1], 0)) * mrow[d].y +
                    static_cast<float>(max(r[2], 0)) * mrow[d].z +
                    static_cast<float>(max(r[3], 0)) * mrow[d].w;

        uint32_t tr = 0, te = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (r[k] >= 0) {
                tr += static_cast<uint32_t>(r[k]);
                te += r[k] == 0 ? 1u : 0u;
            }
        // (copies, empties) before each lane: one 32-bit scan of
        // copies * 256 + empties (a group has at most 128 empties) unless a
        // lane has 2^16 or more copies
        uint32_t c, e, tc, tn;
        if (__any_sync(0xFFFFFFFFu, tr >= (1u << 16))) {
            const uint64_t v = (static_cast<uint64_t>(tr) << 32) | te;
            const uint64_t incl = warp_inclusive_scan(v, OpAdd());
            const uint64_t tot = __shfl_sync(0xFFFFFFFFu, incl, 31);
            const uint64_t ex = incl - v;
            c = coff + static_cast<uint32_t>(ex >> 32);
            e = eoff + static_cast<uint32_t>(ex & 0xFFFFFFFFu);
            tc = static_cast<uint32_t>(tot >> 32);
            tn = static_cast<uint32_t>(tot & 0xFFFFFFFFu);
        } else {
            const uint32_t v = (tr << 8) | te;
            const uint32_t incl = warp_inclusive_scan(v, OpAdd());
            const uint32_t tot = __shfl_sync(0xFFFFFFFFu, incl, 31);
            const uint32_t ex = incl - v;
            c = coff + (ex >> 8);
            e = eoff + (ex & 0xFFu);
            tc = tot >> 8;
            tn = tot & 0xFFu;
        }
        const uint32_t c0 = c, e0 = e;
        int32_t out[4];
        uint32_t rs[4], rl[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t i = i0 + k;
            rs[k] = 0;
            rl[k] = 0;
            if (r[k] == 0) {
                out[k] = -static_cast<int32_t>(e) - 1;
                ++e;
            } else {
                out[k] = static_cast<int32_t>(i);
                if (r[k] >= 2) {
                    rs[k] = c - (i - e);
                    rl[k] = static_cast<uint32_t>(r[k]) - 1;
                }
            }
            if (r[k] > 0)
                c += static_cast<uint32_t>(r[k]);
        }
        // the group's surplus ranks: copies minus kept slots before its
        // first particle, and the sum of its runs
        {
            const uint32_t first = c0 - (i0 - e0);
            const uint32_t W0 = __shfl_sync(0xFFFFFFFFu, first, 0);
            const uint32_t Sw =
                __reduce_add_sync(0xFFFFFFFFu, rl[0] + rl[1] + rl[2] + rl[3]);
            if (Sw != 0) {
                if (Sw > etotal || W0 > etotal - Sw) {
                    err |= DEV_ERR_INTERNAL; // ranks past the empty slots
                } else {
                    write_surplus_runs(a.srcs, rs, rl, i0, W0, Sw, row, err);
                }
            }
        }
        if (i0 + 3 < whi) {
            *reinterpret_cast<int4 *>(a.idx + i0) =
                make_int4(out[0], out[1], out[2], out[3]);
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (r[k] >= 0)
                    a.idx[i0 + k] = out[k];
        }
        coff += tc;
        eoff += tn;
    }
    if (err)
        atomicOr(&a.sc->err, err);
}

// The engine past the words the scheme consumed: U01SequenceSystematic draws
// once in its constructor; U01SequenceStratified draws lazily up to the first
// uniform above the second-to-last cumulative weight
// (rng/u01_sequence.hpp:177-259, resample/transform.hpp:61-70)
__device__ __forceinline__ void scheme_words(const Rs32Args &a, PfScalars &sc)
{
    if (a.scheme == VSMC_CUDA_SYSTEMATIC) {
        engine_advance(sc, 1);
    } else if (a.n >= 2) {
        const uint32_t jf = a.n - static_cast<uint32_t>(a.rep[a.n - 1]);
        engine_advance(sc, jf < a.n ? jf + 1 : a.n);
    }
}

} // namespace vsmc_cuda
