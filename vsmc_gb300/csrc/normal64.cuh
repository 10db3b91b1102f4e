// Box-Muller in 64-bit integers: the radius sqrt(-2 ln u1) and the sine and
// cosine of 2 pi u2 of two uniforms given as 64-bit fractions, as FP64 values
// rounded once.
//
// A warp's FP64 instruction holds its SM's FP64 pipe for 19 clocks, an integer
// one for half a clock or one; the about 70 FP64 operations of log, sqrt and
// sincos a pair took 2^22 + 1 normals 307 us.  Uniforms are integers to begin
// with, so everything up to the three results is fixed point here, no FP64
// operation: 2^22 + 1 normals take 50 us.
//
// Roundings stay those of the FP64 sequence it replaces: -2 ln u1 and the
// angle (FP64 2 pi) u2 are rounded to 53 bits before the root and the sine
// and cosine of them are taken.  Each function is within 0.55 ulp (CUDA's: 1).
//
// Methods.  Logarithm: table-driven reduction (P. T. P. Tang, "Table-driven
// implementation of the logarithm function", ACM TOMS 16, 1990), u = v 2^-lz
// with v in [1/2, 1), v c_i = 1 - t for the table's 16-bit c_i <= 1 / v, then
// -ln(1 - t) = t + t^2 Q(t).  Square root: a single-precision reciprocal root
// as seed and two terms of the series of (1 - h)^(-1/2), h = 1 - m g^2.  Sine
// and cosine: quadrants off the top bits exactly, then 2 x S(x^2) and
// 1 - x^2 C(x^2) with x in [0, 1/2] for [0, pi/4].  S, C, Q interpolate their
// functions at Chebyshev nodes (degree 7, 6, 5; errors below 2^-69, 2^-62 and,
// times t^2 <= 2^-14 against t, 2^-62); the coefficients were solved for with
// 60 decimal digits.  u1 = 0 and its infinite radius are the caller's.
#ifndef VSMC_GB300_NORMAL64_CUH
#define VSMC_GB300_NORMAL64_CUH

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#include <math_constants.h>
#define VSMC_N64 __host__ __device__ __forceinline__
#else
#include <cmath>
#define VSMC_N64 inline
#endif

namespace vsmc_cuda {

// {-ln-reduction value ln(c / 2^15) 2^64, c = floor(2^15 256 / (129 + i))}
struct alignas(16) N64Log {
    uint64_t L;
    uint32_t c, pad;
};

#define VSMC_N64_TABLE                                                         \
    {0xaf731b50a6b6b1a3ull, 65027u, 0u},                                      \
    {0xad793ee16746d6e6ull, 64527u, 0u},                                      \
    {0xab83a335d8413283ull, 64035u, 0u},                                      \
    {0xa99161343342b993ull, 63550u, 0u},                                      \
    {0xa7a2941aca70c882ull, 63072u, 0u},                                      \
    {0xa5b7577c8d98eb0cull, 62601u, 0u},                                      \
    {0xa3cfc73ee1545f94ull, 62137u, 0u},                                      \
    {0xa1ebff97491dd125ull, 61680u, 0u},                                      \
    {0xa00c1d08e34c7277ull, 61230u, 0u},                                      \
    {0x9e303c61b5f5a919ull, 60787u, 0u},                                      \
    {0x9c564eb882351520ull, 60349u, 0u},                                      \
    {0x9a80956cafe41255ull, 59918u, 0u},                                      \
    {0x98ae142159b235d3ull, 59493u, 0u},                                      \
    {0x96dee2bd38d9ed96ull, 59074u, 0u},                                      \
    {0x951319683d961d99ull, 58661u, 0u},                                      \
    {0x934ad0899edc926dull, 58254u, 0u},                                      \
    {0x9184fec5d1c4b236ull, 57852u, 0u},                                      \
    {0x8fc2dafe28b2c589ull, 57456u, 0u},                                      \
    {0x8e03584d5d0e334bull, 57065u, 0u},                                      \
    {0x8c468a0728c4f390ull, 56679u, 0u},                                      \
    {0x8a8dadb77b4e89abull, 56299u, 0u},                                      \
    {0x88d7b11e3a553cd7ull, 55924u, 0u},                                      \
    {0x87237a303844db4bull, 55553u, 0u},                                      \
    {0x857377167aa7d0c6ull, 55188u, 0u},                                      \
    {0x83c55e296fd92dfeull, 54827u, 0u},                                      \
    {0x821a71f3855556f7ull, 54471u, 0u},                                      \
    {0x8072c72d8fbd5886ull, 54120u, 0u},                                      \
    {0x7ecd3abde602106cull, 53773u, 0u},                                      \
    {0x7d29dbb7c15c8d2dull, 53430u, 0u},                                      \
    {0x7b89f55aa7cf84caull, 53092u, 0u},                                      \
    {0x79ec5f0f3cedb376ull, 52758u, 0u},                                      \
    {0x785128681c9ae0feull, 52428u, 0u},                                      \
    {0x76b9a3212d765652ull, 52103u, 0u},                                      \
    {0x75235d1b422193f6ull, 51781u, 0u},                                      \
    {0x738fa65f822a9fc0ull, 51463u, 0u},                                      \
    {0x71ffd71d14d3248cull, 51150u, 0u},                                      \
    {0x707171a4fe0e763bull, 50840u, 0u},                                      \
    {0x6ee4806d7f8392c8ull, 50533u, 0u},                                      \
    {0x6d5baa1111222413ull, 50231u, 0u},                                      \
    {0x6bd465491b374048ull, 49932u, 0u},                                      \
    {0x6a4ebcf1b3474028ull, 49636u, 0u},                                      \
    {0x68cc100813e98dcdull, 49344u, 0u},                                      \
    {0x674c6fa84fb4eadcull, 49056u, 0u},                                      \
    {0x65cd3d0b70d9f64aull, 48770u, 0u},                                      \
    {0x64528b8d6ee82645ull, 48489u, 0u},                                      \
    {0x62d85ea20897c5c4ull, 48210u, 0u},                                      \
    {0x616019dcf4274a38ull, 47934u, 0u},                                      \
    {0x5feb28ef18544bb8ull, 47662u, 0u},                                      \
    {0x5e783ba1e2aaf205ull, 47393u, 0u},                                      \
    {0x5d075ddb19e6c585ull, 47127u, 0u},                                      \
    {0x5b97359a36536cdfull, 46863u, 0u},                                      \
    {0x5a2a98fa4d88439eull, 46603u, 0u},                                      \
    {0x58bec62c1b1e74b5ull, 46345u, 0u},                                      \
    {0x57569b7d54f4baa5ull, 46091u, 0u},                                      \
    {0x55ef4f4efbe5dcebull, 45839u, 0u},                                      \
    {0x548a581cd08f5ab8ull, 45590u, 0u},                                      \
    {0x53265077a5ce5dffull, 45343u, 0u},                                      \
    {0x51c62709c6906c14ull, 45100u, 0u},                                      \
    {0x50658c8e8a9a6f87ull, 44858u, 0u},                                      \
    {0x4f08e9dcbac60a55ull, 44620u, 0u},                                      \
    {0x4dad5ddaf0445a5eull, 44384u, 0u},                                      \
    {0x4c52ef86f2535b80ull, 44150u, 0u},                                      \
    {0x4afb23f3418b3a6dull, 43919u, 0u},                                      \
    {0x49a48844536df48bull, 43690u, 0u},                                      \
    {0x4850a5b4226349d6ull, 43464u, 0u},                                      \
    {0x46fe058d57ae4ef7ull, 43240u, 0u},                                      \
    {0x45acaf2e68e5a71bull, 43018u, 0u},                                      \
    {0x445e32089f71ef78ull, 42799u, 0u},                                      \
    {0x430f879cd369002dull, 42581u, 0u},                                      \
    {0x41c3c9809c411a26ull, 42366u, 0u},                                      \
    {0x40797757d0979a0dull, 42153u, 0u},                                      \
    {0x3f3228d966e6f2f6ull, 41943u, 0u},                                      \
    {0x3deac7c98f37bb41ull, 41734u, 0u},                                      \
    {0x3ca4e9ff14d78f87ull, 41527u, 0u},                                      \
    {0x3b622d619d307e01ull, 41323u, 0u},                                      \
    {0x3a1f6fe44abca15bull, 41120u, 0u},                                      \
    {0x38dfe78ddf9ee133ull, 40920u, 0u},                                      \
    {0x37a06a70432943aeull, 40721u, 0u},                                      \
    {0x366298ae1e7c09a7ull, 40524u, 0u},                                      \
    {0x35267a7823b2e908ull, 40329u, 0u},                                      \
    {0x33ec180d08abcaabull, 40136u, 0u},                                      \
    {0x32b379b92afa5dc6ull, 39945u, 0u},                                      \
    {0x317ca7d62fdcf8a6ull, 39756u, 0u},                                      \
    {0x304602c983466376ull, 39568u, 0u},                                      \
    {0x2f12e10a8206e57eull, 39383u, 0u},                                      \
    {0x2ddff916e70d76caull, 39199u, 0u},                                      \
    {0x2cad4d7c3ba5b2f2ull, 39016u, 0u},                                      \
    {0x2b7e40d6a07b62a2ull, 38836u, 0u},                                      \
    {0x2a4f7dc93789178bull, 38657u, 0u},                                      \
    {0x292107055921bbe6ull, 38479u, 0u},                                      \
    {0x27f64b4b2a5195beull, 38304u, 0u},                                      \
    {0x26cbe9602aa02c5aull, 38130u, 0u},                                      \
    {0x25a1e418acc03c07ull, 37957u, 0u},                                      \
    {0x2479fa542a63c3c5ull, 37786u, 0u},                                      \
    {0x235434fc45ac5394ull, 37617u, 0u},                                      \
    {0x222edd0447c8f667ull, 37449u, 0u},                                      \
    {0x2109f56a796b6c92ull, 37282u, 0u},                                      \
    {0x1fe74539048cab73ull, 37117u, 0u},                                      \
    {0x1ec6d582f6891ab6ull, 36954u, 0u},                                      \
    {0x1da6e7637c46a0fbull, 36792u, 0u},                                      \
    {0x1c877e015f78eeb7ull, 36631u, 0u},                                      \
    {0x1b6a688d9b5b1760ull, 36472u, 0u},                                      \
    {0x1a4de24086f4272cull, 36314u, 0u},                                      \
    {0x1931ee5c50c88b32ull, 36157u, 0u},                                      \
    {0x1818622ea35b7b99ull, 36002u, 0u},                                      \
    {0x16ff7309f8c0031eull, 35848u, 0u},                                      \
    {0x15e8fa4d8591c6fdull, 35696u, 0u},                                      \
    {0x14d1515b987ce306ull, 35544u, 0u},                                      \
    {0x13bc29a634a47519ull, 35394u, 0u},                                      \
    {0x12a98ca42af79bc2ull, 35246u, 0u},                                      \
    {0x1195c7d0380c60faull, 35098u, 0u},                                      \
    {0x108498b51e39b133ull, 34952u, 0u},                                      \
    {0x0f7426df90f9f5c2ull, 34807u, 0u},                                      \
    {0x0e6475e621d0b8c4ull, 34663u, 0u},                                      \
    {0x0d576f687d567e0cull, 34521u, 0u},                                      \
    {0x0c494d09c7b94404ull, 34379u, 0u},                                      \
    {0x0b3de079546ba612ull, 34239u, 0u},                                      \
    {0x0a33476a1671f4c1ull, 34100u, 0u},                                      \
    {0x0927979600c7e5bbull, 33961u, 0u},                                      \
    {0x08209ec4f3222233ull, 33825u, 0u},                                      \
    {0x071896baf3e8b82aull, 33689u, 0u},                                      \
    {0x06117149d7127c61ull, 33554u, 0u},                                      \
    {0x050b324851e221c7ull, 33420u, 0u},                                      \
    {0x0407d5961cd6107dull, 33288u, 0u},                                      \
    {0x03037113d7f3e59cull, 33156u, 0u},                                      \
    {0x0201faaeb0fbce24ull, 33026u, 0u},                                      \
    {0x00ff805515885e02ull, 32896u, 0u},                                      \
    {0x0000000000000000ull, 32768u, 0u}                                      

#ifdef __CUDACC__
static __device__ const N64Log kN64Log[128] = {VSMC_N64_TABLE};
#endif
#ifndef __CUDA_ARCH__
static const N64Log kN64LogHost[128] = {VSMC_N64_TABLE};
#endif

VSMC_N64 N64Log n64_log_entry(uint32_t i)
{
#ifdef __CUDA_ARCH__
    const uint4 v = __ldg(reinterpret_cast<const uint4 *>(kN64Log) + i);
    return {v.x | static_cast<uint64_t>(v.y) << 32, v.z, 0u};
#else
    return kN64LogHost[i];
#endif
}

VSMC_N64 uint32_t n64_mulhi32(uint32_t a, uint32_t b)
{
    return static_cast<uint32_t>((static_cast<uint64_t>(a) * b) >> 32);
}

VSMC_N64 uint64_t n64_mul(uint32_t a, uint32_t b)
{
    return static_cast<uint64_t>(a) * b;
}

// the high half of a b less at most 2: the low halves' product is left out
VSMC_N64 uint64_t n64_mulhi(uint64_t a, uint64_t b)
{
    const uint32_t ah = static_cast<uint32_t>(a >> 32), al = static_cast<uint32_t>(a);
    const uint32_t bh = static_cast<uint32_t>(b >> 32), bl = static_cast<uint32_t>(b);
    return n64_mul(ah, bh) + n64_mulhi32(ah, bl) + n64_mulhi32(al, bh);
}

VSMC_N64 int n64_clz(uint64_t a)
{
#ifdef __CUDA_ARCH__
    return __clzll(static_cast<long long>(a));
#else
    return a == 0 ? 64 : __builtin_clzll(a);
#endif
}

VSMC_N64 float n64_rsqrt(float x)
{
#ifdef __CUDA_ARCH__
    return rsqrtf(x);
#else
    return 1.0f / std::sqrt(x);
#endif
}

// the double of mantissa m53 in [2^52, 2^53]: m53 2^(e - 53)
VSMC_N64 double n64_double(uint64_t m53, int e)
{
    const uint64_t b = (static_cast<uint64_t>(e + 1021) << 52) + m53;
#ifdef __CUDA_ARCH__
    return __longlong_as_double(static_cast<long long>(b));
#else
    double r;
    std::memcpy(&r, &b, 8);
    return r;
#endif
}

// -ln(v 2^-(64 + k)) = m 2^(e - 64), v and m with the top bit set, not for
// v = 2^64 - 1 rounded up to 1 (the logarithm of 1); 0 <= k <= 63, Wide: 1100
template <bool Wide>
VSMC_N64 uint64_t n64_neg_log(uint64_t v, int k, int &e)
{
    const uint32_t i = static_cast<uint32_t>(v >> 56) & 127u;
    const N64Log tab = n64_log_entry(i);
    // t = 1 - v c / 2^15 as a 70-bit fraction: (2^79 - v c) / 2^9, rounded up
    // and exact for the last interval (c = 2^15), where v near 1 needs all of it
    const uint64_t p0 = n64_mul(static_cast<uint32_t>(v), tab.c);
    const uint64_t p1 =
        n64_mul(static_cast<uint32_t>(v >> 32), tab.c) + (p0 >> 32);
    const uint64_t t = 0 - ((p1 << 23) + (static_cast<uint32_t>(p0) >> 9));
    // w = t Q(t) as a 64-bit fraction
    const uint32_t th = static_cast<uint32_t>(t >> 32);
    const uint32_t q4 = 0xaaa3a1b5u + n64_mulhi32(th, 0x025572d9u);
    uint64_t q = 0x00000ccccd432a6eull + (n64_mul(th, q4) >> 26);
    q = 0x0003fffffff1f2a8ull + n64_mulhi(t, q);
    q = 0x015555555555f16full + n64_mulhi(t, q);
    q = 0x7ffffffffffffee7ull + n64_mulhi(t, q);
    const uint64_t w = n64_mulhi(t, q) >> 6;
    // k ln2 + ln c + t + t w: 2^-64 units below 1 (k = 0), else 2^-58 (Wide:
    // 2^-53 from k = 64 on)
    const uint64_t y = t + n64_mulhi(t, w);
    const int sh = k == 0 ? 0 : (Wide && k > 63 ? 11 : 6);
    uint64_t m = (tab.L + (y >> 6)) >> sh;
    if (Wide) // ln2 in two 32-bit halves
        m += (n64_mul(static_cast<uint32_t>(k), 0xb17217f7u) << (32 - sh)) +
            (n64_mul(static_cast<uint32_t>(k), 0xd1cf79acu) >> sh);
    else
        m += static_cast<uint64_t>(k) * 0x02c5c85fdf473de7ull;
    e = sh;
    if (k == 0 && i == 127) { // t + t w alone: keep the bits of a small t
        const int s = n64_clz(t) - 1;
        const uint64_t tn = t << s;
        m = tn + n64_mulhi(tn, w);
        e = -6 - s;
    }
    const int z = n64_clz(m);
    e -= z;
    return m << z;
}

// sqrt(-2 ln(u 2^-64)), u > 0
VSMC_N64 double n64_radius(uint64_t u)
{
    const int lz = n64_clz(u);
    int e;
    uint64_t m = n64_neg_log<false>(u << lz, lz, e);
    ++e; // 2 R
    // -2 ln u as the FP64 logarithm would give it, 53 bits (as 2^-63 units)
    m = ((m >> 1) + 512) & ~1023ull;
    // e even, m in [1/4, 1]
    m >>= e & 1;
    e += e & 1;
    // g = m^(-1/2) (1 + d), |d| < 2^-20, as 2.30; h = 1 - m g^2 as 2.61
    const float f =
        static_cast<float>(static_cast<uint32_t>(m >> 32)) * 0x1p-31f;
    // (1 - 2^-22 keeps g below 2)
    const uint32_t g =
        static_cast<uint32_t>(n64_rsqrt(f) * (0x1p30f - 256.0f));
    const uint64_t g2 = n64_mul(g, g) << 2;
    const int64_t h =
        static_cast<int64_t>((1ull << 61) - n64_mulhi(m, g2));
    const int32_t hs = static_cast<int32_t>(h >> 21); // 2^-40 units, < 2^21
    const int64_t h2 = static_cast<int64_t>(hs) * hs; // 2^-80 units
    // r = s0 + s0 c, c = h / 2 + 3 h^2 / 8 as 2^-82 units, s0 = m g as 2^-61
    const int64_t c = (h << 20) + ((3 * h2) >> 1);
    const uint64_t s0 = n64_mul(static_cast<uint32_t>(m >> 32), g) +
        n64_mulhi32(static_cast<uint32_t>(m), g);
    const uint64_t sa = s0 << 2; // s0 may pass 1
    const int32_t ch = static_cast<int32_t>(c >> 32);
    const uint32_t cl = static_cast<uint32_t>(c);
    const uint32_t sb = static_cast<uint32_t>(sa >> 32);
    const int64_t cor = static_cast<int64_t>(sb) * ch +
        static_cast<int64_t>(n64_mulhi32(sb, cl)) +
        ((static_cast<int64_t>(static_cast<uint32_t>(sa)) * ch) >> 32);
    // in [1/2, 1] as 2^-61 units, to 53 bits
    const uint64_t r = s0 + static_cast<uint64_t>(cor >> 20);
    return n64_double((r + 128) >> 8, e >> 1);
}

// Sine and cosine of th = 2 pi (u 2^-64) rounded to FP64, as the FP64 product
// of the constant 2 pi and the uniform is.  u: a multiple of 2^11.
VSMC_N64 void n64_sincos(uint64_t u, double &sv, double &cv)
{
    // P = K u, K = (FP64 2 pi) 2^50; th is P 2^-114 rounded to 53 bits
    constexpr uint32_t kh = 0x1921fbu, kl = 0x54442d18u;
    const uint32_t uh = static_cast<uint32_t>(u >> 32);
    const uint32_t ul = static_cast<uint32_t>(u);
    const uint64_t p00 = n64_mul(ul, kl);
    const uint64_t p01 = n64_mul(uh, kl) + (p00 >> 32);
    const uint64_t p10 = n64_mul(ul, kh) + static_cast<uint32_t>(p01);
    const uint64_t Ph = n64_mul(uh, kh) + (p01 >> 32) + (p10 >> 32);
    const uint64_t Pl = (p10 << 32) | static_cast<uint32_t>(p00);
    // P minus its rounded value, in 2^-64 ulps: its bits below the 53rd, of
    // which none is above the low word (Ph < 2^53); a tie goes to even
    const int zp = n64_clz(Ph); // 64 for u = 2^11, whose low word is full
    uint64_t rem = Pl << (zp - 11);
    if (rem == 1ull << 63 &&
        ((zp > 11 ? Pl >> (75 - zp) : Ph) & 1u) == 0)
        --rem;
    // The angle in turns is u (1 + rho) - rem / 2 pi, rho the relative error
    // of the constant: a correction in 2^-96 turns
    const bool up = rem >> 63;
    const uint64_t rt = n64_mulhi(up ? 0 - rem : rem, 0x28be60db9391054bull);
    const int64_t er = static_cast<int64_t>((rt >> 7) >> (zp & 63) >> (zp >> 6));
    const int64_t E = (up ? er : -er) -
        static_cast<int64_t>(n64_mulhi(u, 0x2cf15f5c6baull));
    // signed distance to the nearest axis, in 2^-96 turns: (dh, dl)
    const uint32_t qd = static_cast<uint32_t>((u + (1ull << 61)) >> 62);
    const uint64_t d0 = u - (static_cast<uint64_t>(qd) << 62);
    uint64_t dl = (d0 << 32) + static_cast<uint64_t>(E);
    uint32_t dh = static_cast<uint32_t>(d0 >> 32) +
        static_cast<uint32_t>(E < 0 ? ~0u : 0u) +
        (dl < static_cast<uint64_t>(E) ? 1u : 0u);
    const bool neg = dh >> 31;
    if (neg) {
        dh = ~dh + (dl == 0 ? 1u : 0u);
        dl = 0 - dl;
    }
    const uint64_t a = (static_cast<uint64_t>(dh) << 32) | (dl >> 32);
    const uint64_t x = (a << 2) | ((dl >> 30) & 3u);
    const uint64_t w = n64_mulhi(x, x);
    const uint32_t wh = static_cast<uint32_t>(w >> 32);
    // S(w), x = 1/2 for pi/4: 2^-50 units for the last three coefficients
    uint32_t p = 0x01e8eed1u - n64_mulhi32(wh, 0x0005b16eu);
    p = 0x78c1d2d4u - n64_mulhi32(wh, p);
    uint64_t S = 0x000541e0d2172f61ull - (n64_mul(wh, p) >> 18);
    S = 0x0099696673156112ull - n64_mulhi(w, S);
    S = 0x0a335e33bad56c90ull - n64_mulhi(w, S);
    S = 0x52aef39896f94aedull - n64_mulhi(w, S);
    S = 0xc90fdaa22168c235ull - n64_mulhi(w, S);
    // C(w) / 2: 2^-53 units for the last two
    p = 0x7e738917u - n64_mulhi32(wh, 0x01b2f3ebu);
    uint64_t C = 0x0000d368f77a3cdfull - (n64_mul(wh, p) >> 21);
    C = 0x001e1f5068688d5bull - n64_mulhi(w, C);
    C = 0x02aba78fc796481eull - n64_mulhi(w, C);
    C = 0x20783e1036b5808aull - n64_mulhi(w, C);
    C = 0x9de9e64df22ef2ceull - n64_mulhi(w, C);
    // 1 - w C in (0.7, 1], as 2^-63 units, to 53 bits
    const double co = n64_double(
        ((1ull << 63) + 512 - n64_mulhi(w, C)) >> 10, 0);
    // sin = 2 x S, 2 x = an 2^(-z - 64 + 3), an normalised
    const int z0 = n64_clz(a), z = a != 0 ? z0 : 32 + n64_clz(dl);
    const uint64_t an = a != 0
        ? (a << (z0 & 63)) | (((dl << 32) >> 1) >> (63 - (z0 & 63)))
        : dl << (z & 31);
    const uint64_t sm = n64_mulhi(an, S);
    // (in [0.35, 0.79): normalised, to 53 bits)
    const int zs = sm >> 63 ? 0 : 1;
    const double si = an == 0
        ? 0.0
        : n64_double((((sm << zs) >> 1) + 512) >> 10, 3 - z - zs);
    // quadrant
    const double p1 = neg ? -si : si;
    const bool swap = qd & 1u;
    const double s1 = swap ? co : p1, c1 = swap ? p1 : co;
    sv = qd & 2u ? -s1 : s1;
    cv = (qd + 1u) & 2u ? -c1 : c1;
}

#ifdef __CUDACC__
// sqrt(-2 ln u1), sin(2 pi u2), cos(2 pi u2) of u = U 2^-64 in [0, 1)
__device__ __forceinline__ void n64_polar(
    uint64_t U1, uint64_t U2, double &t, double &sv, double &cv)
{
    if (U1 == 0) { // an infinite radius, and the angle rounded as before
        t = CUDART_INF;
        sincos(__dmul_rn(6.28318530717958647693,
                   __ull2double_rn(U2) * 0x1p-64), &sv, &cv);
        return;
    }
    t = n64_radius(U1);
    n64_sincos(U2, sv, cv);
}

// the 64-bit fraction of u in [0, 1), a multiple of 2^-64
__device__ __forceinline__ uint64_t n64_fraction(double u)
{
    return __double2ull_rz(__dmul_rn(u, 0x1p64));
}
#endif

} // namespace vsmc_cuda

#endif // VSMC_GB300_NORMAL64_CUH
