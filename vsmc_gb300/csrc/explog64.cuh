// exp, log and quotients of FP64 numbers in 64-bit integers, rounded once.
//
// A warp's FP64 instruction holds its SM's FP64 pipe for 19 clocks: exp is
// about 20 of them, log 25, a quotient 10.  2^20 exponentials took 35 us and 9
// in integers (two FP64 operations are left), 10^6 logarithms and quotients 78
// and 11.  The arguments that the weights and the sorted uniforms bring are
// taken here, everything else (signs, infinities, NaN, results below 2^-1016)
// goes to the CUDA functions.
//
// exp(-a): a = K ln2 / 64 + s exactly to 2^-64, K = 64 k + j, then 2^-k
// 2^(-j/64) (1 - s H(s)) with 64 tabulated powers and the Taylor polynomial of
// (1 - exp(-s)) / s, s < 2^-5.5 (the next term is below 2^-61); P. T. P. Tang,
// "Table-driven implementation of the exponential function", ACM TOMS 15,
// 1989.  log: n64_neg_log.  Quotient by a 32-bit integer: reciprocal from a
// single-precision seed and two terms of 1 / (1 - E).  Each is within 0.55 ulp.
#ifndef VSMC_GB300_EXPLOG64_CUH
#define VSMC_GB300_EXPLOG64_CUH

#include "normal64.cuh"

namespace vsmc_cuda {

#define VSMC_N64_POWERS                                                        \
    0x8000000000000000ull,                                                    \
    0x7e9f06067a4360baull,                                                    \
    0x7d41d96db915019dull,                                                    \
    0x7be86fb985689ddcull,                                                    \
    0x7a92be8a92436616ull,                                                    \
    0x7940bb9e2cffd89dull,                                                    \
    0x77f25ccdee6d7ae6ull,                                                    \
    0x76a7980f6cca15c2ull,                                                    \
    0x75606373ee921c97ull,                                                    \
    0x741cb5281e25ee34ull,                                                    \
    0x72dc8373be41a454ull,                                                    \
    0x719fc4b95f452d29ull,                                                    \
    0x70666f76154a7089ull,                                                    \
    0x6f307a412f074892ull,                                                    \
    0x6dfddbcbed791babull,                                                    \
    0x6cce8ae13c57ebdbull,                                                    \
    0x6ba27e656b4eb57aull,                                                    \
    0x6a79ad55e7f6fd10ull,                                                    \
    0x69540ec8f895722dull,                                                    \
    0x683199ed779592caull,                                                    \
    0x6712460a8fc24072ull,                                                    \
    0x65f60a7f79393e2eull,                                                    \
    0x64dcdec3371793d1ull,                                                    \
    0x63c6ba6455dcd8aeull,                                                    \
    0x62b39508aa836d6full,                                                    \
    0x61a3666d124bb204ull,                                                    \
    0x6096266533384a2bull,                                                    \
    0x5f8bccdb3d398841ull,                                                    \
    0x5e8451cfac061b5full,                                                    \
    0x5d7fad59099f22feull,                                                    \
    0x5c7dd7a3b17dcf75ull,                                                    \
    0x5b7ec8f19468bbc9ull,                                                    \
    0x5a827999fcef3242ull,                                                    \
    0x5988e20954889245ull,                                                    \
    0x5891fac0e95612c8ull,                                                    \
    0x579dbc56b48521baull,                                                    \
    0x56ac1f752150a563ull,                                                    \
    0x55bd1cdad49f699cull,                                                    \
    0x54d0ad5a753e077cull,                                                    \
    0x53e6c9da74b29ab5ull,                                                    \
    0x52ff6b54d8a89c75ull,                                                    \
    0x521a8ad704f3404full,                                                    \
    0x513821818624b40cull,                                                    \
    0x50582887dcb8a7e1ull,                                                    \
    0x4f7a993048d088d7ull,                                                    \
    0x4e9f6cd3967fdba8ull,                                                    \
    0x4dc69cdceaa72a9cull,                                                    \
    0x4cf022c9905bfd32ull,                                                    \
    0x4c1bf828c6dc54b8ull,                                                    \
    0x4b4a169b900c2d00ull,                                                    \
    0x4a7a77d47f7b84b1ull,                                                    \
    0x49ad159789f37496ull,                                                    \
    0x48e1e9b9d588e19bull,                                                    \
    0x4818ee218a3358eeull,                                                    \
    0x47521cc5a2e6a9e0ull,                                                    \
    0x468d6fadbf2dd4f3ull,                                                    \
    0x45cae0f1f545eb73ull,                                                    \
    0x450a6abaa4b77ecdull,                                                    \
    0x444c0740496d4294ull,                                                    \
    0x438fb0cb4f468808ull,                                                    \
    0x42d561b3e6243d8aull,                                                    \
    0x421d1461d66f2023ull,                                                    \
    0x4166c34c5615d0ecull,                                                    \
    0x40b268f9de0183baull                                                    

#ifdef __CUDACC__
static __device__ const uint64_t kN64Pow[64] = {VSMC_N64_POWERS};
#endif
#ifndef __CUDA_ARCH__
static const uint64_t kN64PowHost[64] = {VSMC_N64_POWERS};
#endif

// 2^(-j / 64) 2^63
VSMC_N64 uint64_t n64_power(uint32_t j)
{
#ifdef __CUDA_ARCH__
    return __ldg(reinterpret_cast<const unsigned long long *>(kN64Pow) + j);
#else
    return kN64PowHost[j];
#endif
}

VSMC_N64 float n64_rcp(float x)
{
#ifdef __CUDA_ARCH__
    return __frcp_rn(x);
#else
    return 1.0f / x;
#endif
}

VSMC_N64 uint64_t n64_bits(double x)
{
#ifdef __CUDA_ARCH__
    return static_cast<uint64_t>(__double_as_longlong(x));
#else
    uint64_t b;
    std::memcpy(&b, &x, 8);
    return b;
#endif
}

// whether n64_exp_neg takes a = |x|: at most 704
VSMC_N64 bool n64_exp_ok(uint64_t bits)
{
    return (bits & ~(1ull << 63)) <= 0x4086000000000000ull;
}

// exp(-a), a = the double of bits (sign ignored), n64_exp_ok
VSMC_N64 double n64_exp_neg(uint64_t bits)
{
    const int e = static_cast<int>((bits >> 52) & 2047u) - 1023;
    const uint64_t mant = (bits & ((1ull << 52) - 1)) | (1ull << 52);
    // a: its 22 fraction bits and up, and its 64 fraction bits
    const int r = 30 - e > 63 ? 63 : 30 - e;
    const uint32_t a22 = static_cast<uint32_t>(mant >> r);
    const int l = e + 12;
    const uint64_t a64 =
        l >= 0 ? mant << l : (l > -64 ? mant >> (-l) : 0);
    // K = floor(64 a / ln2) or one less
    const uint32_t K = static_cast<uint32_t>(n64_mul(a22, 0x5c551d94u) >> 46);
    // s = a - K ln2 / 64, its 64 fraction bits
    const uint64_t s = a64 -
        (n64_mul(K, 0xdf473de6u) + (n64_mul(K, 0x02c5c85fu) << 32) +
            (n64_mul(K, 0xaf278eceu) >> 32));
    const uint64_t t = s << 5;
    const uint32_t th = static_cast<uint32_t>(t >> 32);
    // H: 1 / 2^66 units for the last two coefficients
    const uint32_t h5 = 0xb60b60b6u - n64_mulhi32(th, 0x00d00d01u);
    uint64_t h = 0x0000002222222222ull - (n64_mul(th, h5) >> 34);
    h = 0x0000155555555555ull - n64_mulhi(t, h);
    h = 0x000aaaaaaaaaaaabull - n64_mulhi(t, h);
    h = 0x0400000000000000ull - n64_mulhi(t, h);
    // 1 - exp(-s) = s (1 - t h), as 2^-64 units
    const uint64_t p = s - n64_mulhi(s, n64_mulhi(t, h));
    const uint64_t T = n64_power(K & 63u);
    const uint64_t m = T - n64_mulhi(T, p); // (0.48, 1] 2^63
    const int z = m >> 62 ? 0 : 1;
    return n64_double(((m << z) + 512) >> 10, -static_cast<int>(K >> 6) - z);
}

// whether n64_log_below takes x: normal and below 1
VSMC_N64 bool n64_log_ok(uint64_t bits)
{
    return bits - 0x0010000000000000ull < 0x3FE0000000000000ull;
}

// -ln of the double of bits, n64_log_ok
VSMC_N64 double n64_neg_log_double(uint64_t bits)
{
    int e;
    const uint64_t m = n64_neg_log<true>((bits << 11) | (1ull << 63),
        1022 - static_cast<int>(bits >> 52), e);
    return n64_double(((m >> 1) + 512) >> 10, e);
}

// -ln(w 2^-32) rounded to FP64, over d, rounded again; w, d > 0
VSMC_N64 double n64_neg_log_over(uint32_t w, uint32_t d)
{
    const int lz = n64_clz(static_cast<uint64_t>(w) << 32);
    int e;
    uint64_t m =
        n64_neg_log<false>((static_cast<uint64_t>(w) << 32) << lz, lz, e);
    m = ((m >> 1) + 512) & ~1023ull; // 53 bits, as 2^-63 units
    // D = d 2^zd 2^-32 in [1/2, 1), R = 1 / D as 2^-62 units
    const int zd = n64_clz(static_cast<uint64_t>(d) << 32);
    const uint32_t dn = d << zd;
    const uint32_t r0 = static_cast<uint32_t>(
        n64_rcp(static_cast<float>(dn)) * (0x1p62f - 0x1p40f));
    const int64_t E = static_cast<int64_t>((1ull << 62) - n64_mul(dn, r0));
    const int32_t Es = static_cast<int32_t>(E >> 20); // 2^-42 units
    const int64_t E2 = E + ((static_cast<int64_t>(Es) * Es) >> 22);
    const uint64_t R = (static_cast<uint64_t>(r0) << 32) +
        static_cast<uint64_t>(
            (static_cast<int64_t>(r0) * (E2 >> 12)) >> 18) +
        (n64_mul(r0, static_cast<uint32_t>(E2) & 4095u) >> 30);
    // m R as 2^-61 units, in [1/4, 1] 2^62
    const uint64_t q = n64_mulhi(m, R);
    const int z = n64_clz(q) - 1;
    return n64_double(((q << z) + 512) >> 10, e - 30 + zd - z);
}

// whether a - b > 2^-50 for sure, a >= b >= 0 the doubles of their bits (by
// their 53 fraction bits; never for values from 1024 on)
VSMC_N64 bool n64_apart(uint64_t a, uint64_t b)
{
    const int ea = static_cast<int>(a >> 52) - 1022;
    const int eb = static_cast<int>(b >> 52) - 1022;
    const uint64_t ma = (a & ((1ull << 52) - 1)) | (1ull << 52);
    const uint64_t mb = (b & ((1ull << 52) - 1)) | (1ull << 52);
    const uint64_t fa = ea >= 0 ? ma << (ea & 63) : (ea > -64 ? ma >> -ea : 0);
    const uint64_t fb = eb >= 0 ? mb << (eb & 63) : (eb > -64 ? mb >> -eb : 0);
    return ea <= 10 && static_cast<int64_t>(fa - fb) >= 9;
}

// exp(x) for x <= 0 and anything else exp takes
VSMC_N64 double exp_of_negative(double x)
{
    const uint64_t b = n64_bits(x);
    if ((b >> 63 || b == 0) && n64_exp_ok(b))
        return n64_exp_neg(b);
    return exp(x);
}

// uniform of a sum s >= 0 of the sorted sequence
struct SortedUniform {
    VSMC_N64 double operator()(double s) const
    {
        return 1.0 - exp_of_negative(-s);
    }
};

// The running maximum up to j of the sorted uniforms u_i = form(s_i), for
// non-decreasing sums s_i >= 0.  form is 1 - exp(-s) with an exp within an
// ulp, so u_j can only be below a u_i whose sum is within 2^-50 of s_j: the
// few predecessors that near (a look at one neighbour nearly always) are
// formed again.  Nothing is above u_j = 1, which an infinite sum and every
// one from 38 on gives.
template <class Sums, class Form>
VSMC_N64 double n64_sorted_max(const Sums &s, size_t j, const Form &form)
{
    const double sj = s[j];
    double u = form(sj);
    for (size_t i = j; i > 0 && u < 1.0; --i) {
        const double si = s[i - 1];
        if (n64_apart(n64_bits(sj), n64_bits(si)))
            break;
        const double v = form(si);
        u = v > u ? v : u;
    }
    return u;
}

#ifdef __CUDACC__
// log(x) for x in (0, 1) and anything else log takes
__device__ __forceinline__ double log_of_fraction(double x)
{
    const uint64_t b = n64_bits(x);
    if (n64_log_ok(b))
        return -n64_neg_log_double(b);
    return log(x);
}
#endif

} // namespace vsmc_cuda

#endif // VSMC_GB300_EXPLOG64_CUH
