// Correctly rounded binary64 division and square root on the integer units.
//
// The GB300 issues one binary64 warp instruction per 16 cycles and SM, and
// its divide and square root take about nine of them: 145 cycles per warp
// (measured; add and multiply: 17). The binary64 kernels were bound by that
// pipe, most of it divisions, while the integer units stood idle. The
// functions here work on the significands as integers: a binary32 seed
// (rcp / rsqrt of the leading 24 bits), then three digits of 17 or 18 bits by
// long division (Knuth, The Art of Computer Programming 2, 4.3.1: each digit
// estimated from the remainder's leading bits, the remainder exact), so that
// the quotient's 54 bits are those of the infinite expansion and rounding to
// nearest is adding its last bit (neither a quotient nor a square root of
// 53-bit numbers can be a tie): 31 cycles per warp, and no binary64
// instruction. The results are IEEE ones, bit for bit those of a / b and
// sqrt(a): zero numerators are handled in line, everything else that is not
// a normal number with a normal result goes to the general operation.
//
// Plain C++ for the host as well (the tests run every step of it there with
// the seed moved by several units in the last place).
#pragma once

#include <cmath>
#include <cstring>

#ifdef __CUDACC__
#define TJQ_HD __host__ __device__ __forceinline__
#define TJQ_SLOW static __host__ __device__ __noinline__
#else
#define TJQ_HD inline
#define TJQ_SLOW static inline
#endif

namespace tj {

typedef unsigned long long tjq_u64;

TJQ_HD unsigned tjq_mulhi(unsigned a, unsigned b)
{
#ifdef __CUDA_ARCH__
    return __umulhi(a, b);
#else
    return (unsigned)(((tjq_u64)a * b) >> 32);
#endif
}

TJQ_HD tjq_u64 tjq_bits(double x)
{
#ifdef __CUDA_ARCH__
    return (tjq_u64)__double_as_longlong(x);
#else
    tjq_u64 u;
    std::memcpy(&u, &x, 8);
    return u;
#endif
}

TJQ_HD double tjq_double(tjq_u64 u)
{
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)u);
#else
    double x;
    std::memcpy(&x, &u, 8);
    return x;
#endif
}

TJQ_HD float tjq_float(unsigned u)
{
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float x;
    std::memcpy(&x, &u, 4);
    return x;
#endif
}

TJQ_HD unsigned tjq_fbits(float x)
{
#ifdef __CUDA_ARCH__
    return __float_as_uint(x);
#else
    unsigned u;
    std::memcpy(&u, &x, 4);
    return u;
#endif
}

#if !defined(__CUDA_ARCH__) && defined(TJQ_TEST_SEED)
extern int tjq_seed_ulps;  // the tests move the seeds
#endif

// 1 / f for f in [1, 2], within two units in the last place.
TJQ_HD float tjq_rcp(float f)
{
#ifdef __CUDA_ARCH__
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(f));
    return y;
#elif defined(TJQ_TEST_SEED)
    return tjq_float(tjq_fbits(1.0f / f) + (unsigned)tjq_seed_ulps);
#else
    return 1.0f / f;
#endif
}

// 1 / sqrt(f) for f in [1, 4], within two units in the last place.
TJQ_HD float tjq_rsqrt(float f)
{
#ifdef __CUDA_ARCH__
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(f));
    return y;
#elif defined(TJQ_TEST_SEED)
    return tjq_float(tjq_fbits(1.0f / std::sqrt(f)) + (unsigned)tjq_seed_ulps);
#else
    return 1.0f / std::sqrt(f);
#endif
}

// y in (1/2, 1] as a 32-bit fraction, 2^-21 to 2^-20 below it: a lower bound
// of the exact reciprocal whatever the seed's rounding.
TJQ_HD unsigned tjq_fraction(float y)
{
    const float g = y + (1.0f - 4.76837158203125e-07f);  // in [1.5 - 2^-21, 2)
    return tjq_fbits(g) << 9;
}

TJQ_SLOW double tjq_div_general(double a, double b) { return a / b; }
TJQ_SLOW double tjq_sqrt_general(double a)
{
#ifdef __CUDA_ARCH__
    return ::sqrt(a);
#else
    return std::sqrt(a);
#endif
}

// One digit: rem = rem * 2^BITS - d * den with d <= rem * 2^BITS / den, short
// of it by less than 1.52 (the seed's 2^-20, the dropped bits and the floor),
// so that rem stays in [0, 1.52 den): computed modulo 2^64, rem * 2^BITS
// itself does not fit. nlo / nhi hold -den.
template <int BITS>
TJQ_HD unsigned tjq_digit(tjq_u64& rem, unsigned V, unsigned nlo, unsigned nhi)
{
    const unsigned d = tjq_mulhi((unsigned)(rem >> 22), V) >> (30 - BITS);
    rem = (rem << BITS) + (tjq_u64)d * nlo + ((tjq_u64)(d * nhi) << 32);
    return d;
}

// a / b, rounded to nearest.
TJQ_HD double tjq_div(double a, double b)
{
    const tjq_u64 ua = tjq_bits(a), ub = tjq_bits(b), mask = 0xFFFFFFFFFFFFFull;
    const int ea = (int)(ua >> 52) & 0x7ff, eb = (int)(ub >> 52) & 0x7ff;
    const tjq_u64 ma = (ua & mask) | (mask + 1), mb = (ub & mask) | (mask + 1);
    const bool lt = ma < mb;
    const int er = ea - eb + (lt ? 1022 : 1023);
    const tjq_u64 sign = (ua ^ ub) & 0x8000000000000000ull;
    const bool zero = (ua << 1) == 0;
    if ((unsigned)(eb - 1) >= 2046u || (!zero && ((unsigned)(ea - 1) >= 2046u || (unsigned)(er - 1) >= 2046u)))
        return tjq_div_general(a, b);
    // the quotient's leading one is taken out: rem in [0, mb)
    tjq_u64 rem = (lt ? ma << 1 : ma) - mb;
    const unsigned V = tjq_fraction(tjq_rcp(tjq_float(0x3F800000u | ((unsigned)(mb >> 29) & 0x7FFFFFu))));
    const tjq_u64 nmb = 0ull - mb;
    const unsigned nlo = (unsigned)nmb, nhi = (unsigned)(nmb >> 32);
    const unsigned d1 = tjq_digit<18>(rem, V, nlo, nhi);
    const unsigned d2 = tjq_digit<18>(rem, V, nlo, nhi);
    const unsigned d3 = tjq_digit<17>(rem, V, nlo, nhi);
    tjq_u64 q = ((tjq_u64)d1 << 35) + ((tjq_u64)d2 << 17) + d3 + (rem >= mb ? 2 : 1);
    q = (q >> 1) + ((tjq_u64)er << 52);  // the leading one is the exponent's
    return tjq_double((zero ? 0ull : q) | sign);
}

// sqrt(a), rounded to nearest.
TJQ_HD double tjq_sqrt(double a)
{
    const tjq_u64 ua = tjq_bits(a), mask = 0xFFFFFFFFFFFFFull;
    const int ea = (int)(ua >> 52);  // with the sign: a negative number is out of range
    if ((unsigned)(ea - 1) >= 2046u) return tjq_sqrt_general(a);
    const int odd = (ea & 1) ^ 1;  // of the unbiased exponent
    const tjq_u64 M = ((ua & mask) | (mask + 1)) << odd;  // a = M 2^-52 4^k, M 2^-52 in [1, 4)
    const float f = tjq_float(((unsigned)(127 + odd) << 23) | ((unsigned)(ua >> 29) & 0x7FFFFFu));
    const float y = tjq_rsqrt(f);
    const unsigned Y = tjq_fraction(y);
    // 18 bits of the root, not above it
    const float g = f * y - 1.9073486328125e-06f;
    const unsigned s1 = ((tjq_fbits(g < 1.0f ? 1.0f : g) & 0x7FFFFFu) | 0x800000u) >> 6;
    tjq_u64 r = (M >> 18) - (tjq_u64)s1 * s1;
    r = (r << 36) + ((M & 0x3FFFFull) << 18);
    // (2 s1 2^18 + d) d <= r: the quotient by 2 s1 2^18 alone is up to one too large
    unsigned d = tjq_mulhi((unsigned)(r >> 24), Y) >> 12;
    d -= d > 0 ? 1u : 0u;
    r -= (((tjq_u64)s1 << 19) + d) * d;
    const tjq_u64 s2 = ((tjq_u64)s1 << 18) + d;
    d = tjq_mulhi((unsigned)(r >> 7), Y) >> 11;
    r = (r << 36) - ((s2 << 19) + d) * d;  // modulo 2^64: the difference fits
    tjq_u64 s = (s2 << 18) + d;
    // up to two short: the second digit's 3 2^18 times the seed's 2^-20, and the floor
    if (r > 2 * s) {
        r -= 2 * s + 1;
        ++s;
        if (r > 2 * s) ++s;
    }
    s = (s + 1) >> 1;
    return tjq_double(s + ((tjq_u64)((ea + 1021 - odd) / 2) << 52));
}

// Conversions between binary64 and binary32 on the integer units (the
// conversion instruction takes the binary64 pipe's 16 cycles a warp as well):
// the bits of the cast, which is left what is not a normal number or zero in
// both types.
TJQ_HD float narrow(double x)
{
    const tjq_u64 u = tjq_bits(x);
    const unsigned hi = (unsigned)(u >> 32), lo = (unsigned)u, sign = hi & 0x80000000u;
    const unsigned e = (hi >> 20) & 0x7ffu;
    if ((u << 1) == 0) return tjq_float(sign);
    if (e - 897u > 253u) return (float)x;
    const unsigned f = ((e - 896u) << 23) | ((hi & 0xFFFFFu) << 3) | (lo >> 29), rest = lo << 3;
    // to nearest, ties to even; a carry goes into the exponent
    return tjq_float(sign | (f + (rest > 0x80000000u || (rest == 0x80000000u && (f & 1u)) ? 1u : 0u)));
}
TJQ_HD double widen(float x)
{
    const unsigned b = tjq_fbits(x), e = (b >> 23) & 0xffu, sign = b & 0x80000000u;
    if ((b << 1) == 0) return tjq_double((tjq_u64)sign << 32);
    if (e - 1u > 253u) return (double)x;
    return tjq_double(((tjq_u64)(sign | ((e + 896u) << 20) | ((b & 0x7FFFFFu) >> 3)) << 32) | ((tjq_u64)(b << 29) & 0xFFFFFFFFull));
}

// Division and square root of the templated device code, by working type.
// TJ_QUOT_CALL: called out of line (the kernels whose straight-line code does
// not fit the instruction cache and whose warps are too few to hide its misses).
#if defined(__CUDACC__) && defined(TJ_QUOT_CALL)
#define TJQ_OP static __host__ __device__ __noinline__
#else
#define TJQ_OP TJQ_HD
#endif
TJQ_OP double quot(double a, double b)
{
#ifdef __CUDA_ARCH__
    return tjq_div(a, b);
#else
    return a / b;
#endif
}
TJQ_HD float quot(float a, float b) { return a / b; }
TJQ_OP double root(double a)
{
#ifdef __CUDA_ARCH__
    return tjq_sqrt(a);
#else
    return std::sqrt(a);
#endif
}
TJQ_HD float root(float a) { return sqrtf(a); }

// TJ_QUOT_EXPR: quot(a, b) stands for the expression a / b itself (the binary64
// one by way of an overloaded operator). As an argument of a function the
// divisor is evaluated before the dividend, and the compiler then contracts
// other pairs of products and sums: with fast math the binary32 results of
// stiff mixtures differ as much as two roundings of them do.
#if defined(__CUDACC__) && defined(TJ_QUOT_EXPR)
struct QuotBy {
    double v;
};
TJQ_HD float quot_by(float b) { return b; }
TJQ_HD QuotBy quot_by(double b) { return {b}; }
TJQ_HD double operator/(double a, QuotBy b) { return quot(a, b.v); }
#define quot(a, b) ((a) / quot_by(b))
#endif

}  // namespace tj
