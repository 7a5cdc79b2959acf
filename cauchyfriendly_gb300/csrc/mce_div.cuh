// IEEE double division and multiplication on the integer pipe.
//
// sm_103a has two FP64 lanes per SM: every FP64 warp instruction holds its
// sub-partition's pipe for 64 cycles, and a division is a chain of such
// instructions, while the integer pipe next to it idles.  Here the quotient of
// the two 53-bit significands is found by schoolbook long division in two
// digits of 30 and 22 bits (Knuth, The Art of Computer Programming vol. 2,
// 4.3.1, algorithm D, with the digits estimated through a 32-bit reciprocal
// instead of a division), and rounded by its exact remainder: the same bits as
// IEEE round-to-nearest division, for any seed within an ulp or so.
//
//   D        the divisor's significand, 2^52 <= D < 2^53
//   N        the dividend's, doubled when it is below D: 1 <= N/D < 2
//   rec      2^84 / D from below (relative error under 2^-29): the hardware's
//            single-precision reciprocal, one Newton step in integers
//   q1       floor-estimate of 2^30 N/D: at most 8 below it, never above
//   R1       2^30 N - q1 D, exact (below 2^56; mod 2^64 arithmetic suffices)
//   q2       floor-estimate of 2^22 R1/D, biased by 3/32: never above the
//            nearest integer, at most one below
//   R2       2^22 R1 - q2 D, exact: one more when 2 R2 > D.  (A quotient of
//            two doubles is never halfway between two normal doubles.)
//
// Measured (GB300, full SMs, cycles an SM spends per warp division): a / b
// 153, divide 28, with a shared divisor 24; a complex division was 391.  The
// batched 3-state run (4,096 estimators) went from 189.6 to 149.0 ms with it,
// the 5-state relative system's pairs and 13 x 13 grid from 1,177 to 728 ms,
// 256 points of the 4-state joint pdf from 322 to 211 ms.
//
// Operands outside [2^-255, 2^257) take the ordinary division (zeros over an
// operand inside give the signed zero at once), so no result of the long
// division is subnormal or overflows.
#pragma once
#include <cstdint>
#include <cstring>
#ifndef __CUDACC__
#define MCE_HD
#else
#define MCE_HD __host__ __device__
#endif

namespace mce {

struct DivBy {
    unsigned top, lo;  // the divisor's words
    unsigned rec;      // 2^84 / significand, from below
};

MCE_HD inline unsigned div_hi_word(double x)
{
#ifdef __CUDA_ARCH__
    return (unsigned)__double2hiint(x);
#else
    uint64_t u;
    std::memcpy(&u, &x, 8);
    return (unsigned)(u >> 32);
#endif
}
MCE_HD inline unsigned div_lo_word(double x)
{
#ifdef __CUDA_ARCH__
    return (unsigned)__double2loint(x);
#else
    uint64_t u;
    std::memcpy(&u, &x, 8);
    return (unsigned)u;
#endif
}
MCE_HD inline double div_words(unsigned hi, unsigned lo)
{
#ifdef __CUDA_ARCH__
    return __hiloint2double((int)hi, (int)lo);
#else
    const uint64_t u = ((uint64_t)hi << 32) | lo;
    double x;
    std::memcpy(&x, &u, 8);
    return x;
#endif
}
MCE_HD inline unsigned div_mulhi(unsigned a, unsigned b)
{
#ifdef __CUDA_ARCH__
    return __umulhi(a, b);
#else
    return (unsigned)(((uint64_t)a * b) >> 32);
#endif
}

// Bits of the single-precision reciprocal of 1 <= x < 2 (given by its bits),
// to about an ulp.
#ifdef __CUDA_ARCH__
MCE_HD inline unsigned div_seed(unsigned x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(x)));
    return __float_as_uint(y);
}
#else
#ifndef MCE_DIV_SEED_ULPS
#define MCE_DIV_SEED_ULPS 0
#endif
MCE_HD inline unsigned div_seed(unsigned x)
{
    float f, y;
    std::memcpy(&f, &x, 4);
    y = 1.0f / f;
    unsigned u;
    std::memcpy(&u, &y, 4);
    return u + (MCE_DIV_SEED_ULPS);
}
#endif

// The divisor's part, shared by every division by it.
MCE_HD inline DivBy div_by(double b)
{
    DivBy d;
    d.top = div_hi_word(b);
    d.lo = div_lo_word(b);
    // the significand's 23 bits after the leading one, as a float in [1, 2)
    const unsigned f = (((d.top << 3) | (d.lo >> 29)) & 0x7fffffu) | 0x3f800000u;
    unsigned y = div_seed(f);
    y = y < 0x3f7fffffu ? y : 0x3f7fffffu;  // in [1/2, 1), so that bit 31 leads in r0
    y = y > 0x3f000000u ? y : 0x3f000000u;
    const unsigned r0 = (y << 8) | 0x80000000u;           // 2^32 / d', d' = D / 2^52
    const unsigned d32 = (d.top << 11) | 0x80000000u | (d.lo >> 21);  // 2^31 d'
    const int e = (int)(0x7ffffffeu - div_mulhi(d32, r0));  // 2^31 (1 - d' r0 / 2^32), from below
    d.rec = r0 + (unsigned)((e * (int)(r0 >> 16)) >> 15);
    return d;
}

MCE_HD inline double div_slow(double a, const DivBy& d)
{
    const unsigned ah = div_hi_word(a), al = div_lo_word(a);
    if (((ah << 1) | al) == 0 && (((d.top + 0x10000000u) ^ 0x40000000u) & 0x60000000u) == 0)
        return div_words((ah ^ d.top) & 0x80000000u, 0);
    return a / div_words(d.top, d.lo);
}

// a / b, d = div_by(b)
MCE_HD inline double divide(double a, const DivBy& d)
{
    const unsigned top = div_hi_word(a);
    const unsigned xa = top + 0x10000000u, xb = d.top + 0x10000000u;
    if ((((xa ^ 0x40000000u) | (xb ^ 0x40000000u)) & 0x60000000u) != 0) return div_slow(a, d);
    const uint64_t D = ((uint64_t)((d.top & 0xfffffu) | 0x100000u) << 32) | d.lo;
    uint64_t N = ((uint64_t)((top & 0xfffffu) | 0x100000u) << 32) | div_lo_word(a);
    const int s = N < D ? 1 : 0;
    N <<= s;
    const unsigned q1 = div_mulhi((unsigned)(N >> 22), d.rec);
    uint64_t R = (N << 30) - (uint64_t)q1 * D;
    const unsigned q2 = (div_mulhi((unsigned)(R >> 24), d.rec) + 26u) >> 6;
    const uint64_t q = ((uint64_t)q1 << 22) + q2;
    R = (R << 22) - (uint64_t)q2 * D;
    const long long c = (long long)((R << 1) - D);
    const uint64_t qr = q + (uint64_t)(1 + (c >> 63));
    // exponent field minus one (the leading bit of qr adds it), sign
    const unsigned ex = ((top & 0x7ff00000u) - (d.top & 0x7ff00000u)) + ((1022u - (unsigned)s) << 20);
    const unsigned sg = (top ^ d.top) & 0x80000000u;
    return div_words(((unsigned)(qr >> 32) + ex) | sg, (unsigned)qr);
}

MCE_HD inline double divide(double a, double b) { return divide(a, div_by(b)); }

// a * b on the integer pipe: the 106-bit product of the significands from
// four 32-bit ones, rounded to nearest even; the same bits as the FP64 product.
// It costs an SM 18 cycles a warp, where the FP64 pipe takes 20 for one
// instruction, so it is no faster alone: a kernel bound by the FP64 pipe does
// some of its products here, next to additions and the other products there
// (one of each in turn: 10.3 cycles an operation).  How many is each kernel's
// balance between the two pipes, divisions included.  Zeros, which structured
// models are full of, are answered at once; other operands outside
// [2^-255, 2^257) take the FP64 pipe (a call, so that the compiler does not run
// both).
#ifdef __CUDACC__
static __device__ __noinline__ double mul_slow(double a, double b) { return a * b; }
#else
static inline double mul_slow(double a, double b) { return a * b; }
#endif

#ifdef __CUDACC__
__device__
#endif
inline double imul(double a, double b)
{
    const unsigned ha = div_hi_word(a), hb = div_hi_word(b);
    const unsigned xa = ha + 0x10000000u, xb = hb + 0x10000000u;
    const unsigned la = div_lo_word(a), lb = div_lo_word(b);
    const unsigned oa = (xa ^ 0x40000000u) & 0x60000000u, ob = (xb ^ 0x40000000u) & 0x60000000u;
    if ((oa | ob) != 0) {
        const bool za = ((ha << 1) | la) == 0, zb = ((hb << 1) | lb) == 0;
        if ((za && (zb || ob == 0)) || (zb && oa == 0)) return div_words((ha ^ hb) & 0x80000000u, 0);
        return mul_slow(a, b);
    }
    const unsigned ma = (ha & 0xfffffu) | 0x100000u, mb = (hb & 0xfffffu) | 0x100000u;
    const uint64_t w0 = (uint64_t)la * lb;
    const uint64_t w1 = (uint64_t)ma * lb + (unsigned)(w0 >> 32);
    const uint64_t w2 = (uint64_t)la * mb + w1;
    const uint64_t w3 = (uint64_t)ma * mb + (unsigned)(w2 >> 32);
    // the product is w3 : low w2 : low w0, of 105 bits or (n = 1) 106
    const unsigned n = (unsigned)(w3 >> 41) & 1u;
    const int sh = 22 - (int)n;  // its leading bit to bit 62 of T
    const unsigned v = (unsigned)w3, u = (unsigned)w2;
    const unsigned th = ((unsigned)(w3 >> 32) << sh) | (v >> (32 - sh));
    const unsigned tl = (v << sh) | (u >> (32 - sh));
    const unsigned rest = (u << sh) | (unsigned)w0;
    // 53 bits at 62..10 of T, the rounding bit at 9, everything below in bit 0
    const uint64_t T = (((uint64_t)th << 32) | tl | (rest ? 1u : 0u)) + 0x1ffu + ((tl >> 10) & 1u);
    const uint64_t m = T >> 10;
    const unsigned ex = (ha & 0x7ff00000u) + (hb & 0x7ff00000u) - ((1024u - n) << 20);
    return div_words(((unsigned)(m >> 32) + ex) | ((ha ^ hb) & 0x80000000u), (unsigned)m);
}

}  // namespace mce
