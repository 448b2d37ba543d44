// FP64 arithmetic moved off GB300's FP64 pipe, bit for bit.
#ifndef LGD_K_FP64_CUH
#define LGD_K_FP64_CUH

#include "k_common.cuh"

namespace lgd {

// a * fl(1/7), the correctly rounded IEEE product, in integer arithmetic.
// With a = M * 2^k (M the 53-bit significand) and fl(1/7) = C7 * 2^-54, the
// exact product M * C7 has 104 or 105 bits; hi = floor(M * C7 / 2^41) holds
// its top 63 or 64, of which the result keeps 53.  Adding half of the last
// kept bit before the shift rounds to nearest unless the product lies
// exactly between two doubles: C7 is odd, so that needs M divisible by 2^50
// (four leading values only).  Those, zeros, subnormals, infinities, NaN and
// results near the subnormal range take the FP64 multiplication.
#define LGD_FP64_C7_SHIFT 12
__device__ __forceinline__ double mul_seventh(double a)
{
    const unsigned long long u = (unsigned long long)__double_as_longlong(a);
    const unsigned e = (unsigned)(u >> 52) & 0x7ffu;
    if (e - 8u < 2038u && (u & 0x0003ffffffffffffull) != 0) {       // 8 <= e <= 2045
        const unsigned long long hi =
            __umul64hi((u << 11) | 0x8000000000000000ull, (unsigned long long)LGD_FIX_C7 << LGD_FP64_C7_SHIFT);
        const unsigned big = (unsigned)(hi >> 63);
        const unsigned long long m = (hi + (512ull << big)) >> (10u + big);
        // m holds its leading bit, which adds one to the exponent field
        const unsigned long long r = m + ((unsigned long long)(e - 4u + big) << 52);
        return __longlong_as_double((long long)(r | (u & 0x8000000000000000ull)));
    }
    return __dmul_rn(a, 1.0 / 7.0);
}

// fl(fl(fl(a + b) + c) + d), the IEEE sum in that order, in integer arithmetic;
// false where that does not hold (the caller adds in FP64): operands of
// different sign or more than six binary exponents apart, zeros, subnormals,
// infinities, NaN and the ends of the exponent range.  With drop_d, d stands
// for +-0 and its value is not looked at.
// The operands become integers in units of 2^-53 times the smallest one's
// power of two (so that the first rounding already has a bit to drop); a sum of
// four is below 2^62.  A sum of 53 + k bits drops k: half a unit minus one,
// plus the last kept bit, rounds to nearest even.
#define LGD_FP64_SUM_REACH 7
__device__ __forceinline__ bool sum4(double a, double b, double c, double d, bool drop_d, double& sum)
{
    const unsigned ha = (unsigned)__double2hiint(a), sign = ha & 0x80000000u;
    const unsigned h[4] = {ha ^ sign, (unsigned)__double2hiint(b) ^ sign, (unsigned)__double2hiint(c) ^ sign,
                           drop_d ? ha ^ sign : (unsigned)__double2hiint(d) ^ sign};
    const unsigned lo[4] = {(unsigned)__double2loint(a), (unsigned)__double2loint(b), (unsigned)__double2loint(c),
                            (unsigned)__double2loint(d)};
    const unsigned e0 = (min(min(h[0], h[1]), min(h[2], h[3])) >> 20) - 1u;
    unsigned long long v[4];
    unsigned reach = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const unsigned shift = (h[i] >> 20) - e0;           // 1 .. 7; another sign's exponent is far above
        const unsigned m = (h[i] & 0xfffffu) | 0x100000u;
        reach |= shift;
        v[i] = ((unsigned long long)__funnelshift_l(lo[i], m, shift) << 32) | (lo[i] << (shift & 31u));
    }
    if (drop_d) v[3] = 0;
    unsigned long long s = v[0];
    unsigned k = 0;
#pragma unroll
    for (int i = 1; i < 4; ++i) {
        s += v[i];
        k = 11u - (unsigned)__clz((int)(s >> 32));
        const unsigned unit = 1u << (k & 31u);
        s += (unit >> 1) - 1u + (((unsigned)s >> (k & 31u)) & 1u);
        s &= ~(unsigned long long)(unit - 1u);
    }
    // s >> k holds the leading bit, which adds one to the exponent field
    const unsigned long long r = (s >> (k & 31u)) + ((unsigned long long)(e0 + k - 1u) << 52);
    sum = __longlong_as_double((long long)(r | ((unsigned long long)sign << 32)));
    return reach <= LGD_FP64_SUM_REACH && e0 - 1u < 2030u;
}

// fl(a b) in integer arithmetic; ok becomes false where an operand is subnormal,
// infinite or NaN or the result leaves the middle of the exponent range.  A product
// of the significands has 105 or 106 bits, hi its top 63 or 64; of the rest only
// whether it is zero matters.
__device__ __forceinline__ double mul_integer(double a, double b, bool& ok)
{
    const unsigned ha = (unsigned)__double2hiint(a), hb = (unsigned)__double2hiint(b);
    const unsigned ea = (ha >> 20) & 0x7ffu, eb = (hb >> 20) & 0x7ffu;
    const unsigned sign = (ha ^ hb) & 0x80000000u;
    const unsigned long long ma = ((unsigned long long)__double_as_longlong(a) << 11) | 0x8000000000000000ull;
    const unsigned long long mb = ((unsigned long long)__double_as_longlong(b) << 11) | 0x8000000000000000ull;
    const unsigned long long hi = __umul64hi(ma, mb), lo = ma * mb;
    const unsigned big = (unsigned)(hi >> 63), drop = 10u + big;
    const unsigned odd = ((unsigned)hi >> drop) & 1u;
    const unsigned long long m = (hi + ((512u << big) - 1u) + (odd | (lo != 0))) >> drop;
    // m holds its leading bit, which adds one to the exponent field
    const unsigned e = ea + eb + big - 1024u;
    const unsigned long long r = (m + ((unsigned long long)e << 52)) | ((unsigned long long)sign << 32);
    const bool zero = ((ha & 0x7fffffffu) | (unsigned)__double2loint(a)) == 0u ||
                      ((hb & 0x7fffffffu) | (unsigned)__double2loint(b)) == 0u;
    ok = ok && ea < 2047u && eb < 2047u && (zero || (ea != 0u && eb != 0u && e - 2u < 2040u));
    return __longlong_as_double((long long)(zero ? (unsigned long long)sign << 32 : r));
}

}  // namespace lgd

#endif
