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

}  // namespace lgd

#endif
