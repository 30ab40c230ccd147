// a / b of two integers, rounded as the FP64 division rounds it, without the FP64 pipe.
//
// Schoolbook division by digits of 19 bits: a digit is the remainder times a single-precision
// reciprocal of b, rounded to an integer (signed, within 0.82 of the exact quotient of that
// remainder: half a unit, and 2.5 x 2^-23 of a first digit below 2^20), and the next remainder
// is exact in 64 bits. Three digits give 57 or 58 bits of the quotient and the sign of what is
// left, which is all that rounding to nearest even needs. The device's FP64 pipe does about two operations a clock and SM and a division takes ten of them
// with its conversions; this takes about sixty integer and single-precision operations at 64 or
// more a clock.
//
// Valid for 1 <= a < 2^32 and 1 <= b < 2^53; the quotient is then a normal number.
#pragma once

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define SCD_HD __host__ __device__ __forceinline__
#else
#define SCD_HD inline
#endif

namespace scd {

SCD_HD int msb32(uint32_t x) {
#ifdef __CUDA_ARCH__
    return 31 - __clz((int)x);
#else
    return 31 - __builtin_clz(x);
#endif
}

SCD_HD int msb64(uint64_t x) {
#ifdef __CUDA_ARCH__
    return 63 - __clzll((long long)x);
#else
    return 63 - __builtin_clzll(x);
#endif
}

// round(r * f), |result| < 2^21
SCD_HD int div_digit(int64_t r, float f) {
#ifdef __CUDA_ARCH__
    return __float2int_rn(__fmul_rn(__ll2float_rn(r), f));
#else
    const float x = (float)r * f;
    return (int)(x < 0 ? x - 0.5f : x + 0.5f);
#endif
}

SCD_HD double exact_div(uint32_t a, uint64_t b) {
    constexpr int DIGIT = 19;
    const int ma = msb32(a), mb = msb64(b);
    const uint64_t d = b << (52 - mb);                          // in [2^52, 2^53)
    int64_t r = (int64_t)((uint64_t)a << (52 - ma));            // in [2^52, 2^53): r / d in (1/2, 2)
    const float top = (float)(uint32_t)(d >> 29);               // 24 bits, exact
#ifdef __CUDA_ARCH__
    const float inv = __frcp_rn(top);
#else
    const float inv = 1.0f / top;
#endif
    const float f = inv * (1.0f / 1024.0f);                     // 2^DIGIT / (top 2^29)
    uint64_t q = 0;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int i = 0; i < 3; i++) {
        const int digit = div_digit(r, f);
        q = (q << DIGIT) + (uint64_t)(int64_t)digit;
        r = (int64_t)(((uint64_t)r << DIGIT) - (uint64_t)(int64_t)digit * d);   // |r| <= 0.82 d
    }
    if (r < 0) {   // q + r / d with 0 <= r < d
        q--;
        r += (int64_t)d;
    }
    const int mq = msb64(q), drop = mq - 52;                    // mq is 56 or 57
    uint64_t m = q >> drop;
    const uint64_t rest = q & ((1ull << drop) - 1), half = 1ull << (drop - 1);
    if (rest > half || (rest == half && (r != 0 || (m & 1)))) m++;
    // value = m 2^drop 2^(-3 DIGIT) 2^(ma - mb); a carry into 2^53 raises the exponent by itself
    const uint64_t bits = ((uint64_t)(mq - 3 * DIGIT + ma - mb + 1022) << 52) + m;
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)bits);
#else
    double out;
    std::memcpy(&out, &bits, 8);
    return out;
#endif
}

}  // namespace scd
