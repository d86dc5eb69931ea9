// Correctly rounded FP64 division on the integer and FP32 pipes.
//
// GB300 does two FP64 operations per clock and SM, so a division by
// multiply-add iterations (about ten FP64 operations) holds that pipe for
// some 160 cycles per warp.  This one is long division in three digits of
// about 20 bits, each estimated by one 32-bit multiplication with an FP32
// reciprocal of the divisor and followed by the exact remainder in 64-bit
// integers (the schoolbook method with a large radix and a quotient-digit
// estimate, Knuth, TAOCP vol. 2, 4.3.1).  The last remainder makes the
// quotient exact before it is rounded, so the result is IEEE
// round-to-nearest-even, bit for bit.  Operands or results that are not
// normal numbers (but for 0 / normal) go to the built-in division.
#pragma once

#include <cstdint>

namespace tflows {

#if defined(__CUDACC__)
#define TF_HD __host__ __device__ __forceinline__
#else
#define TF_HD inline
#endif

// An approximation of 1 / x for x in [1, 2), good to a few units in the last place.
TF_HD float div_rcp_estimate(float x) {
#if defined(__CUDA_ARCH__)
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    float r = 1.0f / x;
#ifdef TF_DIV_ESTIMATE_OFF  // (tests: the estimate off by so many units)
    uint32_t b;
    __builtin_memcpy(&b, &r, 4);
    b += TF_DIV_ESTIMATE_OFF;
    __builtin_memcpy(&r, &b, 4);
#endif
    return r;
#endif
}

// The digits: a quotient of the 53-bit significands ma / mb as the integer
// floor(ma 2^54 / mb), with y = 2^83 / mb to within 2^-21 of its value.
// Digit estimates are low by less than 2^9 units (the shifts round down, y
// may be off either way), so the remainders stay below 2^63 and the last one
// within two divisors.
TF_HD uint64_t div_significands(uint64_t ma, uint64_t mb, int32_t y) {
#if defined(__CUDA_ARCH__)
#define TF_MULHI(a, b) __mulhi((a), (b))
#else
#define TF_MULHI(a, b) (int32_t)(((int64_t)(a) * (int64_t)(b)) >> 32)
#endif
    // d1 = q 2^29: (ma 2^-22) y 2^-32 = q 2^29
    const int32_t d1 = TF_MULHI((int32_t)(ma >> 22), y);
    const int64_t r1 = (int64_t)((ma << 29) - (uint64_t)(uint32_t)d1 * mb);
    // d2 = (r1 / mb) 2^20: (r1 2^-31) y 2^-32 = (r1 / mb) 2^20
    const int32_t d2 = TF_MULHI((int32_t)(r1 >> 31), y);
    const int64_t r2 = (int64_t)(((uint64_t)r1 << 20) - (uint64_t)((int64_t)d2 * (int64_t)mb));
    // d3 = (r2 / mb) 2^5: (r2 2^-31) y 2^-32 = (r2 / mb) 2^20
    const int32_t d3 = TF_MULHI((int32_t)(r2 >> 31), y) >> 15;
    int64_t r3 = (int64_t)(((uint64_t)r2 << 5) - (uint64_t)((int64_t)d3 * (int64_t)mb));
    int64_t q = ((int64_t)d1 << 25) + ((int64_t)d2 << 5) + d3;
    if (r3 < 0) { --q; r3 += (int64_t)mb; }
    if (r3 < 0) { --q; r3 += (int64_t)mb; }
    if (r3 >= (int64_t)mb) { ++q; r3 -= (int64_t)mb; }
    if (r3 >= (int64_t)mb) ++q;
    return (uint64_t)q;
#undef TF_MULHI
}

// (An opaque move on the device: the compiler turns tests of a number's bits
// back into FP64 comparisons where it can see where they came from.)
TF_HD uint64_t div_bits(double v) {
#if defined(__CUDA_ARCH__)
    uint64_t b;
    asm("mov.b64 %0, %1;" : "=l"(b) : "d"(v));
    return b;
#else
    uint64_t b;
    __builtin_memcpy(&b, &v, 8);
    return b;
#endif
}
TF_HD double div_value(uint64_t b) {
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)b);
#else
    double v;
    __builtin_memcpy(&v, &b, 8);
    return v;
#endif
}
TF_HD uint32_t div_float_bits(float v) {
#if defined(__CUDA_ARCH__)
    return __float_as_uint(v);
#else
    uint32_t b;
    __builtin_memcpy(&b, &v, 4);
    return b;
#endif
}
TF_HD float div_float(uint32_t b) {
#if defined(__CUDA_ARCH__)
    return __uint_as_float(b);
#else
    float v;
    __builtin_memcpy(&v, &b, 4);
    return v;
#endif
}

// a / b, rounded to nearest even.
TF_HD double div_rn(double a, double b) {
    const uint64_t ba = div_bits(a), bb = div_bits(b);
    const int ea = (int)(ba >> 52) & 0x7ff, eb = (int)(bb >> 52) & 0x7ff;
    const int e = ea - eb + 1023;  // exponent of a quotient >= 1
    // both normal; the quotient normal before and after rounding
    if ((unsigned)(ea - 1) >= 2046u || (unsigned)(eb - 1) >= 2046u || (unsigned)(e - 2) >= 2044u) {
        if ((ba << 1) == 0 && (unsigned)(eb - 1) < 2046u) return div_value((ba ^ bb) & 0x8000000000000000ull);
        return a / b;
    }
    const uint64_t kOne = 1ull << 52, kFrac = kOne - 1;
    const uint64_t ma = (ba & kFrac) | kOne, mb = (bb & kFrac) | kOne;
    // 2^31 / x for the divisor's leading bits x in [1, 2), in (2^30, 2^31)
    const uint32_t rb = div_float_bits(
        div_rcp_estimate(div_float(0x3f800000u | ((uint32_t)(mb >> 29) & 0x7fffffu))));
    const int32_t y = rb >= 0x3f800000u   ? 0x7fffffff
                      : rb < 0x3f000000u ? 1 << 30
                                         : (int32_t)((rb & 0x7fffffu) | 0x800000u) << 7;
    const uint64_t q = div_significands(ma, mb, y);
    // q has 54 or 55 bits; a quotient of two 53-bit significands is never a
    // tie, so its first dropped bit decides the rounding
    const int big = (int)(q >> 54);  // quotient >= 1
    const uint64_t m = q >> big;
    const uint64_t r = ((uint64_t)(e - 2 + big) << 52) + (m >> 1) + (m & 1);
    return div_value(r | ((ba ^ bb) & 0x8000000000000000ull));
}

}  // namespace tflows
