// FP64 products and comparisons on the integer pipe, for kernels that the
// FP64 pipe bounds.
//
// GB300 does two FP64 operations per clock and SM: a product or a comparison
// holds that pipe for 16 cycles per warp.  The product below is the 106-bit
// product of the significands from four 32-bit ones (the schoolbook method,
// Knuth, TAOCP vol. 2, 4.3.1), rounded to nearest even from its exact lower
// half, some 40 instructions of which an SM issues up to four per clock.  A
// kernel with as many sums as products does its sums on the one pipe and its
// products on the other.  Operands or results that are not normal numbers go
// to the built-in operation: the result is the IEEE one, bit for bit.
#pragma once

#include "fp64_div.cuh"

namespace tflows {

// (hi:lo) >> s, its lower word, s in 0..31.
TF_HD uint32_t funnel_right(uint32_t lo, uint32_t hi, int s) {
#if defined(__CUDA_ARCH__)
    return __funnelshift_r(lo, hi, s);
#else
    return s ? (hi << (32 - s)) | (lo >> s) : lo;
#endif
}

// The built-in product.  Out of line: inlined, the compiler makes it a
// predicated instruction, which the FP64 pipe does for every product.
#if defined(__CUDACC__)
__host__ __device__ __noinline__ static double mul_special(double a, double b) { return a * b; }
#else
static double mul_special(double a, double b) { return a * b; }
#endif

// a * b, rounded to nearest even.
TF_HD double mul_rn(double a, double b) {
    const uint64_t ba = div_bits(a), bb = div_bits(b);
    const uint32_t ah = (uint32_t)(ba >> 32), al = (uint32_t)ba, bh = (uint32_t)(bb >> 32), bl = (uint32_t)bb;
    const uint32_t kOne = 1u << 20, kExp = 0x7ff00000u, kFrac = kOne - 1;
    // both from 2^-511 to below 2^513 (the exponent's two upper bits differ),
    // so the product is no subnormal; and it is below 2^1024 when rounded up
    const uint32_t e = (ah & kExp) + (bh & kExp);
    if (!((ah ^ ah << 1) & (bh ^ bh << 1) & 0x40000000u) || e > 3067 * kOne) return mul_special(a, b);
    const uint32_t xh = (ah & kFrac) | kOne, yh = (bh & kFrac) | kOne;
    const uint64_t t0 = (uint64_t)al * bl;
    const uint64_t t1 = (uint64_t)al * yh + (uint32_t)(t0 >> 32);
    const uint64_t t2 = (uint64_t)xh * bl + (uint32_t)t1;
    const uint64_t t3 = (uint64_t)xh * yh + (uint32_t)(t1 >> 32) + (uint32_t)(t2 >> 32);
    // the product is t3 2^64 + (lower words of t2 and t0), 105 or 106 bits
    const uint32_t th = (uint32_t)(t3 >> 32), tl = (uint32_t)t3, w1 = (uint32_t)t2;
    const uint32_t s = th >> 9;  // 106
    const int drop = 20 + (int)s;
    const uint32_t ml = funnel_right(w1, tl, drop), mh = funnel_right(tl, th, drop);
    // what is dropped, from the top, its last bit set for any lower word
    const uint32_t rest = funnel_right(0, w1, drop) | ((uint32_t)t0 != 0);
    const uint32_t up = ((ah ^ bh) & 0x80000000u) + e + (s << 20) - 1024 * kOne;
    return div_value(((uint64_t)(mh + up) << 32 | ml) + (rest + (ml & 1) > 0x80000000u));
}

// 2 x and x / 2: the exponent where it stays a normal one, else the
// subnormal significand shifted (x / 2 rounded to even).
TF_HD double twice(double x) {
    const uint64_t b = div_bits(x), kSign = 1ull << 63, kOne = 1ull << 52;
    const uint32_t e = (uint32_t)(b >> 52) & 0x7ff;
    if (e - 1 < 2045) return div_value(b + kOne);
    if (e == 0) return div_value((b & kSign) | b << 1);
    return div_value(e == 2047 ? b : (b & kSign) | 0x7ff0000000000000ull);
}
TF_HD double half(double x) {
    const uint64_t b = div_bits(x), kSign = 1ull << 63, kOne = 1ull << 52;
    const uint32_t e = (uint32_t)(b >> 52) & 0x7ff;
    if (e - 2 < 2045) return div_value(b - kOne);
    if (e == 2047) return x;
    const uint64_t m = b & ~kSign;  // 2^-1074 units
    return div_value((b & kSign) | ((m >> 1) + (m >> 1 & m & 1)));
}
// 0 + x and 0 - x: x and -x, but a zero is positive.
TF_HD double zero_plus(double x) { return div_value((div_bits(x) << 1) == 0 ? 0 : div_bits(x)); }
TF_HD double zero_minus(double x) {
    return div_value((div_bits(x) << 1) == 0 ? 0 : div_bits(x) ^ 0x8000000000000000ull);
}

// -x where `neg`, else x: in front of a sum that is done once (of a condition
// around two sums the FP64 pipe does both).
TF_HD double signed_by(double x, bool neg) { return div_value(div_bits(x) ^ ((uint64_t)neg << 63)); }

// x > 0 and x < 0 (false for NaN).
TF_HD bool above_zero(double x) { return div_bits(x) - 1 < 0x7ff0000000000000ull; }
TF_HD bool below_zero(double x) { return div_bits(x) - 0x8000000000000001ull < 0x7ff0000000000000ull; }

// a < b.
TF_HD bool less(double a, double b) {
    const int64_t x = (int64_t)div_bits(a), y = (int64_t)div_bits(b);
    const int64_t kInf = 0x7ff0000000000000ll, kAbs = 0x7fffffffffffffffll;
    if ((x & kAbs) > kInf || (y & kAbs) > kInf) return false;
    // negative numbers run backwards; the zeros are equal
    const int64_t kx = x ^ ((x >> 63) & kAbs), ky = y ^ ((y >> 63) & kAbs);
    return kx < ky && ((x | y) & kAbs) != 0;
}

}  // namespace tflows
