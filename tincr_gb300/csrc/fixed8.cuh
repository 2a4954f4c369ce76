// Fixed-point digits of FP64 values for exact tensor-core products.
//
// Digits.  A value x of a row with |x| < 0.98 * 2^(E+1) is the integer X = round(x 2^(62-E)) in eight
// balanced digits of 8 bits, X = sum_s d_s 2^(8 (7-s)), -128 <= d_s <= 127 (exact in bf16): the bytes
// of X + 0x8080808080808080, less 128.  A level sum over a chunk of 128 k is at most 8 * 128 * 2^14 =
// 2^24, exact in an FP32 accumulator.  The operands carry 62 to 63 bits below the row's largest value
// and the dropped levels s + t >= 8, products of balanced digits and so of either sign, are near
// 2^-64 of the row maxima per term: a result is the rounded exact sum but for rows whose largest
// value is hundreds of times above the others.
// The value of a product is sum over levels g = s + t <= 7 of G_g 2^(8 (14 - g)) 2^(Ea + Eb - 124) with the level
// sums G_g of the digit products, i.e. (H 2^32 + L) 2^(Ea + Eb - 68) with H = sum_{g<4} G_g 2^(8 (3 - g)) and
// L = sum_{g>=4} G_g 2^(8 (7 - g)).
#pragma once

#include <cuda_runtime.h>

namespace tincr {

constexpr int CD_POISON = 1 << 20;   // bound exponent of a row with a non-finite value: its results are NaN

// high word of |x|
__device__ __forceinline__ unsigned cd_hi(double x) { return (unsigned)__double2hiint(x) & 0x7fffffffu; }

// E with max |x| < 0.98 * 2^(E+1) from the largest high word (0 for a row of zeros or subnormals):
// X = x 2^(62-E) then stays in the range of eight balanced digits, 127/255 2^64
__device__ __forceinline__ int cd_bound(unsigned hi) {
    if (hi >= 0x7ff00000u) return CD_POISON;
    if (hi < 0x00100000u) return 0;
    return (int)(hi >> 20) - ((hi & 0xfffffu) < 0xf5c00u ? 1023 : 1022);
}

// round(x 2^(62-E)) + 0x8080808080808080 (the digits are its bytes less 128)
__device__ __forceinline__ unsigned long long cd_fixed(double x, int E) {
    const unsigned long long bits = (unsigned long long)__double_as_longlong(x);
    const int ex = (int)((bits >> 52) & 0x7ff);
    unsigned long long X = 0;
    if (ex != 0) {
        const unsigned long long mant = (bits & 0xFFFFFFFFFFFFFull) | (1ull << 52);
        const int rs = 1013 + E - ex;   // X = mant 2^(ex - 1075 + 62 - E) = mant >> rs, rs >= -10
        if (rs <= 0) X = mant << (-rs);
        else if (rs <= 54) X = (mant + (1ull << (rs - 1))) >> rs;
    }
    return 0x8080808080808080ull + ((bits >> 63) ? 0ull - X : X);
}


// digit p of two values as a pair of bf16 (the first value in the low half): 2^23 + byte has the byte in
// its low mantissa bits, less 2^23 + 128
__device__ __forceinline__ unsigned cd_pair(unsigned long long y0, unsigned long long y1, int p) {
    const unsigned lo = (unsigned)(y0 >> (56 - 8 * p)) & 255u, hi = (unsigned)(y1 >> (56 - 8 * p)) & 255u;
    const float fl = __uint_as_float(0x4B000000u | lo) - 8388736.0f, fh = __uint_as_float(0x4B000000u | hi) - 8388736.0f;
    return __byte_perm(__float_as_uint(fl), __float_as_uint(fh), 0x7632);
}

// (H 2^32 + L) 2^e rounded to nearest even, in integer arithmetic (an FP64 instruction holds its
// sub-partition for 64 clocks).  |H|, |L| < 2^60; results below the normal range are zero.
__device__ __forceinline__ double cd_value(long long H, long long L, int e) {
    const int sh = min(32, __clzll((unsigned long long)(H < 0 ? -H : H)) - 2);   // |H| 2^sh < 2^62
    const long long T = (H << sh) + (L >> (32 - sh));
    if (T == 0) return 0.0;
    const unsigned long long a = (unsigned long long)(T < 0 ? -T : T);
    const int lz = __clzll(a);
    const unsigned long long m = a << lz, q = m >> 11, rem = m & 0x7ffull;
    const unsigned long long up = (rem > 0x400ull || (rem == 0x400ull && (q & 1ull))) ? 1ull : 0ull;
    const int ex = 1023 + 63 - lz + e + 32 - sh;   // biased exponent of the leading bit
    if (ex <= 0) return 0.0;
    if (ex >= 2046) return __longlong_as_double(0x7ff8000000000000ll);
    const unsigned long long bits = ((unsigned long long)(ex - 1) << 52) + q + up;
    return __longlong_as_double((long long)(bits | ((unsigned long long)T & 0x8000000000000000ull)));
}

}  // namespace tincr
