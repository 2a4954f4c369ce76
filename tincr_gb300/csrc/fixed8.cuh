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
// Range.  Bounds, digits and results cover all finite doubles; a row with an infinity or a NaN has no digits.
#pragma once

#include <cuda_runtime.h>

namespace tincr {

constexpr int CD_POISON = 1 << 20;   // bound exponent of a row with a non-finite value, which has no digits

// high word of |x|
__device__ __forceinline__ unsigned cd_hi(double x) { return (unsigned)__double2hiint(x) & 0x7fffffffu; }
// ... its last bit set where the low word is not zero (so that a subnormal without a high word
// is not taken for zero; no bound of cd_bound lies between an even word and the next)
__host__ __device__ __forceinline__ unsigned cd_hi_bits(unsigned long long bits) {
    return ((unsigned)(bits >> 32) & 0x7fffffffu) | ((unsigned)bits != 0u ? 1u : 0u);
}
__device__ __forceinline__ unsigned cd_hi_any(double x) { return cd_hi_bits((unsigned long long)__double_as_longlong(x)); }

// E with max |x| < 0.98 * 2^(E+1) from the largest high word (0 for a row of zeros):
// X = x 2^(62-E) then stays in the range of eight balanced digits, 127/255 2^64
__host__ __device__ __forceinline__ int cd_bound(unsigned hi) {
    if (hi >= 0x7ff00000u) return CD_POISON;
    if (hi < 0x00100000u) {   // subnormal: |x| < (hi + 1) 2^-1042
        int e = 0;
        if (hi)
            for (e = -1042; hi; hi >>= 1) ++e;
        return e;
    }
    return (int)(hi >> 20) - ((hi & 0xfffffu) < 0xf5c00u ? 1023 : 1022);
}

// round(x 2^(62-E)) + 0x8080808080808080 (the digits are its bytes less 128), x from its bits.  ANY: subnormal
// x too; otherwise they count as zero (the SCC's matrices are of order one; its splits are bound by these
// instructions).
template <bool ANY>
__host__ __device__ __forceinline__ unsigned long long cd_fixed_bits(unsigned long long bits, int E) {
    const int ex = (int)((bits >> 52) & 0x7ff);
    unsigned long long X = 0;
    if (ANY || ex != 0) {
        const int e1 = ex > 1 ? ex : 1;
        const unsigned long long hidden = ANY && ex == 0 ? 0ull : 1ull << 52;
        const unsigned long long mant = (bits & 0xFFFFFFFFFFFFFull) | hidden;
        const int rs = 1013 + E - (ANY ? e1 : ex);   // X = mant 2^(e1 - 1075 + 62 - E) = mant >> rs < 2^63
        if (rs <= 0) X = mant << (-rs);
        else if (rs <= 54) X = (mant + (1ull << (rs - 1))) >> rs;
    }
    return 0x8080808080808080ull + ((bits >> 63) ? 0ull - X : X);
}
template <bool ANY = false>
__device__ __forceinline__ unsigned long long cd_fixed(double x, int E) {
    return cd_fixed_bits<ANY>((unsigned long long)__double_as_longlong(x), E);
}

// digit p of two values as a pair of bf16 (the first value in the low half): 2^23 + byte has the byte in
// its low mantissa bits, less 2^23 + 128
__device__ __forceinline__ unsigned cd_pair(unsigned long long y0, unsigned long long y1, int p) {
    const unsigned lo = (unsigned)(y0 >> (56 - 8 * p)) & 255u, hi = (unsigned)(y1 >> (56 - 8 * p)) & 255u;
    const float fl = __uint_as_float(0x4B000000u | lo) - 8388736.0f, fh = __uint_as_float(0x4B000000u | hi) - 8388736.0f;
    return __byte_perm(__float_as_uint(fl), __float_as_uint(fh), 0x7632);
}

__host__ __device__ __forceinline__ int cd_clz(unsigned long long x) {   // 64 for zero
#ifdef __CUDA_ARCH__
    return __clzll((long long)x);
#else
    return x ? __builtin_clzll(x) : 64;
#endif
}

// The bits of +-m 2^(ex - 1086) (m with its leading bit set, ex its biased exponent) outside the normal range:
// subnormal results lose their low bits in one rounding, results beyond the largest double are infinite.
__host__ __device__ __noinline__ inline unsigned long long cd_extreme(unsigned long long m, int ex, unsigned long long sign) {
    if (m == 0) return 0ull;
    if (ex > 0) return sign | 0x7ff0000000000000ull;
    const int cut = 12 - ex;   // bits of m below the last one kept
    if (cut > 64) return sign;   // below half of the smallest subnormal
    const unsigned long long q = cut < 64 ? m >> cut : 0ull, rem = m << (64 - cut), half = 0x8000000000000000ull;
    return sign | (q + (rem > half || (rem == half && (q & 1ull)) ? 1ull : 0ull));
}

// The bits of (H 2^32 + L) 2^e rounded to nearest even, in integer arithmetic (an FP64 instruction holds its
// sub-partition for 64 clocks).  |H|, |L| < 2^60.  `outside(m, ex, sign)` gives the bits of a result outside the
// normal range (also of a zero, when e is far out; otherwise zeros are zeros).
template <class F>
__host__ __device__ __forceinline__ unsigned long long cd_value_bits(long long H, long long L, int e, const F &outside) {
    const unsigned long long h = (unsigned long long)(H < 0 ? -H : H);
    const int zh = cd_clz(h) - 2, sh = zh < 32 ? zh : 32;   // |H| 2^sh < 2^62
    const long long T = (long long)((unsigned long long)H << sh) + (L >> (32 - sh));
    const unsigned long long a = (unsigned long long)(T < 0 ? -T : T);
    const int lz = cd_clz(a);
    const unsigned long long m = lz < 64 ? a << lz : 0ull, q = m >> 11, rem = m & 0x7ffull;
    const unsigned long long up = (rem > 0x400ull || (rem == 0x400ull && (q & 1ull))) ? 1ull : 0ull;
    const unsigned long long sign = (unsigned long long)T & 0x8000000000000000ull;
    const int ex = 1023 + 63 - lz + e + 32 - sh;   // biased exponent of the leading bit
    if ((unsigned)(ex - 1) >= 2046u) return outside(m, ex, sign);
    // q holds the hidden bit; a carry of the rounding moves into the exponent (from the last one to infinity)
    return T == 0 ? 0ull : sign | (((unsigned long long)(ex - 1) << 52) + q + up);
}

// The value over the whole range of doubles
__host__ __device__ __forceinline__ unsigned long long cd_value_any(long long H, long long L, int e) {
    return cd_value_bits(H, L, e, [](unsigned long long m, int ex, unsigned long long s) { return cd_extreme(m, ex, s); });
}
// ... where the operands are of order one (the SCC, 3 % faster so on decacene): results below the normal range
// are zero, beyond it NaN
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
