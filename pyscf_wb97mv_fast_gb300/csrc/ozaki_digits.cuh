// Digit arithmetic of the Ozaki split (ozaki.cu, ozaki_tc.cu): the
// fixed-point conversion of FP64 values to balanced base-2^B digits, and
// the exact int64 combination of FP32 level sums back to FP32 / FP64.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "ozaki.hpp"

namespace wb {

// Fixed-point digits.  A value x with |x| < 2^e becomes the integer
// q = rint(x 2^(W - 1 - e)), W = B S bits, |q| < 2^(W-1), written as
// balanced base-2^B digits q = sum_i d_i 2^(B (S-1-i)), |d_i| <= 2^(B-1) (S =
// 7 digits of B = 6 bits, or 6 of 7), with integer arithmetic only.
constexpr int kW = kOzWidth;
// the exponent of a row or column that holds an infinity or a NaN: its digits
// are zero, so every sum with them is, and a sum of this scale is NaN
constexpr int kNonfinite = 1 << 20;

__device__ __forceinline__ double pow2(int k) {
    // exact 2^k for -1022 <= k <= 1023
    return __longlong_as_double((long long)(1023 + k) << 52);
}

// the high word of |x|: it orders magnitudes as far as their exponents go.
// (The compiler takes a mask of the whole bit pattern for a floating-point
// absolute value and issues it to the FP64 pipe.)
__device__ __forceinline__ unsigned abs_hi(const double x) {
    return (unsigned)__double2hiint(x) & 0x7fffffffu;
}

__device__ __forceinline__ int exp_of_hi(const unsigned hi) {
    if (hi >= 0x7ff00000u) return kNonfinite;
    // smallest e with |x| < 2^e from the high word of |x|, clamped to
    // [-400, 500]: rows whose largest entry is below 2^-400 are zero at this
    // precision, and the clamp keeps every scale factor 2^k of the kernels
    // (|k| <= 2 * 500 + 84) inside the normal FP64 range of pow2()
    const int e = (int)(hi >> 20) - 1022;           // |x| < 2^(ebits-1023+1)
    return e < -400 ? -400 : (e > 500 ? 500 : e);
}

// q = rint(x 2^(W-1-e)) from the bit pattern of x with integer arithmetic:
// |x| = m 2^p (m the 53-bit significand), shifted right with round half to
// even -- the same integer as an exact FP64 scaling followed by
// round-to-nearest, without the FP64 pipe (1/64 of the FP32 rate on GB300)
__device__ __forceinline__ long long fixed_q(double x, int e) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int E = (int)((b >> 52) & 0x7ff);
    unsigned long long m = b & 0xfffffffffffffull;
    int p = -1074;
    if (E) { m |= 1ull << 52; p = E - 1075; }
    const int sh = p + kW - 1 - e;
    unsigned long long q = 0;
    if (m) {
        if (sh >= 0) {
            // only small m (|x| < 2^e keeps q below 2^(W-1))
            q = m << (sh < 11 ? sh : 11);
        } else if (sh > -64) {
            const int r = -sh;
            q = m >> r;
            const unsigned long long rem = m & ((1ull << r) - 1);
            const unsigned long long half = 1ull << (r - 1);
            if (rem > half || (rem == half && (q & 1ull))) ++q;
        }
    }
    return (b >> 63) ? -(long long)q : (long long)q;
}

// fixed_q(x, e) + H sum_i 2^(B i), H = 2^(B-1): with every digit biased by H,
// digit i is the bit field i of the sum, no carries to follow.  The same
// integer as fixed_q with fewer instructions: |x| < 2^e leaves at least 12 bits
// to drop, so the shift goes one way and what it drops decides the rounding.
template<int B, int S>
__device__ __forceinline__ unsigned long long biased_q(const double x, const int e) {
    static_assert(S * B == kW && (B == 6 || B == 7), "42 bits in 6- or 7-bit digits");
    unsigned long long bias = 0;
#pragma unroll
    for (int i = 0; i < S; ++i) bias |= 1ull << (B * i + B - 1);
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    // x = +-m 2^-10 2^(E - 1075), m the significand 10 bits up; q = m >> k
    const int k = 1086 - kW + e - (int)((hi >> 20) & 0x7ffu);
    unsigned long long q = 0;
    if (k < 22) {                           // beyond the clamp of exp_of_hi
        return bias + (unsigned long long)fixed_q(x, e);
    } else if (k < 64) {
        const unsigned long long m =
            ((unsigned long long)(((hi & 0xfffffu) | 0x100000u) << 10 | lo >> 22) << 32) |
            (unsigned long long)(lo << 10);
        q = m >> k;
        const unsigned long long rem = m << (64 - k);
        const unsigned rh = (unsigned)(rem >> 32);
        const unsigned sticky = (rh << 1) | (unsigned)rem | ((unsigned)q & 1u);
        if ((int)rh < 0 && sticky) ++q;
    }
    return (int)hi < 0 ? bias - q : bias + q;
}

// the digits in the low B bits (of the most significant digit, `first`, B + 1) of
// two biased words, as a pair of bf16: 128 + field is the bit pattern 0x4300 +
// field, and subtracting 128 + H from it is exact
template<int B>
__device__ __forceinline__ unsigned field_pair(const unsigned a, const unsigned b,
                                               const bool first) {
    constexpr unsigned H = 1u << (B - 1), M = ((1u << B) - 1u) * 0x10001u;
    unsigned t = __byte_perm(a, b, 0x5410);
    t = first ? t + 0x43004300u : (t & M) | 0x43004300u;    // the first goes up to 2^B
    const unsigned h = (0x4300u + H) * 0x10001u;
    const __nv_bfloat162 d = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&t),
                                     *reinterpret_cast<const __nv_bfloat162*>(&h));
    return *reinterpret_cast<const unsigned*>(&d);
}

// digit i (0 the most significant) of two biased integers
template<int B, int S>
__device__ __forceinline__ unsigned digit_pair(const unsigned long long a,
                                               const unsigned long long b, const int i) {
    const int sh = B * (S - 1 - i);
    return field_pair<B>((unsigned)(a >> sh), (unsigned)(b >> sh), i == 0);
}

// A pair of exponents e, f as the scale 2^(e + f + K), K the constant of a
// product: the high words of two FP64 numbers whose sum is that scale's.
// Neither is negative, and a kNonfinite one is the largest integer, so that
// the saturated sum is then that and the scale a NaN.  One instruction for a
// scale where adding, testing and shifting exponents took five, which k_combine
// shows (192 AOs, 36,369 points, the K product 207 us, with a test 236).
__device__ __forceinline__ int scale_word(const int e, const int K = 0) {
    return e == kNonfinite ? 0x7fffffff : (e + 400 + K) << 20;
}
__device__ __forceinline__ double scale_of(const int we, const int wf) {
    int hi;
    asm("add.sat.s32 %0, %1, %2;" : "=r"(hi) : "r"(we), "r"(wf));
    return __hiloint2double(hi, 0);
}

// RN(v 2^sc) as FP32 from the int64 v with integer arithmetic (one
// rounding); results outside the normal FP32 range take the FP64 path
__device__ __forceinline__ float scaled_ll_to_float(long long v, int sc) {
    if (v == 0) return 0.0f;
    const unsigned long long a = v < 0 ? 0ull - (unsigned long long)v
                                       : (unsigned long long)v;
    const int nb = 64 - __clzll((long long)a);
    unsigned long long q;
    int e2;
    if (nb > 24) {
        int r = nb - 24;
        q = a >> r;
        const unsigned long long rem = a & ((1ull << r) - 1);
        const unsigned long long half = 1ull << (r - 1);
        if (rem > half || (rem == half && (q & 1ull))) ++q;
        if (q == (1ull << 24)) { q >>= 1; ++r; }
        e2 = r;
    } else {
        q = a << (24 - nb);
        e2 = nb - 24;
    }
    const int E = e2 + sc + 23 + 127;
    if (E <= 0 || E >= 255)
        return __double2float_rn((double)v * pow2(sc < -1000 ? -1000 : (sc > 1000 ? 1000 : sc)));
    const unsigned bits = ((unsigned)E << 23) | ((unsigned)q & 0x7fffffu) |
                          (v < 0 ? 0x80000000u : 0u);
    return __uint_as_float(bits);
}

// v 2^sc as FP64: one rounding of v to 53 bits, then an exact scaling (sc
// stays inside pow2's range for the clamped exponents of the split)
__device__ __forceinline__ double scaled_ll_to_double(long long v, int sc) {
    return (double)v * pow2(sc);
}

// the combined value in the output type of an F product (FP32 or FP64); the
// caller replaces it where the scale is not_finite
__device__ __forceinline__ bool not_finite(const int sc) { return sc > kNonfinite / 2; }
template<typename T> __device__ __forceinline__ T scaled_ll_to(long long v, int sc);
template<> __device__ __forceinline__ float scaled_ll_to<float>(long long v, int sc) {
    return scaled_ll_to_float(v, sc);
}
template<> __device__ __forceinline__ double scaled_ll_to<double>(long long v, int sc) {
    return scaled_ll_to_double(v, sc);
}

// a level's contribution to the combined value sum_l C_l 2^(B (S-1-l)), an
// exact int64 (every level, or piece of one, is an integer up to 2^24 in
// magnitude: 32-bit conversion)
template<int B, int S>
__device__ __forceinline__ long long level_term(const int l, const float c) {
    return ((long long)__float2int_rn(c)) << (B * (S - 1 - l));
}

}  // namespace wb
