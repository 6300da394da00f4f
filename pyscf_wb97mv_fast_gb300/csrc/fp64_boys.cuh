// Boys function values and the exponential in FP64 at few FP64 instructions.
//
// GB300 issues FP64 at 1/64 of the FP32 rate (2 lanes per clock and SM): in
// the FP64 kernels of this library every other pipe is idle, and a
// conversion, a division or a Horner step on the FP64 pipe is what they
// spend their time on.  So what does not need 53 bits is taken off that
// pipe: the exponential, the argument reduction and the conversions run on the
// integer pipe, the tail of the Taylor series in FP32.
//
// T < 36: Taylor series of F_L about the nearest node T_k = k / 32 (|x| <=
// 1/64), x = T_k - T:
//   F_L(T) = f_0 + x (f_1 + x (f_2 + x (f_3 + tail))),  f_j = F_{L+j}(T_k) / j!
//   tail   = x (f_4 + x (f_5 + x f_6))                              (FP32)
// The FP32 tail is below 2^-28 of F_L, its rounding below 2^-52; the series
// ends with an error below 2^-59.  Then the downward recursion
// F_n = (2T F_{n+1} + e^-T) / (2n + 1).  5 FP64 instructions for F_0, 4 + 2 L
// for F_L: a 1/4 node spacing without the FP32 tail, the factors 1/j in the
// Horner steps and an FP64 exp took 27 and 20 + 3 L more; a series for each
// order from shared rows 6 + 4 L.
// T >= 36: F_0 = sqrt(pi / T) / 2 from an FP32 rsqrt and one third-order
// step, then the upward recursion F_{n+1} = ((2n+1) F_n - e^-T) / (2T) with
// 1/(2T) from the same rsqrt to the last bit (as half the square of T^(-1/2),
// one instruction fewer, its error grew with every n: 2.1e-15 at F_7).
//
// Error of F_0 .. F_L in units of 2^-53, largest and root mean square over
// 60,000 arguments each, against this form with a 1/4 node spacing, a libm exp
// and divisions in FP64 throughout:
//             T < 1           1 .. 36          36 .. 150
//   L = 0   1.3 0.47 (1.1 0.41)   1.9 0.60 (1.9 0.59)   2.2 0.72 (2.7 0.83)
//   L = 1   2.3 0.57 (1.9 0.57)   2.6 0.67 (2.5 0.66)   3.7 0.85 (3.9 0.94)
//   L = 4   2.8 0.76 (2.9 0.76)   5.6 1.06 (5.5 1.07)   8.1 1.48 (8.8 1.57)
//   L = 7   3.2 0.80 (3.0 0.79)   6.6 1.26 (7.4 1.25)    12 2.19 ( 14 2.27)
// (below 1 the coarse table's row T = 0, where F_0 is exactly 1, served T < 1/8;
// the rest is the rounding of the table's entries).
#pragma once
#include <cuda_runtime.h>

#include "cosx_fp64.hpp"

namespace wb {
namespace f64 {

// float -> double on the integer pipe (normal values; zero and subnormals
// give a magnitude below 2^-126)
__device__ __forceinline__ double widen(const float f) {
    const unsigned u = __float_as_uint(f);
    const unsigned hi = (u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + 0x38000000u);
    return __hiloint2double((int)hi, (int)(u << 29));
}

// double -> float, truncated, on the integer pipe; magnitudes below 2^-126
// give zero; what is not below 2^127 (infinities and NaN too) gives some float
// that its caller does not use
__device__ __forceinline__ float narrow(const double d) {
    const unsigned hi = (unsigned)__double2hiint(d);
    const unsigned lo = (unsigned)__double2loint(d);
    const unsigned m = hi & 0x7fffffffu;
    const unsigned u = ((m - 0x38000000u) << 3) | (lo >> 29);
    return __uint_as_float(m < 0x38100000u ? 0u : (hi & 0x80000000u) | u);
}

// double -> float to nearest on the integer pipe, as narrow
__device__ __forceinline__ float narrow_rn(const double d) {
    return narrow(__longlong_as_double(__double_as_longlong(d) + 0x10000000ll));
}

// d / 2 on the integer pipe (zero and subnormals give zero)
__device__ __forceinline__ double half_of(const double d) {
    const unsigned hi = (unsigned)__double2hiint(d);
    return (hi & 0x7fffffffu) < 0x00200000u
               ? 0.0 : __hiloint2double((int)(hi - 0x00100000u), __double2loint(d));
}

// 2 d on the integer pipe (zero and subnormals stay negligible)
__device__ __forceinline__ double twice(const double d) {
    return __hiloint2double(__double2hiint(d) + 0x00100000, __double2loint(d));
}

// exp(-a) for 0 <= a < 70, rounded to FP64, on the integer pipe.  Table-driven
// as P. T. P. Tang, "Table-driven implementation of the exponential function in
// IEEE floating-point arithmetic", ACM TOMS 15 (1989) 144-157, in fixed point:
//   a = n ln2/64 + r, n = rint(64 a / ln2), |r| < 0.00543, a and ln2/64 in
//   units of 2^-56 (ln2/64 with 24 bits more);
//   exp(-r) = 1 + r^2/2 + r^4/24 + r^6/720 - r (1 + r^2/6 + r^4/120), each term
//   with the bits that 2^-62 needs;
//   exp(-a) = 2^-(n >> 6) 2^-((n & 63)/64) exp(-r), the middle factor from a
//   64-entry table of 64-bit fractions.
// At most 0.57 ulp over 3e6 arguments against 64-bit extended precision; the
// same method with FP64 instructions took 12 of them and 1.85 ulp.
__device__ __forceinline__ double exp_neg(const double a,
                                          const unsigned long long* tab) {
    typedef unsigned long long u64;
    const u64 b = (u64)__double_as_longlong(a);
    const int sh = (int)(b >> 52) - 1075 + 56;          // <= 10
    const u64 m = (b & 0xfffffffffffffull) | (1ull << 52);
    const u64 A = sh >= 0 ? m << sh : (sh > -64 ? m >> -sh : 0ull);
    const unsigned n = (unsigned)__float2int_rn(narrow(a) * 92.33248f);
    // n ln2/64 = n (780414346020669 + 15118119 2^-24) 2^-56
    const long long R = (long long)(A - (u64)n * 780414346020669ull -
                                    (((u64)n * 15118119u) >> 24));
    const u64 X = (u64)(R < 0 ? -R : R) << 14;          // |r| 2^70
    const u64 X2 = __umul64hi(X, X);                    // r^2 2^76
    const unsigned x1 = (unsigned)((X + (1ull << 30)) >> 31);      // |r| 2^39
    const unsigned x2 = (unsigned)((X2 + (1ull << 28)) >> 29);     // r^2 2^47
    const u64 p3 = (u64)x2 * x1;                        // |r|^3 2^86
    const u64 x4 = ((u64)x2 * x2) >> 32;                // r^4 2^62
    const u64 odd = ((X + 128) >> 8) + (__umul64hi(p3, 3074457345618258603ull) >> 24) +
                    ((((p3 >> 32) * x2 >> 39) * 35791394ull) >> 32);
    const u64 even = ((X2 + (1ull << 14)) >> 15) + ((x4 * 178956971ull) >> 32) +
                     ((((x4 * x2) >> 47) * 5965232ull) >> 32);
    const u64 Y = (1ull << 62) + even + (R < 0 ? odd : 0ull - odd);
    const u64 P = __umul64hi(tab[n & 63], Y);           // in (0.49, 1.01) 2^61
    const int lz = __clzll((long long)P);
    const u64 q = P << lz;
    const u64 mant = (q >> 11) + ((q >> 10) & 1ull);
    const u64 ef = (u64)(1025 - lz - (int)(n >> 6));
    return __longlong_as_double((long long)((ef << 52) + (mant - (1ull << 52))));
}

// the shared-memory rows of order L: f_0 .. f_3 (FP64), f_4 .. f_6 (FP32) of
// F_L, in an odd stride of 8-byte words (it spreads the rows of a warp over
// the banks), then the table of exp_neg
template<int L>
struct BoysTable {
    static constexpr int kStride = 7;
    static constexpr int kExp = kBoysFineNodes * kStride;
    static constexpr int kBytes = (kExp + 64) * 8;
};

// block-wide copy from the (kBoysFineNodes, kBoysFineCols) table of F_m(T_k)
// and the 64 entries of exp_neg behind it
template<int L>
__device__ __forceinline__ void load_boys(const double* __restrict__ fine, double* tab) {
    typedef BoysTable<L> B;
    static_assert(L + 7 <= kBoysFineCols, "table columns");
    for (int k = threadIdx.x; k < kBoysFineNodes; k += blockDim.x) {
        const double* f = fine + k * kBoysFineCols + L;
        double* row = tab + k * B::kStride;
        float* frow = reinterpret_cast<float*>(row + 4);
        row[0] = f[0];
        row[1] = f[1];
        row[2] = 0.5 * f[2];
        row[3] = f[3] * (1.0 / 6.0);
        frow[0] = (float)(f[4] * (1.0 / 24.0));
        frow[1] = (float)(f[5] * (1.0 / 120.0));
        frow[2] = (float)(f[6] * (1.0 / 720.0));
    }
    for (int k = threadIdx.x; k < 64; k += blockDim.x)
        tab[B::kExp + k] = fine[kBoysFineNodes * kBoysFineCols + k];
}

template<int L>
__device__ __forceinline__ void boys_fast(const double T, const double* tab, double* F) {
    typedef BoysTable<L> B;
    const float tf = narrow(T);
    const unsigned long long* etab =
        reinterpret_cast<const unsigned long long*>(tab + B::kExp);
    // the ranges of T by its high word, unsigned: a NaN of either sign is above
    // all of them (signed, one with its sign bit set would pick a table row)
    const unsigned ht = (unsigned)__double2hiint(T);
    if (ht < 0x40420000u) {                          // T < 36
        const int k = __float2int_rn(tf * 32.0f);
        const double* row = tab + k * B::kStride;
        const float* frow = reinterpret_cast<const float*>(row + 4);
        const double x = widen((float)k * 0.03125f) - T;
        const float xf = narrow_rn(x);
        double s = row[3] + widen(xf * fmaf(xf, fmaf(xf, frow[2], frow[1]), frow[0]));
        s = fma(x, s, row[2]);
        s = fma(x, s, row[1]);
        F[L] = fma(x, s, row[0]);
        if constexpr (L > 0) {
            const double e = exp_neg(T, etab), t2 = twice(T);
#pragma unroll
            for (int n = L - 1; n >= 0; --n) {
                const double v = fma(t2, F[n + 1], e);
                F[n] = n == 0 ? v : v * (1.0 / (2 * n + 1));
            }
        }
    } else {
        double y, h;                                 // T^(-1/2), 1 / (2T)
        if (ht < 0x47e00000u) {                      // T < 2^127
            // T y0^2 = 1 - e, |e| below 2^-21; y0^2 has 48 bits and is exact
            const double y0 = widen(rsqrtf(tf)), q = y0 * y0;
            const double e = fma(-T, q, 1.0);
            y = fma(y0 * e, fma(e, 0.375, 0.5), y0);
            h = half_of(q);
            if constexpr (L > 0) h = fma(h, fma(e, e, e), h);
        } else {
            y = rsqrt(T);                            // infinity: 0, NaN: NaN
            h = half_of(y * y);
        }
        F[0] = 0.88622692545275801365 * y;
        if constexpr (L > 0) {
            const double ex = ht < 0x40518000u ? -exp_neg(T, etab) : 0.0;
#pragma unroll
            for (int n = 0; n < L; ++n) F[n + 1] = fma((double)(2 * n + 1), F[n], ex) * h;
        }
    }
}

}  // namespace f64
}  // namespace wb
