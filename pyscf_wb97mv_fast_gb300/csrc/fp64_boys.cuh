// Boys function values in FP64 at few FP64 instructions.
//
// GB300 issues FP64 at 1/64 of the FP32 rate (2 lanes per clock and SM): in
// the FP64 kernels of this library every other pipe is idle, and a
// conversion, a division or a Horner step on the FP64 pipe is what they
// spend their time on.  So what does not need 53 bits is taken off that
// pipe: the argument reduction and the conversions run on the integer pipe,
// the tail of the Taylor series in FP32.
//
// T < 36: Taylor series about the nearest node T_k = k / 32 (|x| <= 1/64),
// x = T_k - T:
//   F_n(T) = F_n + x (F_{n+1} + x/2 (F_{n+2} + x/3 (F_{n+3} + tail)))
//   tail   = x/4 (F_{n+4} + x/5 (F_{n+5} + x/6 F_{n+6}))          (FP32)
// The FP32 tail is below 2^-28 of F_n, its rounding below 2^-52; the series
// ends with an error below 2^-59.  4 FP64 instructions an order and 2 shared
// by all orders; a 1/4 node spacing without the FP32 tail, the factors 1/j
// in the Horner steps and a downward recursion from an FP64 exp took 27 for
// F_0 and 20 + 3 L more for F_L.
// T >= 36: F_0 = sqrt(pi / T) / 2 from an FP32 rsqrt and one third-order
// step, then the upward recursion F_{n+1} = ((2n+1) F_n - e^-T) / (2T); the
// exponential is below 2e-9 of (2n+1) F_n there (n <= 6), so FP32 serves.
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
// give zero (the callers' values stay below 2^127)
__device__ __forceinline__ float narrow(const double d) {
    const unsigned hi = (unsigned)__double2hiint(d);
    const unsigned lo = (unsigned)__double2loint(d);
    const unsigned m = hi & 0x7fffffffu;
    const unsigned u = ((m - 0x38000000u) << 3) | (lo >> 29);
    return __uint_as_float(m < 0x38100000u ? 0u : (hi & 0x80000000u) | u);
}

// d / 2 on the integer pipe (zero and subnormals give zero)
__device__ __forceinline__ double half_of(const double d) {
    const unsigned hi = (unsigned)__double2hiint(d);
    return (hi & 0x7fffffffu) < 0x00200000u
               ? 0.0 : __hiloint2double((int)(hi - 0x00100000u), __double2loint(d));
}

// the shared-memory rows of order L: F_0 .. F_{L+3} (FP64), then
// F_4 .. F_{L+6} (FP32); an odd stride in 8-byte words spreads the rows of
// a warp over the banks
template<int L>
struct BoysTable {
    static constexpr int kD = L + 4, kF = L + 3;
    static constexpr int kStride = (kD + (kF + 1) / 2) | 1;
    static constexpr int kBytes = kBoysFineNodes * kStride * 8;
};

// block-wide copy of the rows from the (kBoysFineNodes, kBoysFineCols) table
template<int L>
__device__ __forceinline__ void load_boys(const double* __restrict__ fine, double* tab) {
    typedef BoysTable<L> B;
    static_assert(L + 7 <= kBoysFineCols, "table columns");
    for (int k = threadIdx.x; k < kBoysFineNodes; k += blockDim.x) {
        double* row = tab + k * B::kStride;
        float* frow = reinterpret_cast<float*>(row + B::kD);
#pragma unroll
        for (int m = 0; m < L + 7; ++m) {
            const double v = fine[k * kBoysFineCols + m];
            if (m < B::kD) row[m] = v;
            if (m >= 4) frow[m - 4] = (float)v;
        }
    }
}

// F_0 .. F_L from the rows of order LT >= L
template<int L, int LT>
__device__ __forceinline__ void boys_fast(const double T, const double* tab, double* F) {
    typedef BoysTable<LT> B;
    const float tf = narrow(T);
    if (__double2hiint(T) < 0x40420000) {            // T < 36
        const int k = __float2int_rn(tf * 32.0f);
        const double* row = tab + k * B::kStride;
        const float* frow = reinterpret_cast<const float*>(row + B::kD);
        const double x = widen((float)k * 0.03125f) - T;
        const float xf = narrow(x);
        const float x4 = 0.25f * xf, x5 = 0.2f * xf, x6 = xf * (1.0f / 6.0f);
        const double x2 = half_of(x), x3 = x * (1.0 / 3.0);
#pragma unroll
        for (int n = 0; n <= L; ++n) {
            const float tail = x4 * fmaf(x5, fmaf(x6, frow[n + 2], frow[n + 1]), frow[n]);
            double s = row[n + 3] + widen(tail);
            s = fma(x3, s, row[n + 2]);
            s = fma(x2, s, row[n + 1]);
            F[n] = fma(x, s, row[n]);
        }
    } else {
        const double y0 = widen(rsqrtf(tf));
        const double e = fma(-(T * y0), y0, 1.0);
        const double y = fma(y0 * e, fma(e, 0.375, 0.5), y0);
        F[0] = 0.88622692545275801365 * y;
        if constexpr (L > 0) {
            // e^-T = e^-tf (1 - (T - tf)), T - tf from the 29 bits cut off
            const int hi = __double2hiint(T);
            const float cut = (float)(__double2loint(T) & 0x1fffffff) *
                              __uint_as_float((unsigned)min((hi >> 20) - 1023 - 52 + 127, 127) << 23);
            const float ef = tf < 80.0f ? expf(-tf) * (1.0f - cut) : 0.0f;
            const double ex = widen(-ef), h = half_of(y * y);
#pragma unroll
            for (int n = 0; n < L; ++n) F[n + 1] = fma((double)(2 * n + 1), F[n], ex) * h;
        }
    }
}

}  // namespace f64
}  // namespace wb
