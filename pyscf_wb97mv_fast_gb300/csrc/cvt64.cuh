// FP32 <-> FP64 conversions on the integer pipe, exactly the hardware's values
// (round to nearest even).  A conversion instruction takes 16 cycles of an
// SM's FP64 pipe for a warp, a dozen integer instructions about 6.  Subnormals,
// infinities and NaN, rare in the arrays these run over, take the instruction.
#pragma once
#include <cuda_runtime.h>

namespace wb {

__device__ __forceinline__ double to_f64(const float f) {
    const unsigned u = __float_as_uint(f), m = u & 0x7fffffffu;
    if (m - 1u < 0x007fffffu || m >= 0x7f800000u) return (double)f;
    const unsigned hi = (u & 0x80000000u) | (m ? (m >> 3) + 0x38000000u : 0u);
    return __hiloint2double((int)hi, (int)(u << 29));
}

__device__ __forceinline__ float to_f32(const double d) {
    const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
    const unsigned m = hi & 0x7fffffffu;
    // magnitudes in [2^-126, 2^128) and zero
    if ((m - 0x38100000u >= 0x0fe00000u) && (m | lo) != 0u) return __double2float_rn(d);
    const unsigned t = lo + 0x0fffffffu + ((lo >> 29) & 1u);
    const unsigned c = m + (t < lo);
    const unsigned u = m ? ((c - 0x38000000u) << 3) | (t >> 29) : 0u;
    return __uint_as_float((hi & 0x80000000u) | u);
}

}  // namespace wb
