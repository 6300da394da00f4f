// The device intrinsics that csrc/fp64_boys.cuh uses, for the host compiler:
// the header's own functions run on the CPU (tests/test_boys_range.py).
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#include <cuda_runtime.h>

template<typename To, typename From> static To bits_as(const From f) {
    To t;
    static_assert(sizeof(To) == sizeof(From), "same size");
    std::memcpy(&t, &f, sizeof(t));
    return t;
}
static int __double2hiint(const double d) { return (int)(bits_as<uint64_t>(d) >> 32); }
static int __double2loint(const double d) { return (int)bits_as<uint64_t>(d); }
static double __hiloint2double(const int hi, const int lo) {
    return bits_as<double>((uint64_t)(uint32_t)hi << 32 | (uint32_t)lo);
}
static long long __double_as_longlong(const double d) { return bits_as<long long>(d); }
static double __longlong_as_double(const long long v) { return bits_as<double>(v); }
static unsigned __float_as_uint(const float f) { return bits_as<unsigned>(f); }
static float __uint_as_float(const unsigned u) { return bits_as<float>(u); }
// saturating, NaN to 0, as the device's conversion
static int __float2int_rn(const float f) {
    return f != f ? 0 : f >= 2147483648.0f ? INT32_MAX : f < -2147483648.0f ? INT32_MIN
                                                       : (int)std::nearbyintf(f);
}
static unsigned long long __umul64hi(const unsigned long long a, const unsigned long long b) {
    return (unsigned long long)((unsigned __int128)a * b >> 64);
}
static int __clzll(const long long v) {
    return v ? __builtin_clzll((unsigned long long)v) : 64;
}
static float rsqrtf(const float x) { return (float)(1.0 / std::sqrt((double)x)); }
static double rsqrt(const double x) { return 1.0 / std::sqrt(x); }
struct { unsigned x = 0; } threadIdx;
struct { unsigned x = 1; } blockDim;
