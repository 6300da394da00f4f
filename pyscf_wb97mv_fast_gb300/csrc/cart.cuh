// Cartesian components of a shell (libcint order) and the nonzero pattern of
// the Cartesian -> spherical transforms, at compile time.
#pragma once

namespace wb {
namespace f64 {

constexpr __host__ __device__ int ncart_c(int l) { return (l + 1) * (l + 2) / 2; }
// Cartesian exponents of component c of shell l (libcint order)
constexpr __host__ __device__ int cx(int l, int c) {
    int n = 0;
    for (int x = l; x >= 0; --x)
        for (int y = l - x; y >= 0; --y) {
            if (n == c) return x;
            ++n;
        }
    return 0;
}
constexpr __host__ __device__ int cy(int l, int c) {
    int n = 0;
    for (int x = l; x >= 0; --x)
        for (int y = l - x; y >= 0; --y) {
            if (n == c) return y;
            ++n;
        }
    return 0;
}
constexpr __host__ __device__ int cz(int l, int c) { return l - cx(l, c) - cy(l, c); }
// position of the Cartesian component x^i y^j z^(l-i-j) (libcint order)
constexpr __host__ __device__ int cidx(int l, int i, int j) {
    return (l - i) * (l - i + 1) / 2 + (l - i - j);
}
// whether Cartesian component c enters the real solid harmonic m = -l + s
constexpr __host__ __device__ bool c2s_nz(int l, int c, int s) {
    // one bit per component: 6 bits a column (d), 10 bits a column (f)
    return l <= 1 ? c == s
           : l == 2 ? ((0x02ull | 0x10ull << 6 | 0x29ull << 12 | 0x04ull << 18 |
                        0x09ull << 24) >> (6 * s + c)) & 1
           : s < 4 ? ((0x042ull | 0x010ull << 10 | 0x142ull << 20 | 0x284ull << 30) >>
                      (10 * s + c)) & 1
                   : ((0x029ull | 0x084ull << 10 | 0x009ull << 20) >> (10 * (s - 4) + c)) & 1;
}

}  // namespace f64
}  // namespace wb
