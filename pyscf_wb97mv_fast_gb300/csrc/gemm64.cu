// FP64 GEMMs of the FP64 flows on the bf16 tensor cores.
//
// GB300's FP64 rate is 1.2 TFLOP/s, DGEMM included (0.95 measured), so in an
// FP64 Fock build, in VV10 and in the gradient the products with D and X
// outweighed the kernels between them.  They run here as an Ozaki split
// (K. Ozaki et al., Numer. Algorithms 59 (2012) 95-118), as the 42-bit split
// of ozaki.cu, but wide enough to lose nothing of FP64: S balanced digits of B = 7
// bits below the largest entry of the row (point) or column (AO), S = 10 (W = 70
// bits) for F and 9 (63 bits) for K, against the 53 of a double.  An entry is cut
// where it is below 2^(53 - W) of that largest one, and then by 2^-W of it; the
// dropped products (digit levels i + j >= S) are as small.  So an entry of the
// result is exact to some 2^-68 (F) or 2^-61 (K) of the product of the row's and
// the column's largest entries, and its relative error grows as it falls below
// them.  K's rows are the 512 points of a chunk of one AO, which share their
// magnitude; F's are all AOs at one point, from a nucleus to far away, and take
// the tenth digit (with nine its entries below 1e-6 of the maxima were up to 40
// times further off than DGEMM's).
//
// Relative error against extended precision, root mean square over the entries
// of each size (of the maxima for F, of the largest K), on converged densities,
// FP64 AO values and quadrature weights; in brackets cuBLAS DGEMM:
//                     2-norm             1e-2 and more      1e-4 .. 1e-2
//   8 waters F    4.4e-17 (1.9e-16)   4.7e-17 (4.2e-16)   5.7e-17 (3.7e-15)
//   C6H14/TZ F    4.0e-17 (7.1e-16)   4.7e-17 (2.1e-15)   5.8e-17 (3.7e-14)
//   8 waters K    9.9e-17 (7.4e-16)   1.3e-16 (1.1e-15)   3.8e-16 (8.4e-15)
//   C6H14/TZ K    7.4e-17 (6.7e-16)   1.0e-16 (9.2e-16)   3.7e-16 (4.6e-15)
//                   1e-6 .. 1e-4        1e-9 .. 1e-6       1e-12 .. 1e-9
//   8 waters F    1.7e-15 (1.7e-14)   7.6e-14 (5.1e-13)
//   C6H14/TZ F    2.0e-15 (2.2e-12)   4.4e-12 (1.4e-10)   2.0e-10 (9.9e-10)
//   8 waters K    2.5e-16 (3.2e-15)   1.9e-16 (2.3e-15)   1.3e-15 (3.9e-14)
//   C6H14/TZ K    3.3e-15 (5.6e-14)   1.3e-14 (9.1e-13)
//
// Exactness: digits are at most 64 in magnitude (exact in bf16), products
// 2^12, so a bf16 GEMM of at most kPiece = 4096 terms has only integers up to
// 2^24 as partial sums: FP32 accumulation is exact in any order.  Level l =
// i + j is the product of the first (l + 1) slices of A with the last (l + 1)
// slices of B, cut every 4096 terms into pieces; pieces and levels are added
// as integers and rounded once.  55 and 45 slice products, so 55/2 and 45/2 x the
// flops of a DGEMM at some 1500 times its rate.
//
// Measured against cuBLAS DGEMM, 192 AOs x 70,478 points: F 4.8 -> 0.68 ms (nine
// digits 0.61), K 5.0 -> 0.76 ms; below some 64 AOs and 10,000 points the fixed
// 0.11 ms of launches is about the DGEMM's time, so there is no other path.
//
// Point tiles (F) and groups of chunks (K) bound the workspace: 65,536 points and
// 128 chunks up to some 700 AOs (3.7 GB at 648), fewer above, where their digits
// and level planes would pass 4 GiB (at 4,000 AOs 4,128 points and 6 chunks).
// A row or column with an infinity or a NaN gives NaN, as FP64 arithmetic
// mostly would; magnitudes from subnormal to the largest double are taken.
#include <cuda_bf16.h>

#include <algorithm>

#include "gemm64.hpp"
#include "launch.hpp"
#include "ozaki_digits.cuh"

namespace wb {
namespace {

constexpr int kBits = 7;
constexpr int kSF = 10, kSK = 9;         // digits of the F and the K product
constexpr int kPiece = 4096;             // terms of an exact FP32 sum
constexpr int kKc = 512;                 // points per chunk of the K product
constexpr int kGroup = 128;              // chunks in flight
constexpr int64_t kTile = 65536;         // points per tile of the F product
constexpr size_t kBudget = (size_t)4 << 30;     // bytes of either

size_t al(size_t x) { return (x + 255) & ~(size_t)255; }
// slices are padded to 8 entries: cuBLAS needs 16-byte rows for its
// tensor-memory kernels (unaligned ones ran on mma.sync kernels at a third of
// the rate)
int pad8(int n) { return (n + 7) & ~7; }
int pieces(int terms) { return (terms + kPiece - 1) / kPiece; }
int planes(int S, int inner) {
    int n = 0;
    for (int l = 0; l < S; ++l) n += pieces((l + 1) * inner);
    return n;
}
int f_planes(int np) { return planes(kSF, np); }
int k_planes() { return planes(kSK, kKc); }

// e with |x| < 2^e from the high word of the largest |x|
__device__ __forceinline__ int exponent_of(const unsigned hi) {
    const int E = (int)(hi >> 20);
    if (E == 0x7ff) return kNonfinite;
    return E ? E - 1022 : -1022;
}

// q = rint(x 2^(7 S - 1 - e)), |x| < 2^e, with 64 added to each of its S digits,
// which are then bit fields of the sum: nine fill 63 bits, the tenth goes on in
// a second word
template<int S> struct Biased;
template<> struct Biased<9> {
    unsigned long long q;
    __device__ __forceinline__ unsigned field(const int k) const {
        return (unsigned)(q >> (kBits * k));
    }
};
template<> struct Biased<10> {
    unsigned long long q;               // digits 0 .. 8 and the lowest bit of the last
    unsigned top;                       // its other bits
    __device__ __forceinline__ unsigned field(const int k) const {
        return k < 9 ? (unsigned)(q >> (kBits * k)) : (unsigned)(q >> 63) | top << 1;
    }
};

template<int S>
__device__ __forceinline__ Biased<S> biased(const double x, const int e) {
    static_assert(S == 9 || S == 10, "one or two words");
    unsigned __int128 bias = 0;
#pragma unroll
    for (int i = 0; i < S; ++i) bias |= (unsigned __int128)64 << (kBits * i);
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const int E = (int)((hi >> 20) & 0x7ffu);
    // |x| = m 2^-10 2^(E - 1075), m the significand 10 bits up, so q = (m << a) >> k,
    // a the bits beyond 63, with 1 <= k; a subnormal x has no leading one
    const unsigned top = E ? (hi & 0xfffffu) | 0x100000u : hi & 0xfffffu;
    constexpr int a = kBits * S - 63;
    const int k = max(1023 + e - max(E, 1), 1);
    unsigned long long q = 0;
    unsigned qt = 0;
    if (e != kNonfinite && k < 64 + a) {
        const unsigned long long m = ((unsigned long long)(top << 10 | lo >> 22) << 32) |
                                     (unsigned long long)(lo << 10);
        if (a == 0 || k > a) {
            const int r = k - a;                // 1 .. 63 bits to drop
            q = m >> r;
            const unsigned long long rem = m << (64 - r);
            const unsigned rh = (unsigned)(rem >> 32);
            const unsigned sticky = (rh << 1) | (unsigned)rem | ((unsigned)q & 1u);
            if ((int)rh < 0 && sticky) ++q;
        } else {
            q = m << (a - k);                   // the ten low bits of m are zero
            qt = a == k ? 0u : (unsigned)(m >> (64 - (a - k)));
        }
    }
    Biased<S> b;
    if constexpr (S == 9) {
        b.q = (int)hi < 0 ? (unsigned long long)bias - q : (unsigned long long)bias + q;
    } else {
        const unsigned __int128 v = (unsigned __int128)qt << 64 | q;
        const unsigned __int128 t = (int)hi < 0 ? bias - v : bias + v;
        b.q = (unsigned long long)t;
        b.top = (unsigned)(t >> 64);
    }
    return b;
}

// digit i (0 the most significant) of two values as a pair of bf16 (digit_pair of
// ozaki_digits.cuh)
template<int S>
__device__ __forceinline__ unsigned digits(const Biased<S>& a, const Biased<S>& b,
                                           const int i) {
    return field_pair<kBits>(a.field(S - 1 - i), b.field(S - 1 - i), i == 0);
}

// RN(v 2^sc), v = hi 2^up + lo, with integer arithmetic (the conversions
// would be FP64-pipe instructions)
__device__ __forceinline__ double round_sum(const long long hi, const long long lo,
                                            const int up, const int sc) {
    const __int128 v = ((__int128)hi << up) + lo;
    if (v == 0) return 0.0;
    const unsigned __int128 a = v < 0 ? (unsigned __int128)0 - (unsigned __int128)v
                                      : (unsigned __int128)v;
    const unsigned long long ah = (unsigned long long)(a >> 64), alo = (unsigned long long)a;
    const int nb = ah ? 128 - __clzll((long long)ah) : 64 - __clzll((long long)alo);
    const int r = nb - 53;
    unsigned long long q;
    if (r > 0) {
        q = (unsigned long long)(a >> r);
        const unsigned __int128 rem = a & (((unsigned __int128)1 << r) - 1);
        const unsigned __int128 half = (unsigned __int128)1 << (r - 1);
        if (rem > half || (rem == half && (q & 1ull))) ++q;
    } else {
        q = alo << -r;
    }
    const int E = r + sc + 52 + 1023;           // exponent field of q = 2^52
    double out;
    if (E >= 1 && E <= 2045)
        out = __longlong_as_double((long long)(((unsigned long long)E << 52) +
                                               (q - (1ull << 52))));
    else
        out = scalbn((double)q, max(-4000, min(4000, r + sc)));
    return v < 0 ? -out : out;
}

// integer sums of the levels: hi = levels 0 .. 4, lo = 5 .. S - 1, so that the
// value is (hi 2^(7 (S - 5)) + lo) 2^(sc)
template<int S>
struct LevelSum {
    long long hi = 0, lo = 0;
    __device__ __forceinline__ void add(const int l, const float c) {
        const long long t = (long long)__float2int_rn(c);
        if (l <= 4) hi += t << (kBits * (4 - l));
        else lo += t << (kBits * (S - 1 - l));
    }
    // x y = 2^(ex + ey - 2 (7 S - 1) + 7 (S - 1)) sum_l C_l 2^(7 (S - 1 - l))
    __device__ __forceinline__ double finish(const int ex, const int ey) const {
        if (ex == kNonfinite || ey == kNonfinite)
            return __longlong_as_double(0x7ff8000000000000ll);
        return round_sum(hi, lo, kBits * (S - 5),
                         ex + ey - 2 * (kBits * S - 1) + kBits * (S - 1));
    }
};

// exponent of each point's largest |X(l, g)|, g0 <= g < g0 + n
__global__ void point_exponents_kernel(const double* __restrict__ X, const int nao,
                                       const int64_t ld, const int n, int* __restrict__ e) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n) return;
    unsigned m = 0;
    int l = 0;
    for (; l + 8 <= nao; l += 8) {
        double b[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) b[u] = __ldg(X + (int64_t)(l + u) * ld + g);
#pragma unroll
        for (int u = 0; u < 8; ++u) m = max(m, abs_hi(b[u]));
    }
    for (; l < nao; ++l) m = max(m, abs_hi(__ldg(X + (int64_t)l * ld + g)));
    e[g] = exponent_of(m);
}

// A (n x S np, column-major): column i np + l = digit i of X(l, :), zero for
// l >= nao; one thread per (l, two points)
__global__ void slice_points_kernel(const double* __restrict__ X, const int nao, const int np,
                                    const int64_t ld, const int n, const int* __restrict__ e,
                                    __nv_bfloat16* __restrict__ A) {
    const int l = blockIdx.y;
    const int g = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
    if (g >= n) return;                         // n is even
    double2 x = make_double2(0.0, 0.0);
    if (l < nao) x = *reinterpret_cast<const double2*>(X + (int64_t)l * ld + g);
    const Biased<kSF> q0 = biased<kSF>(x.x, e[g]), q1 = biased<kSF>(x.y, e[g + 1]);
#pragma unroll
    for (int i = 0; i < kSF; ++i)
        *reinterpret_cast<unsigned*>(A + ((int64_t)i * np + l) * n + g) = digits(q0, q1, i);
}

// the largest of a block of 256 threads
__device__ __forceinline__ unsigned block_max(unsigned m) {
    __shared__ unsigned red[8];
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 8; ++j) m = max(m, red[j]);
    __syncthreads();
    return m;
}

// B (S np x nao, column-major): row (S - 1 - i) np + l of column mu = digit i
// of QD(l, mu); one block of 256 threads per column
__global__ void __launch_bounds__(256)
slice_matrix_kernel(const double* __restrict__ QD, const int nao, const int np,
                    int* __restrict__ e, __nv_bfloat16* __restrict__ B) {
    const int mu = blockIdx.x;
    unsigned m = 0;
    for (int l = threadIdx.x; l < nao; l += 256) m = max(m, abs_hi(QD[(int64_t)l * nao + mu]));
    const int ec = exponent_of(block_max(m));
    if (threadIdx.x == 0) e[mu] = ec;
    for (int l = threadIdx.x; l < np; l += 256) {
        const Biased<kSF> q = biased<kSF>(l < nao ? QD[(int64_t)l * nao + mu] : 0.0, ec);
#pragma unroll
        for (int i = 0; i < kSF; ++i)
            B[((int64_t)mu * kSF + (kSF - 1 - i)) * np + l] =
                __ushort_as_bfloat16((unsigned short)digits(q, q, i));
    }
}

// F[mu][g] from the level planes C (plane, mu, n)
__global__ void combine_points_kernel(const float* __restrict__ C, const int nao, const int np,
                                      const int64_t ld, const int n,
                                      const int* __restrict__ ep, const int* __restrict__ ec,
                                      double* __restrict__ F) {
    const int mu = blockIdx.y;
    const int g = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
    if (g >= n) return;
    const int64_t plane = (int64_t)nao * n;
    const float* c = C + (int64_t)mu * n + g;
    LevelSum<kSF> v0, v1;
#pragma unroll
    for (int l = 0; l < kSF; ++l)
        for (int left = (l + 1) * np; left > 0; left -= kPiece, c += plane) {
            const float2 t = __ldg(reinterpret_cast<const float2*>(c));
            v0.add(l, t.x);
            v1.add(l, t.y);
        }
    const int e = ec[mu];
    *reinterpret_cast<double2*>(F + (int64_t)mu * ld + g) =
        make_double2(v0.finish(ep[g], e), v1.finish(ep[g + 1], e));
}

// Digits of one chunk's column of X (ascending slices) or of w o G
// (descending): out (chunk, column, S, kKc), columns past nao zero.  One block
// of 256 threads, two points a thread, per (chunk, column).
template<bool WG>
__global__ void __launch_bounds__(256)
slice_chunk_kernel(const double* __restrict__ X, const double* __restrict__ w, const int nao,
                   const int64_t ld, const int64_t npts, const int64_t g_base,
                   int* __restrict__ e, __nv_bfloat16* __restrict__ out) {
    const int np = gridDim.y, col = blockIdx.y;
    const int64_t slot = (int64_t)blockIdx.x * np + col;
    const int k = 2 * threadIdx.x;
    const int64_t g = g_base + (int64_t)blockIdx.x * kKc + k;
    double x0 = 0.0, x1 = 0.0;
    if (col < nao) {
        const double* x = X + (int64_t)col * ld;
        if (g < npts) x0 = WG ? w[g] * x[g] : x[g];
        if (g + 1 < npts) x1 = WG ? w[g + 1] * x[g + 1] : x[g + 1];
    }
    const int ee = exponent_of(block_max(max(abs_hi(x0), abs_hi(x1))));
    if (threadIdx.x == 0) e[slot] = ee;
    const Biased<kSK> q0 = biased<kSK>(x0, ee), q1 = biased<kSK>(x1, ee);
    __nv_bfloat16* o = out + slot * kSK * kKc + k;
#pragma unroll
    for (int i = 0; i < kSK; ++i)
        *reinterpret_cast<unsigned*>(o + (WG ? kSK - 1 - i : i) * kKc) = digits(q0, q1, i);
}

// K (+)= the chunks of one group, in chunk order: C (plane, chunk, np x np)
__global__ void combine_chunks_kernel(const float* __restrict__ C, const int nao, const int np,
                                      const int nchunk, const int* __restrict__ ex,
                                      const int* __restrict__ eg, const int add,
                                      double* __restrict__ K) {
    const int64_t nn = (int64_t)np * np;
    const int64_t plane = nn * nchunk;
    const int mu = blockIdx.x * blockDim.x + threadIdx.x, nu = blockIdx.y;
    if (mu >= nao) return;
    double acc = 0.0;
#pragma unroll 2
    for (int c = 0; c < nchunk; ++c) {
        const float* p = C + (int64_t)c * nn + (int64_t)nu * np + mu;
        LevelSum<kSK> v;
#pragma unroll
        for (int l = 0; l < kSK; ++l)
#pragma unroll
            for (int left = (l + 1) * kKc; left > 0; left -= kPiece, p += plane)
                v.add(l, __ldg(p));
        acc += v.finish(ex[c * np + mu], eg[c * np + nu]);
    }
    const int64_t o = (int64_t)mu * nao + nu;
    K[o] = add ? K[o] + acc : acc;
}

// points of a tile and chunks of a group within the budget
int64_t tile_points(int nao) {
    const size_t np = pad8(nao);
    const size_t per = sizeof(int) + 2 * kSF * np + sizeof(float) * f_planes((int)np) * nao;
    const size_t qd = 2 * kSF * np * nao;               // the digits of QD
    const size_t left = kBudget > qd ? kBudget - qd : 0;
    return std::min(kTile, std::max<int64_t>((int64_t)(left / per) / 32 * 32, 32));
}
int group_chunks(int nao) {
    const size_t np = pad8(nao);
    const size_t per = 2 * (sizeof(int) * np + 2 * kSK * kKc * np) +
                       sizeof(float) * k_planes() * np * np;
    return (int)std::min<size_t>(kGroup, std::max<size_t>(kBudget / per, 1));
}

size_t f_bytes(int nao, int64_t ld) {
    const size_t np = pad8(nao), n = (size_t)std::min(ld, tile_points(nao));
    return al(sizeof(int) * n) + al(sizeof(int) * nao) + al(2 * kSF * np * n) +
           al(2 * kSF * np * nao) + al(sizeof(float) * f_planes((int)np) * nao * n);
}

size_t k_bytes(int nao, int64_t ld) {
    const size_t np = pad8(nao);
    const size_t nc = (size_t)std::min<int64_t>((ld + kKc - 1) / kKc, group_chunks(nao));
    return 2 * (al(sizeof(int) * nc * np) + al(2 * kSK * kKc * nc * np)) +
           al(sizeof(float) * k_planes() * nc * np * np);
}

}  // namespace

size_t gemm64_bytes(int nao, int64_t ld) { return std::max(f_bytes(nao, ld), k_bytes(nao, ld)); }

int gemm64_f_launches(int nao, int64_t ld) {
    const int64_t tile = tile_points(nao);
    return 1 + (int)((ld + tile - 1) / tile) * (3 + f_planes(pad8(nao)));
}
int gemm64_k_launches(int nao, int64_t npts) {
    const int64_t group = (int64_t)kKc * group_chunks(nao);
    return (int)((npts + group - 1) / group) * (3 + k_planes());
}

#define G64_CUBLAS(call)                                          \
    do {                                                          \
        cublasStatus_t st_ = (call);                              \
        if (st_ != CUBLAS_STATUS_SUCCESS) return (int)st_ + 1000; \
    } while (0)
#define G64_CUDA(call)                       \
    do {                                     \
        cudaError_t e_ = (call);             \
        if (e_ != cudaSuccess) return (int)e_; \
    } while (0)

int gemm64_f(cublasHandle_t hb, const double* X, const double* QD, int nao, int64_t ld,
             double* F, void* ws, cudaStream_t s) {
    const int np = pad8(nao);
    const int64_t tile = tile_points(nao), nmax = std::min(ld, tile);
    char* p = static_cast<char*>(ws);
    int* ep = reinterpret_cast<int*>(p); p += al(sizeof(int) * nmax);
    int* ec = reinterpret_cast<int*>(p); p += al(sizeof(int) * nao);
    __nv_bfloat16* A = reinterpret_cast<__nv_bfloat16*>(p);
    p += al((size_t)2 * kSF * np * nmax);
    __nv_bfloat16* B = reinterpret_cast<__nv_bfloat16*>(p);
    p += al((size_t)2 * kSF * np * nao);
    float* C = reinterpret_cast<float*>(p);
    slice_matrix_kernel<<<nao, 256, 0, s>>>(QD, nao, np, ec, B);
    G64_CUDA(cudaGetLastError());
    const float one = 1.0f, zero = 0.0f;
    for (int64_t g = 0; g < ld; g += tile) {
        const int n = (int)std::min(tile, ld - g);
        const dim3 grid((n / 2 + 255) / 256, np);
        point_exponents_kernel<<<(n + 255) / 256, 256, 0, s>>>(X + g, nao, ld, n, ep);
        G64_CUDA(cudaGetLastError());
        slice_points_kernel<<<grid, 256, 0, s>>>(X + g, nao, np, ld, n, ep, A);
        G64_CUDA(cudaGetLastError());
        float* c = C;
        for (int l = 0; l < kSF; ++l)
            for (int k0 = 0; k0 < (l + 1) * np; k0 += kPiece, c += (size_t)nao * n)
                G64_CUBLAS(cublasGemmEx(hb, CUBLAS_OP_N, CUBLAS_OP_N, n, nao,
                                        std::min(kPiece, (l + 1) * np - k0), &one,
                                        A + (size_t)k0 * n, CUDA_R_16BF, n,
                                        B + (size_t)(kSF - 1 - l) * np + k0, CUDA_R_16BF,
                                        kSF * np, &zero, c, CUDA_R_32F, n,
                                        CUBLAS_COMPUTE_32F, CUBLAS_GEMM_DEFAULT));
        combine_points_kernel<<<dim3((n / 2 + 255) / 256, nao), 256, 0, s>>>(
            C, nao, np, ld, n, ep, ec, F + g);
        G64_CUDA(cudaGetLastError());
    }
    return 0;
}

int gemm64_k(cublasHandle_t hb, const double* X, const double* G, const double* w, int nao,
             int64_t ld, int64_t npts, int accumulate, double* K, void* ws, cudaStream_t s) {
    const int np = pad8(nao);
    const int nchunk = (int)((npts + kKc - 1) / kKc);
    const int group = group_chunks(nao);
    const int gmax = (int)std::min<int64_t>((ld + kKc - 1) / kKc, group);
    char* p = static_cast<char*>(ws);
    int* ex = reinterpret_cast<int*>(p); p += al(sizeof(int) * (size_t)gmax * np);
    int* eg = reinterpret_cast<int*>(p); p += al(sizeof(int) * (size_t)gmax * np);
    __nv_bfloat16* A = reinterpret_cast<__nv_bfloat16*>(p);
    p += al((size_t)2 * kSK * kKc * gmax * np);
    __nv_bfloat16* B = reinterpret_cast<__nv_bfloat16*>(p);
    p += al((size_t)2 * kSK * kKc * gmax * np);
    float* C = reinterpret_cast<float*>(p);
    const float one = 1.0f, zero = 0.0f;
    const long long slab = (long long)kSK * kKc * np, nn = (long long)np * np;
    for (int c0 = 0; c0 < nchunk; c0 += group) {
        const int nc = std::min(group, nchunk - c0);
        const dim3 grid(nc, np);
        slice_chunk_kernel<false><<<grid, 256, 0, s>>>(X, w, nao, ld, npts, (int64_t)c0 * kKc,
                                                       ex, A);
        G64_CUDA(cudaGetLastError());
        slice_chunk_kernel<true><<<grid, 256, 0, s>>>(G, w, nao, ld, npts, (int64_t)c0 * kKc,
                                                      eg, B);
        G64_CUDA(cudaGetLastError());
        float* c = C;
        for (int l = 0; l < kSK; ++l)
            for (int k0 = 0; k0 < (l + 1) * kKc; k0 += kPiece, c += (size_t)nc * nn)
                G64_CUBLAS(cublasGemmStridedBatchedEx(
                    hb, CUBLAS_OP_T, CUBLAS_OP_N, np, np, std::min(kPiece, (l + 1) * kKc - k0),
                    &one, A + k0, CUDA_R_16BF, kSK * kKc, slab,
                    B + (size_t)(kSK - 1 - l) * kKc + k0, CUDA_R_16BF, kSK * kKc, slab, &zero, c,
                    CUDA_R_32F, np, nn, nc, CUBLAS_COMPUTE_32F, CUBLAS_GEMM_DEFAULT));
        combine_chunks_kernel<<<dim3((nao + 127) / 128, nao), 128, 0, s>>>(
            C, nao, np, nc, ex, eg, accumulate || c0 > 0, K);
        G64_CUDA(cudaGetLastError());
    }
    return 0;
}

}  // namespace wb
