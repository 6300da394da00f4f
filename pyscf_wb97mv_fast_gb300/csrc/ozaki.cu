// FP64-accurate GEMMs of the COSX K build on the bf16 tensor cores.
//
// GB300 runs FP64 at ~1 TFLOP/s, so F = X QD and K = X^T (w o G) -- the
// two dense contractions the reference keeps in FP64 (gpu/sgx_k.py:14-28,
// :722, :734) -- would dominate the build.  They run here as an Ozaki
// split (K. Ozaki et al., Numer. Algorithms 59 (2012) 95-118; on tensor
// cores: H. Ootomo, K. Ozaki, R. Yokota, IJHPCA 2024):
//
//   x = 2^(e-W+1) sum_i d_i 2^(B (S-1-i)),  |d_i| <= 2^(B-1)  (bf16-exact)
//
// with e per row / column (chunk), W = B S = 42 bits, the balanced digits cut
// from rint(x 2^(W-1-e)) with integer ops: S = 6 slices of B = 7 bits, 21
// slice products, where the sums below stay exact, else 7 of 6 bits, 28.
// A product level l = i + j collects sum_{i+j=l} A_i B_j in ONE bf16 GEMM
// with FP32 accumulation: storing the A slices ascending and the B slices
// descending along K makes every level a prefix of A times a suffix of B.
// Every product is an integer of magnitude <= 2^(2B-2), so while a GEMM sums
// at most 2^(26-2B) of them every partial sum is an integer up to 2^24: the
// FP32 accumulation is exact, whatever order the tensor cores use.  F sums
// (l+1) nao terms: 7-bit digits to nao = 680, 6-bit ones above.  The K product
// always takes 7-bit digits, its longer levels cut into pieces of 4096 terms,
// each a GEMM of its own (27 waters, 384,998 points: F 7.8 -> 6.4
// ms, K product of one right-hand side 9.1 -> 7.5 ms against 6-bit digits
// throughout).  Pieces and levels are combined exactly in int64 and
// scaled once in FP64.  The result carries W = 42 bits relative to the
// per-row / per-column maxima; the truncated products (i + j >= S) are
// below 2^-W of them.  A row or column with an infinity or a NaN gives NaN.
//
// The level GEMMs are library GEMMs (cuBLAS bf16 GEMMs with FP32
// accumulation, one per level) around this file's slicing and combination
// kernels.  Small F products (ozaki_f_small), or all of them after
// ozaki_set_f_engine(kOzEngineTc), run on this
// library's own tensor-core kernel instead (ozaki_tc.cu: TMA, tcgen05 MMAs
// into TMEM, the level combination fused into its epilogue) -- bitwise the
// same result; its six or seven exact level accumulators leave room for 64-wide
// N tiles only, and it measured 2.4x slower than the library form on the
// bench step (18.4 vs 7.65 ms with 6-bit digits).  The K product's level GEMMs are cuBLAS.
#include <cublas_v2.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>

#include "cvt64.cuh"
#include "launch.hpp"
#include "ozaki.hpp"
#include "ozaki_digits.cuh"

namespace wb {

// ---------------------------------------------------------------------------
// F = X QD.  X (nao, ld) AO-major = column-major A (ld x nao) scaled per row
// g; QD row-major = column-major Q (nao x nao) with Q(mu, l) = QD(l, mu);
// B = Q^T scaled per column mu (= per row mu of Q).
// A_all (ld x S*np, col-major): column block i = slice i.
// B_all (S*np x nao, col-major): row block r = slice S-1-r.
// np = nao rounded up to 8, the slices zero past nao: cuBLAS takes its
// tensor-memory kernels only for operands with 16-byte rows (356 AOs x
// 75,265 points: the seven level GEMMs 2.1 -> 0.6 ms).
// ---------------------------------------------------------------------------
// exponent of max_l |X(l, g)| per point g: eight rows in flight per thread
__global__ void f_rowmax_kernel(const double* __restrict__ X, int nao,
                                int64_t ld, int* __restrict__ erow) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= ld) return;
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
    erow[g] = exp_of_hi(m);
}

// slices of X: one thread per (row l, two points); bf16 pairs per store
template<int B_, int S>
__global__ void f_slice_x_kernel(const double* __restrict__ X, int nao, int np,
                                 int64_t ld, const int* __restrict__ erow,
                                 __nv_bfloat16* __restrict__ A) {
    const int l = blockIdx.y;
    const int64_t g = 2 * ((int64_t)blockIdx.x * blockDim.x + threadIdx.x);
    if (g >= ld) return;                    // ld is even (a multiple of 32)
    double2 x = make_double2(0.0, 0.0);
    if (l < nao) x = *reinterpret_cast<const double2*>(X + (int64_t)l * ld + g);
    const int2 e = *reinterpret_cast<const int2*>(erow + g);
    const unsigned long long q0 = biased_q<B_, S>(x.x, e.x), q1 = biased_q<B_, S>(x.y, e.y);
#pragma unroll
    for (int i = 0; i < S; ++i)
        *reinterpret_cast<unsigned*>(A + ((int64_t)i * np + l) * ld + g) =
            digit_pair<B_, S>(q0, q1, i);
}

template<int B_, int S>
__global__ void f_slice_qd_kernel(const double* __restrict__ QD, int nao, int np,
                                  int* __restrict__ ecol,
                                  __nv_bfloat16* __restrict__ B) {
    // one block per column mu of B = Q^T, i.e. QD(:, mu)
    const int mu = blockIdx.x;
    __shared__ unsigned red[256];
    unsigned m = 0;
    for (int l = threadIdx.x; l < nao; l += blockDim.x)
        m = max(m, abs_hi(QD[(int64_t)l * nao + mu]));
    red[threadIdx.x] = m;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s && red[threadIdx.x + s] > red[threadIdx.x])
            red[threadIdx.x] = red[threadIdx.x + s];
        __syncthreads();
    }
    const int e = exp_of_hi(red[0]);
    if (threadIdx.x == 0) ecol[mu] = e;
    const int64_t ldb = (int64_t)S * np;
    for (int l = threadIdx.x; l < np; l += blockDim.x) {
        const unsigned long long q =
            biased_q<B_, S>(l < nao ? QD[(int64_t)l * nao + mu] : 0.0, e);
#pragma unroll
        for (int i = 0; i < S; ++i)
            B[(int64_t)mu * ldb + (int64_t)(S - 1 - i) * np + l] =
                __ushort_as_bfloat16((unsigned short)digit_pair<B_, S>(q, q, i));
    }
}

// x y = 2^(e+f-2W+2) sum_l C_l 2^(B (2S-2-l))
//     = 2^(e+f-2W+2+B(S-1)) * [sum_l C_l 2^(B (S-1-l))]
template<int B_, int S, typename T>
__global__ void f_combine_kernel(const float* __restrict__ C, int nao,
                                 int64_t ld, const int* __restrict__ erow,
                                 const int* __restrict__ ecol,
                                 T* __restrict__ F) {
    const int mu = blockIdx.y;
    const int64_t g = 4 * ((int64_t)blockIdx.x * blockDim.x + threadIdx.x);
    if (g >= ld) return;                    // ld is a multiple of 4
    const int64_t plane = (int64_t)nao * ld;
    const int64_t i = (int64_t)mu * ld + g;
    float4 c[S];
#pragma unroll
    for (int l = 0; l < S; ++l)
        c[l] = __ldg(reinterpret_cast<const float4*>(C + (int64_t)l * plane + i));
    const int4 er = *reinterpret_cast<const int4*>(erow + g);
    const int base = ecol[mu] - 2 * kW + 2 + B_ * (S - 1);
    long long v[4] = {0, 0, 0, 0};
#pragma unroll
    for (int l = 0; l < S; ++l) {
        v[0] += level_term<B_, S>(l, c[l].x); v[1] += level_term<B_, S>(l, c[l].y);
        v[2] += level_term<B_, S>(l, c[l].z); v[3] += level_term<B_, S>(l, c[l].w);
    }
    T o0 = scaled_ll_to<T>(v[0], er.x + base);
    T o1 = scaled_ll_to<T>(v[1], er.y + base);
    T o2 = scaled_ll_to<T>(v[2], er.z + base);
    T o3 = scaled_ll_to<T>(v[3], er.w + base);
    if (not_finite(max(max(er.x, er.y), max(er.z, er.w)) + base)) {
        const T nan = (T)__int_as_float(0x7fc00000);
        if (not_finite(er.x + base)) o0 = nan;
        if (not_finite(er.y + base)) o1 = nan;
        if (not_finite(er.z + base)) o2 = nan;
        if (not_finite(er.w + base)) o3 = nan;
    }
    if constexpr (sizeof(T) == 4) {
        *reinterpret_cast<float4*>(F + i) = make_float4(o0, o1, o2, o3);
    } else {
        *reinterpret_cast<double2*>(F + i) = make_double2(o0, o1);
        *reinterpret_cast<double2*>(F + i + 2) = make_double2(o2, o3);
    }
}

// ---------------------------------------------------------------------------
// K = X^T (w o G), K dimension = grid points, chunked by KC points with a
// scale per (chunk, column).  Per chunk c, A_c(k, mu) = X[mu, c KC + k] and
// B_c(k, nu) = w_k G[nu, c KC + k]; layouts (col-major, ld = S KC):
//   A: column mu = [slice 0 (KC) | slice 1 | ... ]     (ascending)
//   B: column nu = [slice S-1 | ... | slice 0]          (descending)
// chunk stride S KC np (np = nao rounded up to 8, the columns past nao zero:
// 16-byte rows and outputs, as for F).  One CTA of KC / 8 threads per (chunk,
// column).  Bound by HBM (X, G and the slices once each, 36 bytes per entry of
// both operands): on the FP64 pipe only the product with the weight.  27 waters
// (648 AOs, 384,998 points, two G): 3.8 -> 2.4 ms; 1.2 of them had been spent on
// |x| and G -> FP64 as FP64 instructions.
// ---------------------------------------------------------------------------
// the constant of scale_word: FP64's bias, and what a chunk's sum is scaled by
template<int B_, int S>
constexpr int kScaleK = 1023 - 2 * 400 - 2 * kW + 2 + B_ * (S - 1);

// gridDim.z right-hand sides: B holds nb columns per chunk, those of right-hand
// side r at r np (np = gridDim.y).  The CTAs of the first one also slice X,
// unless slice_x is 0: the X slices and exponents of this tile are then already
// in A / ex (an earlier omega of the same tile).
template<typename GT>
struct KIn {
    const GT* g[8];
};
template<int B_, int S, int KC, typename GT>
__global__ void __launch_bounds__(KC / 8, 4)
k_slice_kernel(const double* __restrict__ X, const __grid_constant__ KIn<GT> Gs, const int slice_x,
               const double* __restrict__ w, int nao, int64_t ld,
               int64_t npts, int* __restrict__ ex, int* __restrict__ ew,
               __nv_bfloat16* __restrict__ A, __nv_bfloat16* __restrict__ B,
               int nb) {
    constexpr int T = KC / 8;               // threads: eight points each
    const int c = blockIdx.x, col = blockIdx.y, np = gridDim.y;
    const int boff = blockIdx.z * np;
    const bool dox = slice_x && blockIdx.z == 0;
    const GT* __restrict__ G = Gs.g[blockIdx.z];
    const int64_t nlive = col < nao ? npts : 0;     // a column past nao is zero
    __shared__ unsigned rx[T / 32], rw[T / 32];
    const int k0 = 8 * threadIdx.x;
    const int64_t g0 = (int64_t)c * KC + k0;
    double xv[8], wv[8];
    unsigned mx = 0, mw = 0;
    if (g0 + 8 <= nlive) {
        const double2* xp = reinterpret_cast<const double2*>(X + (int64_t)col * ld + g0);
        const double2* wp = reinterpret_cast<const double2*>(w + g0);
        double gv[8];
        if constexpr (sizeof(GT) == 4) {
            const float4* gp = reinterpret_cast<const float4*>(G + (int64_t)col * ld + g0);
            const float4 ga = __ldg(gp), gb = __ldg(gp + 1);
            gv[0] = to_f64(ga.x); gv[1] = to_f64(ga.y);
            gv[2] = to_f64(ga.z); gv[3] = to_f64(ga.w);
            gv[4] = to_f64(gb.x); gv[5] = to_f64(gb.y);
            gv[6] = to_f64(gb.z); gv[7] = to_f64(gb.w);
        } else {
            const double2* gp = reinterpret_cast<const double2*>(G + (int64_t)col * ld + g0);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const double2 t = __ldg(gp + u);
                gv[2 * u] = t.x;
                gv[2 * u + 1] = t.y;
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const double2 b = __ldg(wp + u);
            if (dox) {
                const double2 a = __ldg(xp + u);
                xv[2 * u] = a.x; xv[2 * u + 1] = a.y;
            } else {
                xv[2 * u] = 0.0; xv[2 * u + 1] = 0.0;
            }
            wv[2 * u] = b.x * gv[2 * u];
            wv[2 * u + 1] = b.y * gv[2 * u + 1];
        }
    } else {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int64_t g = g0 + u;
            xv[u] = 0.0;
            wv[u] = 0.0;
            if (g < nlive) {
                if (dox) xv[u] = X[(int64_t)col * ld + g];
                wv[u] = w[g] * (double)G[(int64_t)col * ld + g];
            }
        }
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        mx = max(mx, abs_hi(xv[u]));
        mw = max(mw, abs_hi(wv[u]));
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    mw = __reduce_max_sync(0xffffffffu, mw);
    const int warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) { rx[warp] = mx; rw[warp] = mw; }
    __syncthreads();
    mx = 0;
    mw = 0;
#pragma unroll
    for (int j = 0; j < T / 32; ++j) {
        mx = max(mx, rx[j]);
        mw = max(mw, rw[j]);
    }
    const int e1 = exp_of_hi(mx), e2 = exp_of_hi(mw);
    if (threadIdx.x == 0) {
        if (dox) ex[(int64_t)c * np + col] = scale_word(e1, kScaleK<B_, S>);
        ew[(int64_t)c * nb + boff + col] = scale_word(e2);
    }
    const int64_t colbase = (int64_t)c * S * KC * np + (int64_t)col * S * KC;
    const int64_t colbase_b = (int64_t)c * S * KC * nb + (int64_t)(boff + col) * S * KC;
    // one operand's digits at a time: the X slices, then the w o G ones
    // (half the live registers of both at once)
    auto store = [&](const double* v, const int e, __nv_bfloat16* dst, const bool desc) {
        unsigned long long q[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) q[u] = biased_q<B_, S>(v[u], e);
#pragma unroll
        for (int i = 0; i < S; ++i)
            *reinterpret_cast<uint4*>(dst + (int64_t)(desc ? S - 1 - i : i) * KC + k0) =
                make_uint4(digit_pair<B_, S>(q[0], q[1], i), digit_pair<B_, S>(q[2], q[3], i),
                           digit_pair<B_, S>(q[4], q[5], i), digit_pair<B_, S>(q[6], q[7], i));
    };
    if (dox) store(xv, e1, A + colbase, false);
    store(wv, e2, B + colbase_b, true);
}

// K_r[mu, nu] (+)= sum_c 2^(ex+ew-2W+2+B(S-1)) [sum_l C[l][c] 2^(B (S-1-l))]
// for the nb / np right-hand sides r (column r np + nu of C)
constexpr int kKB = 7, kKS = 6;         // the K product's digits
constexpr int kOzPiece = 4096;          // terms of an exact FP32 sum of 7-bit products

struct KOut {
    double* k[8];
};

// C holds the level planes in order, a level of more than kOzPiece terms as
// several planes (pieces), each (chunk, np x nb)
template<int B_, int S, int KC>
__global__ void k_combine_kernel(const float* __restrict__ C, int nao, int np, int nb,
                                 int nchunk, const int* __restrict__ ex,
                                 const int* __restrict__ ew, int accumulate,
                                 const __grid_constant__ KOut Ks) {
    const int64_t nc = (int64_t)np * nb;
    const int64_t plane = nc * nchunk;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nc;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int mu = (int)(i % np), col = (int)(i / np);     // C col-major
        if (mu >= nao || col % np >= nao) continue;
        double acc = 0.0;
        // three chunks' loads in flight at once; the sum stays in chunk order
        constexpr int U = 3;
        auto value = [&](int c) -> long long {
            const float* p = C + (int64_t)c * nc + i;
            long long v = 0;
#pragma unroll
            for (int l = 0; l < S; ++l)
#pragma unroll
                for (int left = (l + 1) * KC; left > 0; left -= kOzPiece, p += plane)
                    v += level_term<B_, S>(l, __ldg(p));
            return v;
        };
        auto scale = [&](int c) {
            return scale_of(ex[(int64_t)c * np + mu], ew[(int64_t)c * nb + col]);
        };
        int c = 0;
        for (; c + U <= nchunk; c += U) {
            long long v[U];
            double sc[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                v[u] = value(c + u);
                sc[u] = scale(c + u);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) acc += (double)v[u] * sc[u];
        }
        for (; c < nchunk; ++c) acc += (double)value(c) * scale(c);
        double* K = Ks.k[col / np];
        const int64_t o = (int64_t)mu * nao + col % np;        // K row-major
        K[o] = accumulate ? K[o] + acc : acc;
    }
}

// ---------------------------------------------------------------------------
static inline size_t al(size_t x) { return (x + 255) & ~(size_t)255; }

static inline int pad8(int n) { return (n + 7) & ~7; }

// level planes of the K product
static inline int k_planes(int kc) {
    int n = 0;
    for (int l = 0; l < kKS; ++l) n += ((l + 1) * kc + kOzPiece - 1) / kOzPiece;
    return n;
}

// Points per chunk of the K product.  2048 is the largest with exact level
// sums and moves the least level output per point; where it would leave SMs
// idle (fewer than one 128 x 128 tile per SM over the chunks of a level GEMM),
// 512 gives four times the tiles, each a quarter as long (48 AOs x 9,931
// points: the seven GEMMs 89 -> 42 us).
static inline int k_chunk(int np, int64_t ld) {
    const int64_t t = (np + 127) / 128;
    return t * t * ((ld + kOzKc - 1) / kOzKc) < sm_count() ? kOzKcSmall : kOzKc;
}

size_t ozaki_f_bytes(int nao, int64_t ld) {
    const size_t S = ozaki_f_seven_bit(nao) ? 6 : 7, np = pad8(nao);
    const size_t lib = al(sizeof(int) * ld) + al(sizeof(int) * nao) +
                       al(sizeof(__nv_bfloat16) * S * np * ld) +
                       al(sizeof(__nv_bfloat16) * S * np * nao) +
                       al(sizeof(float) * S * nao * ld);
    return std::max(lib, ozaki_f_tc_bytes(nao, ld));
}

size_t ozaki_k_bytes(int nao, int64_t ld, int nrhs) {
    const size_t S = kKS, np = pad8(nao);
    auto bytes = [&](size_t kc, int64_t n) {
        const size_t nchunk = (n + kc - 1) / kc;
        return al(sizeof(int) * nchunk * np) + al(sizeof(int) * nchunk * np * nrhs) +
               al(sizeof(__nv_bfloat16) * S * kc * nchunk * np) +
               al(sizeof(__nv_bfloat16) * S * kc * nchunk * np * nrhs) +
               al(sizeof(float) * k_planes((int)kc) * nchunk * np * np * nrhs);
    };
    // enough for every grid of up to ld points (a ragged last tile may take
    // the small chunks where the full one does not)
    const int64_t t = ((int64_t)np + 127) / 128;
    const int64_t small = std::min(ld, (sm_count() - 1) / (t * t) * (int64_t)kOzKc);
    return std::max(bytes(kOzKc, ld), bytes(kOzKcSmall, small));
}

#define OZ_CUBLAS(call)                                        \
    do {                                                       \
        cublasStatus_t st_ = (call);                           \
        if (st_ != CUBLAS_STATUS_SUCCESS) return (int)st_ + 1000; \
    } while (0)
#define OZ_CUDA(call)                                          \
    do {                                                       \
        cudaError_t e_ = (call);                               \
        if (e_ != cudaSuccess) return (int)e_;                 \
    } while (0)

void f_rowmax(const double* X, int nao, int64_t ld, int* erow, cudaStream_t s) {
    f_rowmax_kernel<<<(unsigned)((ld + 255) / 256), 256, 0, s>>>(X, nao, ld, erow);
}

namespace {
std::atomic<int> g_f_engine{kOzEngineAuto};
}

void ozaki_set_f_engine(int engine) { g_f_engine.store(engine); }
int ozaki_get_f_engine() { return g_f_engine.load(); }
bool ozaki_f_small(int nao, int64_t ld) {
    return nao <= 64 && (ld + 127) / 128 <= sm_count();
}
bool ozaki_f_on_tc(int nao, int64_t ld) {
    const int e = g_f_engine.load();
    return e == kOzEngineTc || (e == kOzEngineAuto && ozaki_f_small(nao, ld));
}

int ozaki_f_gemm(cublasHandle_t hb, const double* X, const double* QD,
                 int nao, int64_t ld, float* F, void* ws, cudaStream_t s,
                 unsigned long long* status) {
    if (ozaki_f_on_tc(nao, ld))
        return ozaki_f_gemm_tc(X, QD, nao, ld, F, ws, s, status);
    return ozaki_f_gemm_cublas(hb, X, QD, nao, ld, F, ws, s);
}

int ozaki_f_gemm64(cublasHandle_t hb, const double* X, const double* QD,
                   int nao, int64_t ld, double* F, void* ws, cudaStream_t s,
                   unsigned long long* status) {
    if (ozaki_f_on_tc(nao, ld))
        return ozaki_f_gemm_tc64(X, QD, nao, ld, F, ws, s, status);
    return ozaki_f_gemm_cublas64(hb, X, QD, nao, ld, F, ws, s);
}

template<int B_, int S, typename T>
static int f_gemm_cublas_t(cublasHandle_t hb, const double* X, const double* QD,
                           int nao, int64_t ld, T* F, void* ws, cudaStream_t s) {
    const int np = pad8(nao);
    char* p = static_cast<char*>(ws);
    int* erow = reinterpret_cast<int*>(p); p += al(sizeof(int) * ld);
    int* ecol = reinterpret_cast<int*>(p); p += al(sizeof(int) * nao);
    __nv_bfloat16* A = reinterpret_cast<__nv_bfloat16*>(p);
    p += al(sizeof(__nv_bfloat16) * (size_t)S * np * ld);
    __nv_bfloat16* B = reinterpret_cast<__nv_bfloat16*>(p);
    p += al(sizeof(__nv_bfloat16) * (size_t)S * np * nao);
    float* C = reinterpret_cast<float*>(p);
    f_rowmax_kernel<<<(unsigned)((ld + 255) / 256), 256, 0, s>>>(X, nao, ld, erow);
    OZ_CUDA(cudaGetLastError());
    {
        dim3 grid((unsigned)((ld / 2 + 255) / 256), (unsigned)np);
        f_slice_x_kernel<B_, S><<<grid, 256, 0, s>>>(X, nao, np, ld, erow, A);
        OZ_CUDA(cudaGetLastError());
    }
    f_slice_qd_kernel<B_, S><<<nao, 256, 0, s>>>(QD, nao, np, ecol, B);
    OZ_CUDA(cudaGetLastError());
    const float one = 1.0f, zero = 0.0f;
    for (int l = 0; l < S; ++l) {
        // C_l (ld x nao) = A[:, 0:(l+1) np] * B[(S-1-l) np : S np, :]
        OZ_CUBLAS(cublasGemmEx(hb, CUBLAS_OP_N, CUBLAS_OP_N, (int)ld, nao,
                               (l + 1) * np, &one, A, CUDA_R_16BF, (int)ld,
                               B + (size_t)(S - 1 - l) * np, CUDA_R_16BF,
                               S * np, &zero, C + (size_t)l * nao * ld,
                               CUDA_R_32F, (int)ld, CUBLAS_COMPUTE_32F,
                               CUBLAS_GEMM_DEFAULT));
    }
    {
        dim3 grid((unsigned)((ld / 4 + 255) / 256), (unsigned)nao);
        f_combine_kernel<B_, S, T><<<grid, 256, 0, s>>>(C, nao, ld, erow, ecol, F);
        OZ_CUDA(cudaGetLastError());
    }
    return 0;
}

int ozaki_f_gemm_cublas(cublasHandle_t hb, const double* X, const double* QD,
                        int nao, int64_t ld, float* F, void* ws, cudaStream_t s) {
    return ozaki_f_seven_bit(nao)
               ? f_gemm_cublas_t<7, 6, float>(hb, X, QD, nao, ld, F, ws, s)
               : f_gemm_cublas_t<6, 7, float>(hb, X, QD, nao, ld, F, ws, s);
}

int ozaki_f_gemm_cublas64(cublasHandle_t hb, const double* X, const double* QD,
                          int nao, int64_t ld, double* F, void* ws, cudaStream_t s) {
    return ozaki_f_seven_bit(nao)
               ? f_gemm_cublas_t<7, 6, double>(hb, X, QD, nao, ld, F, ws, s)
               : f_gemm_cublas_t<6, 7, double>(hb, X, QD, nao, ld, F, ws, s);
}

template<int KC, typename GT>
static int k_gemm_multi_t(cublasHandle_t hb, const double* X, const GT* const* G,
                          int nrhs, const double* w, int nao, int64_t ld,
                          int64_t npts, int accumulate, double* const* K, void* ws,
                          cudaStream_t s, bool x_sliced) {
    constexpr int S = kKS;
    if (nrhs < 1 || nrhs > 8) return (int)cudaErrorInvalidValue;
    const int nchunk = (int)((ld + KC - 1) / KC);
    const int np = pad8(nao), nb = nrhs * np;
    // the X side (ex, A) first, at offsets independent of nrhs, so that a
    // later call with x_sliced finds them whatever its nrhs
    char* p = static_cast<char*>(ws);
    int* ex = reinterpret_cast<int*>(p); p += al(sizeof(int) * (size_t)nchunk * np);
    const size_t slab = (size_t)S * KC * nchunk * np;
    __nv_bfloat16* A = reinterpret_cast<__nv_bfloat16*>(p);
    p += al(sizeof(__nv_bfloat16) * slab);
    int* ew = reinterpret_cast<int*>(p); p += al(sizeof(int) * (size_t)nchunk * nb);
    __nv_bfloat16* B = reinterpret_cast<__nv_bfloat16*>(p);
    p += al(sizeof(__nv_bfloat16) * slab * nrhs);
    float* C = reinterpret_cast<float*>(p);
    KOut Kd = {};
    for (int r = 0; r < nrhs; ++r) Kd.k[r] = K[r];
    KIn<GT> in = {};
    for (int r = 0; r < nrhs; ++r) in.g[r] = G[r];
    k_slice_kernel<kKB, S, KC, GT><<<dim3(nchunk, np, nrhs), KC / 8, 0, s>>>(
        X, in, x_sliced ? 0 : 1, w, nao, ld, npts, ex, ew, A, B, nb);
    OZ_CUDA(cudaGetLastError());
    const float one = 1.0f, zero = 0.0f;
    const long long stride_a = (long long)S * KC * np;
    const long long stride_b = (long long)S * KC * nb;
    const long long nc = (long long)np * nb;
    float* c = C;
    for (int l = 0; l < S; ++l)
        for (int k0 = 0; k0 < (l + 1) * KC; k0 += kOzPiece, c += (size_t)nchunk * nc)
            OZ_CUBLAS(cublasGemmStridedBatchedEx(
                hb, CUBLAS_OP_T, CUBLAS_OP_N, np, nb, std::min(kOzPiece, (l + 1) * KC - k0),
                &one, A + k0, CUDA_R_16BF, S * KC, stride_a,
                B + (size_t)(S - 1 - l) * KC + k0, CUDA_R_16BF, S * KC, stride_b, &zero, c,
                CUDA_R_32F, np, nc, nchunk, CUBLAS_COMPUTE_32F, CUBLAS_GEMM_DEFAULT));
    const int64_t blocks = grid_stride_blocks(nc, 256, 32);
    k_combine_kernel<kKB, S, KC><<<(unsigned)blocks, 256, 0, s>>>(C, nao, np, nb, nchunk, ex, ew,
                                                        accumulate, Kd);
    OZ_CUDA(cudaGetLastError());
    return 0;
}

int ozaki_k_launches(int nao, int64_t ld) {
    return 2 + k_planes(k_chunk(pad8(nao), ld));
}

template<typename GT>
static int k_gemm_any(cublasHandle_t hb, const double* X, const GT* const* G, int nrhs,
                      const double* w, int nao, int64_t ld, int64_t npts, int accumulate,
                      double* const* K, void* ws, cudaStream_t s, bool x_sliced) {
    return k_chunk(pad8(nao), ld) == kOzKc
               ? k_gemm_multi_t<kOzKc, GT>(hb, X, G, nrhs, w, nao, ld, npts, accumulate, K,
                                           ws, s, x_sliced)
               : k_gemm_multi_t<kOzKcSmall, GT>(hb, X, G, nrhs, w, nao, ld, npts, accumulate,
                                                K, ws, s, x_sliced);
}

int ozaki_k_gemm_multi(cublasHandle_t hb, const double* X, const float* const* G,
                       int nrhs, const double* w, int nao, int64_t ld,
                       int64_t npts, int accumulate, double* const* K, void* ws,
                       cudaStream_t s, bool x_sliced) {
    return k_gemm_any<float>(hb, X, G, nrhs, w, nao, ld, npts, accumulate, K, ws, s,
                             x_sliced);
}

int ozaki_k_gemm64(cublasHandle_t hb, const double* X, const double* G,
                   const double* w, int nao, int64_t ld, int64_t npts,
                   int accumulate, double* K, void* ws, cudaStream_t s) {
    return k_gemm_any<double>(hb, X, &G, 1, w, nao, ld, npts, accumulate, &K, ws, s, false);
}

int ozaki_k_gemm(cublasHandle_t hb, const double* X, const float* G,
                 const double* w, int nao, int64_t ld, int64_t npts,
                 int accumulate, double* K, void* ws, cudaStream_t s,
                 bool x_sliced) {
    return ozaki_k_gemm_multi(hb, X, &G, 1, w, nao, ld, npts, accumulate, &K, ws,
                              s, x_sliced);
}

}  // namespace wb
