// Supporting kernels of the COSX K build: per-omega primitive constants,
// grid coordinate split, sub-block statistics for the screen, FP64 AO
// evaluation, precision casts, the dense validation kernel and the Boys
// batch kernel.
#include <algorithm>
#include <cmath>

#include "boys.cuh"
#include "cart.cuh"
#include "cvt64.cuh"
#include "fp64_boys.cuh"
#include "launch.hpp"
#include "screen.cuh"

namespace wb {

// -- per-omega primitive-pair constants (gpu/sgx_k.py:783-811) --------------
// theta = w^2 / (w^2 + p) (1 for w = 0), tp = theta p and the R000
// coefficients c_n = pref sqrt(theta) (-2 p theta)^n, n = 0..6, formed in
// FP64 (IEEE-rounded, so identical to a host evaluation) and stored as FP32
// hi + lo.  pref already carries C_a C_b K_AB 2 pi / p and the s/p
// spherical normalisation.
__global__ void omega_kernel(int npp, const double* __restrict__ p,
                             const double* __restrict__ pref, double omega,
                             float4* __restrict__ om) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= npp) return;
    const double pm = p[m];
    double th = 1.0, sth = 1.0;
    if (omega > 0.0) {
        const double w2 = omega * omega;
        th = w2 / (w2 + pm);
        sth = sqrt(th);
    }
    const double tp = th * pm;
    const double q = -2.0 * pm * th;
    float rec[20];
    rec[0] = (float)tp;
    rec[1] = (float)(tp - (double)rec[0]);
    double c = pref[m] * sth;
    // far field (T = tp r^2 >= 36, erf(sqrt T) = 1 in FP64): R000_n =
    // (-1)^n (2n-1)!! K0 r^-(2n+1) with K0 = c_0 sqrt(pi) / (2 sqrt(tp))
    const double k0 = c * 0.88622692545275801365 / sqrt(tp);
    for (int n = 0; n < 7; ++n) {
        const float hi = (float)c;
        rec[2 + 2 * n] = hi;
        rec[3 + 2 * n] = (float)(c - (double)hi);
        c *= q;
    }
    rec[16] = (float)k0;
    rec[17] = (float)(k0 - (double)rec[16]);
    rec[18] = (float)(36.0 / tp);            // r^2 at which T reaches 36
    rec[19] = 0.0f;
    float4* o = om + 5 * (long long)m;
    o[0] = make_float4(rec[0], rec[1], rec[2], rec[3]);
    o[1] = make_float4(rec[4], rec[5], rec[6], rec[7]);
    o[2] = make_float4(rec[8], rec[9], rec[10], rec[11]);
    o[3] = make_float4(rec[12], rec[13], rec[14], rec[15]);
    o[4] = make_float4(rec[16], rec[17], rec[18], rec[19]);
}

cudaError_t launch_omega(int npp, const double* p, const double* pref,
                         double omega, float4* om, cudaStream_t s) {
    if (npp <= 0) return cudaSuccess;
    omega_kernel<<<(npp + 255) / 256, 256, 0, s>>>(npp, p, pref, omega, om);
    return cudaGetLastError();
}

// Packed per-class primitive-pair records for the class kernels: one
// contiguous record per pair (P hi, P lo, the first n_om float4 of the
// omega record, the Hermite E block) so that a pair is one base address.
__global__ void pack_records_kernel(const RecPack P, int npp,
                                    const float4* __restrict__ geo,
                                    const float4* __restrict__ om,
                                    const float4* __restrict__ E,
                                    float4* __restrict__ rec) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= npp) return;
    int c = 0;
    while (c < 9 && m >= P.pp_end[c]) ++c;
    if (m < P.pp_begin[c] || m >= P.pp_end[c]) return;
    const int ml = m - P.pp_begin[c];
    float4* r = rec + P.rec_off[c] + (long long)ml * P.stride[c];
    r[0] = geo[2 * (long long)m];
    r[1] = geo[2 * (long long)m + 1];
    // omega record: its first n_om - 1 float4 (theta p, c_n), then the
    // far-field float4 (K0 hi, K0 lo, r^2 threshold)
    for (int q = 0; q + 1 < P.nom[c]; ++q) r[2 + q] = om[5 * (long long)m + q];
    r[1 + P.nom[c]] = om[5 * (long long)m + 4];
    const float4* e = E + P.e_off[c] + (long long)ml * P.ne[c];
    for (int q = 0; q < P.ne[c]; ++q) r[2 + P.nom[c] + q] = e[q];
}

cudaError_t launch_pack_records(const RecPack& P, int npp, const float4* geo,
                                const float4* om, const float4* E,
                                float4* rec, cudaStream_t s) {
    if (npp <= 0) return cudaSuccess;
    pack_records_kernel<<<(npp + 127) / 128, 128, 0, s>>>(P, npp, geo, om, E, rec);
    return cudaGetLastError();
}

__global__ void pack_records2_kernel(const RecPack P, int npp,
                                     const float4* __restrict__ geo,
                                     const float4* __restrict__ oma,
                                     const float4* __restrict__ omb,
                                     const float4* __restrict__ E,
                                     float4* __restrict__ rec) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= npp) return;
    int c = 0;
    while (c < 9 && m >= P.pp_end[c]) ++c;
    if (m < P.pp_begin[c] || m >= P.pp_end[c]) return;
    const int ml = m - P.pp_begin[c];
    const int nom = P.nom[c];
    float4* r = rec + P.rec_off[c] + (long long)ml * P.stride[c];
    r[0] = geo[2 * (long long)m];
    r[1] = geo[2 * (long long)m + 1];
    const float4* om[2] = {oma, omb};
    for (int w = 0; w < 2; ++w) {
        for (int q = 0; q + 1 < nom; ++q) r[2 + w * nom + q] = om[w][5 * (long long)m + q];
        r[1 + (w + 1) * nom] = om[w][5 * (long long)m + 4];
    }
    const float4* e = E + P.e_off[c] + (long long)ml * P.ne[c];
    for (int q = 0; q < P.ne[c]; ++q) r[2 + 2 * nom + q] = e[q];
}

cudaError_t launch_pack_records2(const RecPack& P, int npp, const float4* geo,
                                 const float4* om_a, const float4* om_b,
                                 const float4* E, float4* rec, cudaStream_t s) {
    if (npp <= 0) return cudaSuccess;
    pack_records2_kernel<<<(npp + 127) / 128, 128, 0, s>>>(P, npp, geo, om_a, om_b,
                                                         E, rec);
    return cudaGetLastError();
}

// -- FP64 (npts, 3) -> FP32 SoA hi / lo, padded with zeros to ld ----------
__global__ void grid_prep_kernel(const double* __restrict__ c, int64_t npts,
                                 int64_t ld, float* __restrict__ hi,
                                 float* __restrict__ lo) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= ld) return;
    for (int x = 0; x < 3; ++x) {
        float h = 0.0f, l = 0.0f;
        if (g < npts) {
            const double v = c[g * 3 + x];
            h = (float)v;
            l = (float)(v - (double)h);
        }
        hi[x * ld + g] = h;
        lo[x * ld + g] = l;
    }
}

cudaError_t launch_grid_prep(const double* coords, int64_t npts, int64_t ld,
                             float* hi, float* lo, cudaStream_t s) {
    if (ld <= 0) return cudaSuccess;
    grid_prep_kernel<<<(unsigned)((ld + 255) / 256), 256, 0, s>>>(coords, npts,
                                                                  ld, hi, lo);
    return cudaGetLastError();
}

// -- sub-block statistics (gpu/sgx_k.py:866-903) ---------------------------
// One warp per 128-point block (four points per lane): for its 32-point
// quarters (the reference's sub-block size), its 64-point halves and the
// whole block, the FP64 centroid and radius of the valid points (centroid
// rounded to nearest FP32, radius rounded up) and, for every (virtual)
// shell, msh = max_g fl32(w_g) sum_{t in shell} |F_tg| (NaN where one of them
// is).  One pass over F
// serves the 32-, 64- and 128-point class kernels.  Block b of size 32 * 2^k
// covers points [b 32 2^k, (b + 1) 32 2^k); blocks past ld are not written.
__device__ __forceinline__ double warp_sum_d(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// the largest of 32 non-negative doubles, by their bits
__device__ __forceinline__ double warp_max_bits(double v) {
    const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
    return __hiloint2double((int)mh, (int)ml);
}

// The shells are shared out over gridDim.y: one warp walking all of them is a
// serial chain of loads (70 us for the 24 shells and 9,931 points of two
// waters, a third of the HBM rate on large grids).
constexpr int kStatsShells = 6;

__global__ void sub_stats_kernel(const BlockStatsOut O,
                                 const double* __restrict__ coords,
                                 const double* __restrict__ w,
                                 const float* __restrict__ F, int64_t npts,
                                 int64_t ld, int nvshell,
                                 const int* __restrict__ vs_ao0,
                                 const int* __restrict__ vs_nf) {
    const int blk = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int nblk128 = (int)((ld + 127) / 128);
    if (blk >= nblk128) return;
    // this CTA's share of the shells; the first share also writes the centroids
    const int sh0 = blockIdx.y * kStatsShells;
    const int sh1 = min(nvshell, sh0 + kStatsShells);
    // blocks of each level that exist: 32 * 2^k points starting inside ld
    int64_t g[4];
    bool valid[4];
    double c[4][3];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        g[q] = (int64_t)blk * 128 + 32 * q + lane;
        valid[q] = g[q] < npts;
        for (int x = 0; x < 3; ++x) c[q][x] = valid[q] ? coords[g[q] * 3 + x] : 0.0;
    }
    if (blockIdx.y == 0) {
        // The seven blocks: 0-3 the quarters, 4 and 5 the halves, 6 the whole.
        // A warp's FP64 instruction takes 16 cycles whatever its active lanes,
        // so the divisions run once, lane 3 b + x on component x of block b,
        // the square roots once, lane b on the largest distance of block b, and
        // the maxima on the integer pipe.
        double s[7][3];
#pragma unroll
        for (int x = 0; x < 3; ++x) {
#pragma unroll
            for (int q = 0; q < 4; ++q) s[q][x] = warp_sum_d(c[q][x]);
            s[4][x] = s[0][x] + s[1][x];
            s[5][x] = s[2][x] + s[3][x];
            s[6][x] = s[4][x] + s[2][x] + s[3][x];
        }
        auto level = [](int b) { return b < 4 ? 0 : (b < 6 ? 1 : 2); };
        auto first = [](int b) { return b < 4 ? b : (b < 6 ? 2 * (b - 4) : 0); };
        auto count = [&](int b) {
            const int64_t rem = npts - ((int64_t)blk * 128 + 32 * first(b));
            const int full = 32 << level(b);
            return rem >= full ? full : (rem > 0 ? (int)rem : 0);
        };
        double own = 0.0;
#pragma unroll
        for (int i = 0; i < 21; ++i)
            if (lane == i) own = s[i / 3][i % 3];
        const int nown = count(lane < 21 ? lane / 3 : 6);
        own = nown ? own / nown : 0.0;
        double dmax = 0.0;
#pragma unroll
        for (int b = 0; b < 7; ++b) {
            double m[3];
#pragma unroll
            for (int x = 0; x < 3; ++x) m[x] = __shfl_sync(0xffffffffu, own, 3 * b + x);
            double d = 0.0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (q < first(b) || q >= first(b) + (1 << level(b)) || !valid[q]) continue;
                double e2 = 0.0;
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    const double e = c[q][x] - m[x];
                    e2 += e * e;
                }
                d = fmax(d, e2);
            }
            d = warp_max_bits(d);
            if (lane == b) dmax = d;
        }
        const double d = sqrt(dmax);
        float cen[3];
#pragma unroll
        for (int x = 0; x < 3; ++x)
            cen[x] = (float)__shfl_sync(0xffffffffu, own, lane < 7 ? 3 * lane + x : 0);
        float r = (float)d;
        if ((double)r < d) r = nextafterf(r, INFINITY);
        if (lane < 7) {
            const int k = level(lane);
            const int64_t b = ((int64_t)blk * 4 + first(lane)) >> k;
            if (b * (32 << k) < ld) O.cr[k][b] = make_float4(cen[0], cen[1], cen[2], r);
        }
    }
    float wq[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) wq[q] = valid[q] ? (float)w[g[q]] : 0.0f;
    for (int sh = sh0; sh < sh1; ++sh) {
        const int a0 = vs_ao0[sh], nf = vs_nf[sh];
        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        for (int t = 0; t < nf; ++t) {
            const int64_t row = (int64_t)(a0 + t) * ld;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (valid[q]) acc[q] += fabsf(F[row + g[q]]) * wq[q];
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
            for (int o = 16; o > 0; o >>= 1)
                acc[q] = max_nan(acc[q], __shfl_xor_sync(0xffffffffu, acc[q], o));
        if (lane == 0) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int64_t b = (int64_t)blk * 4 + q;
                if (b * 32 < ld) O.msh[0][b * nvshell + sh] = acc[q];
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int64_t b = (int64_t)blk * 2 + j;
                if (b * 64 < ld)
                    O.msh[1][b * nvshell + sh] = max_nan(acc[2 * j], acc[2 * j + 1]);
            }
            O.msh[2][(int64_t)blk * nvshell + sh] =
                max_nan(max_nan(acc[0], acc[1]), max_nan(acc[2], acc[3]));
        }
    }
}

cudaError_t launch_sub_stats(const double* coords, const double* weights,
                             const float* F, int64_t npts, int64_t ld,
                             int nvshell, const int* vs_ao0, const int* vs_nf,
                             const BlockStatsOut& out, cudaStream_t s) {
    const int64_t nblk = (ld + 127) / 128;
    if (nblk <= 0) return cudaSuccess;
    // one warp a CTA while the blocks are fewer than four an SM
    const int warps = nblk < 4 * (int64_t)sm_count() ? 1 : 4;
    const dim3 grid((unsigned)((nblk + warps - 1) / warps),
                    (unsigned)std::max(1, (nvshell + kStatsShells - 1) / kStatsShells));
    sub_stats_kernel<<<grid, 32 * warps, 0, s>>>(
        out, coords, weights, F, npts, ld, nvshell, vs_ao0, vs_nf);
    return cudaGetLastError();
}

// -- casts ---------------------------------------------------------------
__global__ void f64_to_f32_kernel(const double* __restrict__ in,
                                  float* __restrict__ out, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        out[i] = __double2float_rn(in[i]);
}

cudaError_t launch_f64_to_f32(const double* in, float* out, int64_t n,
                              cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const int64_t blocks = grid_stride_blocks(n, 256, 64);
    f64_to_f32_kernel<<<(unsigned)blocks, 256, 0, s>>>(in, out, n);
    return cudaGetLastError();
}

// out[mu, g] = w_g * (double) G[mu, g]  (gpu/sgx_k.py:734: FP64 weights)
__global__ void weight_g_kernel(const float* __restrict__ G,
                                const double* __restrict__ w, int64_t npts,
                                int64_t ld, int64_t total,
                                double* __restrict__ out) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t g = i % ld;
        out[i] = g < npts ? w[g] * (double)G[i] : 0.0;
    }
}

cudaError_t launch_weight_g(const float* G, const double* w, int64_t npts,
                            int64_t ld, int nao, double* out, cudaStream_t s) {
    const int64_t total = ld * nao;
    if (total <= 0) return cudaSuccess;
    const int64_t blocks = grid_stride_blocks(total, 256, 64);
    weight_g_kernel<<<(unsigned)blocks, 256, 0, s>>>(G, w, npts, ld, total, out);
    return cudaGetLastError();
}

// G[mu, g] = sum of the class partial-G rows src[mu] (ascending class
// order, -1 = none): the fixed-order combination of the concurrently
// filled class buffers.  Four points per thread (ld is a multiple of 32).
__global__ void gsum_kernel(const float* __restrict__ gc,
                            const int4* __restrict__ src, int64_t ld,
                            float* __restrict__ G) {
    const int mu = blockIdx.y;
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (i >= ld) return;
    const int4 sr = src[mu];
    const int rows[4] = {sr.x, sr.y, sr.z, sr.w};
    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (rows[j] < 0) continue;
        const float4 v = *reinterpret_cast<const float4*>(gc + rows[j] * ld + i);
        acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    *reinterpret_cast<float4*>(G + (int64_t)mu * ld + i) = acc;
}

// the same over two buffer sets (the two halves of split blocks): the
// first set's rows, then the second's, in fixed order; gridDim.z omegas
__global__ void gsum2_kernel(const __grid_constant__ GSum2 S, const int4* __restrict__ src, int64_t ld) {
    const int mu = blockIdx.y;
    const float* __restrict__ gc0 = S.gc0[blockIdx.z];
    const float* __restrict__ gc1 = S.gc1[blockIdx.z];
    float* __restrict__ G = S.G[blockIdx.z];
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (i >= ld) return;
    const int4 sr = src[mu];
    const int rows[4] = {sr.x, sr.y, sr.z, sr.w};
    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int h = 0; h < 2; ++h) {
        const float* gc = h ? gc1 : gc0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (rows[j] < 0) continue;
            const float4 v = *reinterpret_cast<const float4*>(gc + rows[j] * ld + i);
            acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
        }
    }
    *reinterpret_cast<float4*>(G + (int64_t)mu * ld + i) = acc;
}

// Longest-processing-time order of the point blocks of each class (one
// CTA per class): a counting sort of the blocks by their measured cost in
// 2^(1/8) steps, costliest first.  Each kernel hands its blocks out in this
// order, so the last blocks taken -- the tail of the launch -- are the
// cheap ones.  Within a step the order is arbitrary; results do not depend
// on it (a block's G columns are written by one warp in fixed pair order).
__global__ void block_order_kernel(const BlockOrderArgs P) {
    const int c = blockIdx.x;
    const int n = P.n[c];
    if (n <= 0) return;
    const float* __restrict__ cost = P.cost + (long long)c * P.stride;
    int* __restrict__ order = P.order + (long long)c * P.stride;
    __shared__ unsigned cnt[256];
    for (int b = threadIdx.x; b < 256; b += blockDim.x) cnt[b] = 0u;
    __syncthreads();
    auto bucket = [](float x) {
        // 255 - 8 log2(1 + cost), clamped: bucket 0 holds the costliest
        const float l = 8.0f * __log2f(1.0f + fmaxf(x, 0.0f));
        const int b = 255 - (int)fminf(l, 255.0f);
        return b < 0 ? 0 : b;
    };
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        atomicAdd(&cnt[bucket(cost[i])], 1u);
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned run = 0;
        for (int b = 0; b < 256; ++b) {
            const unsigned t = cnt[b];
            cnt[b] = run;
            run += t;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        order[atomicAdd(&cnt[bucket(cost[i])], 1u)] = i;
}

cudaError_t launch_block_order(const BlockOrderArgs& P, cudaStream_t s) {
    block_order_kernel<<<kClasses, 1024, 0, s>>>(P);
    return cudaGetLastError();
}

// -- semilocal XC flow (reference gpu/xc.py:130-201) -------------------------
// Density parameters at every point: rho = sum_mu T0 X0, grad_d = 2 sum_mu
// T0 X_d and, for MGGA, tau = 1/2 sum_d sum_mu T_d X_d, with X (4, nao, ld)
// the FP64 AO values and gradients and T (1 or 4, nao, ld) = fl32(D^T X_d)
// from the FP64-accurate F GEMM.  Products in FP32 (the reference's flow is
// FP32 throughout), summed in FP32 over 8 AOs and in FP64 across groups.
// Points at or past npts: 0.
//
// Bound by HBM (48 bytes per point and AO for MGGA).  A block takes 64 points,
// two a lane, and its eight warps the groups of 8 AOs in turn, so that a tile
// of the flow (58,000 points) has 7,000 warps in flight; one thread per point
// left 1.5 CTAs an SM waiting on their loads.  X is rounded on the integer
// pipe: a conversion instruction per element takes as long as its 8 bytes.
// 16 waters (384 AOs, 233,999 points), meta-GGA: 2.75 -> 1.38 ms.
template<bool V>
__device__ __forceinline__ double2 load2(const double* p) {
    if constexpr (V) return *reinterpret_cast<const double2*>(p);
    else return make_double2(p[0], p[1]);
}
template<bool V>
__device__ __forceinline__ float2 load2(const float* p) {
    if constexpr (V) return *reinterpret_cast<const float2*>(p);
    else return make_float2(p[0], p[1]);
}
// both elements of a pair load at every even offset from these
inline bool pair_aligned(const void* f64_a, const void* f64_b, const void* f32) {
    return (((uintptr_t)f64_a | (uintptr_t)f64_b) & 15) == 0 && ((uintptr_t)f32 & 7) == 0;
}

template<bool MGGA, bool V>
__global__ void __launch_bounds__(256)
xc_rho_kernel(const double* __restrict__ X, const float* __restrict__ T, int nao, int64_t ld,
              int64_t npts, double* __restrict__ rho) {
    constexpr int NK = MGGA ? 5 : 4;
    __shared__ double2 sum[8][NK][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t g = (int64_t)blockIdx.x * 64 + 2 * lane;
    const int64_t pl = (int64_t)nao * ld;
    double2 acc[NK];
#pragma unroll
    for (int k = 0; k < NK; ++k) acc[k] = make_double2(0.0, 0.0);
    if (g < ld) {
        for (int m0 = 8 * warp; m0 < nao; m0 += 64) {
            float2 part[NK];
#pragma unroll
            for (int k = 0; k < NK; ++k) part[k] = make_float2(0.0f, 0.0f);
            const int m1 = min(nao, m0 + 8);
#pragma unroll 4
            for (int mu = m0; mu < m1; ++mu) {
                const int64_t o = (int64_t)mu * ld + g;
                const float2 t0 = load2<V>(T + o);
                float2 x[4];
#pragma unroll
                for (int d = 0; d < 4; ++d) {
                    const double2 xd = load2<V>(X + d * pl + o);
                    x[d] = make_float2(to_f32(xd.x), to_f32(xd.y));
                    part[d].x = fmaf(t0.x, x[d].x, part[d].x);
                    part[d].y = fmaf(t0.y, x[d].y, part[d].y);
                }
                if constexpr (MGGA) {
#pragma unroll
                    for (int d = 1; d < 4; ++d) {
                        const float2 t = load2<V>(T + d * pl + o);
                        part[4].x = fmaf(t.x, x[d].x, part[4].x);
                        part[4].y = fmaf(t.y, x[d].y, part[4].y);
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < NK; ++k) {
                acc[k].x += to_f64(part[k].x);
                acc[k].y += to_f64(part[k].y);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < NK; ++k) sum[warp][k][lane] = acc[k];
    __syncthreads();
    // warp k adds quantity k of the block's 64 points in warp order
    if (warp < 5 && g < ld) {
        double2 r = make_double2(0.0, 0.0);
        if (warp < NK) {
#pragma unroll
            for (int w = 0; w < 8; ++w) {
                r.x += sum[w][warp][lane].x;
                r.y += sum[w][warp][lane].y;
            }
        }
        const double f = warp == 0 ? 1.0 : (warp == 4 ? 0.5 : 2.0);
        rho[warp * ld + g] = g < npts ? f * r.x : 0.0;
        rho[warp * ld + g + 1] = g + 1 < npts ? f * r.y : 0.0;
    }
}

cudaError_t launch_xc_rho(const double* X, const float* T, int nao, int64_t ld,
                          int64_t npts, int mgga, double* rho, cudaStream_t s) {
    if (ld <= 0) return cudaSuccess;
    const unsigned grid = (unsigned)((ld + 63) / 64);
    if (!pair_aligned(X, X, T))
        (mgga ? xc_rho_kernel<true, false> : xc_rho_kernel<false, false>)
            <<<grid, 256, 0, s>>>(X, T, nao, ld, npts, rho);
    else
        (mgga ? xc_rho_kernel<true, true> : xc_rho_kernel<false, true>)
            <<<grid, 256, 0, s>>>(X, T, nao, ld, npts, rho);
    return cudaGetLastError();
}

// The Fock-side planes, FP32 (nao, ld) each: G0 = 1/2 v0 X0 + sum_d v_d X_d
// (the reference's aow without the weights, which the K GEMM applies) and,
// for MGGA, G_d = 1/2 vtau X_d (d = x, y, z); v (5, ld) FP64 are the
// density-parameter derivatives (chain rule applied).  Points at or past
// npts: 0.  Bound by HBM (48 bytes per point and AO for MGGA): a thread keeps
// v of two points for eight rows and rounds X on the integer pipe.  16 waters
// as above: 1.63 -> 1.11 ms.
constexpr int kAowRows = 8;

template<bool MGGA, bool V>
__global__ void __launch_bounds__(128)
xc_aow_kernel(const double* __restrict__ X, const double* __restrict__ v, int nao, int64_t ld,
              int64_t npts, float* __restrict__ G) {
    const int64_t g = 2 * ((int64_t)blockIdx.x * blockDim.x + threadIdx.x);
    if (g >= ld) return;
    const int m0 = blockIdx.y * kAowRows, m1 = min(nao, m0 + kAowRows);
    const int64_t pl = (int64_t)nao * ld;
    const bool in[2] = {g < npts, g + 1 < npts};
    constexpr int NK = MGGA ? 5 : 4;
    float2 u[NK];
#pragma unroll
    for (int k = 0; k < NK; ++k) {
        const double2 t = load2<V>(v + k * ld + g);
        const bool half = k == 0 || k == 4;
        u[k].x = in[0] ? (float)(half ? 0.5 * t.x : t.x) : 0.0f;
        u[k].y = in[1] ? (float)(half ? 0.5 * t.y : t.y) : 0.0f;
    }
    auto store = [&](float* p, float a, float b) {
        a = in[0] ? a : 0.0f;
        b = in[1] ? b : 0.0f;
        if constexpr (V) {
            *reinterpret_cast<float2*>(p) = make_float2(a, b);
        } else {
            p[0] = a;
            p[1] = b;
        }
    };
#pragma unroll 2
    for (int mu = m0; mu < m1; ++mu) {
        const int64_t o = (int64_t)mu * ld + g;
        float2 x[4];
#pragma unroll
        for (int d = 0; d < 4; ++d) {
            const double2 xd = load2<V>(X + d * pl + o);
            x[d] = make_float2(to_f32(xd.x), to_f32(xd.y));
        }
        float2 a = make_float2(u[0].x * x[0].x, u[0].y * x[0].y);
#pragma unroll
        for (int d = 1; d < 4; ++d) {
            a.x = fmaf(u[d].x, x[d].x, a.x);
            a.y = fmaf(u[d].y, x[d].y, a.y);
        }
        store(G + o, a.x, a.y);
        if constexpr (MGGA) {
#pragma unroll
            for (int d = 1; d < 4; ++d)
                store(G + d * pl + o, u[4].x * x[d].x, u[4].y * x[d].y);
        }
    }
}

cudaError_t launch_xc_aow(const double* X, const double* v, int nao, int64_t ld,
                          int64_t npts, int mgga, float* G, cudaStream_t s) {
    if (ld <= 0 || nao <= 0) return cudaSuccess;
    const dim3 grid((unsigned)((ld + 255) / 256), (unsigned)((nao + kAowRows - 1) / kAowRows));
    if (!pair_aligned(X, v, G))
        (mgga ? xc_aow_kernel<true, false> : xc_aow_kernel<false, false>)
            <<<grid, 128, 0, s>>>(X, v, nao, ld, npts, G);
    else
        (mgga ? xc_aow_kernel<true, true> : xc_aow_kernel<false, true>)
            <<<grid, 128, 0, s>>>(X, v, nao, ld, npts, G);
    return cudaGetLastError();
}

// GGA density in FP64 (the VV10 flow, gpu/vv10.py:286-291): rho = sum_mu T X_0,
// grad_d = 2 sum_mu T X_d.  A block takes 32 points; its eight warps take the
// rows in turn (256-byte rows, four planes read once beside T) and their sums
// are added in warp order.  Bound by HBM: 40 bytes per (point, AO) against 4
// FP64 FMAs.
template<typename T>
__global__ void __launch_bounds__(256)
gga_rho_kernel(const double* __restrict__ X, const T* __restrict__ t, int nao, int64_t ld,
               int64_t npts, double* __restrict__ rho) {
    __shared__ double part[8][4][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t g = (int64_t)blockIdx.x * 32 + lane;      // ld is a multiple of 32
    const int64_t pl = (int64_t)nao * ld;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
    for (int mu = warp; mu < nao; mu += 8) {
        const int64_t o = (int64_t)mu * ld + g;
        const double tv = (double)t[o];
#pragma unroll
        for (int d = 0; d < 4; ++d) acc[d] = fma(tv, X[d * pl + o], acc[d]);
    }
#pragma unroll
    for (int d = 0; d < 4; ++d) part[warp][d][lane] = acc[d];
    __syncthreads();
    if (warp < 4) {
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < 8; ++w) s += part[w][warp][lane];
        rho[warp * ld + g] = g < npts ? (warp ? 2.0 * s : s) : 0.0;
    }
}

cudaError_t launch_gga_rho(const double* X, const void* t, bool t32, int nao, int64_t ld,
                           int64_t npts, double* rho, cudaStream_t s) {
    if (ld <= 0) return cudaSuccess;
    const unsigned grid = (unsigned)(ld / 32);
    if (t32)
        gga_rho_kernel<<<grid, 256, 0, s>>>(X, static_cast<const float*>(t), nao, ld, npts,
                                            rho);
    else
        gga_rho_kernel<<<grid, 256, 0, s>>>(X, static_cast<const double*>(t), nao, ld, npts,
                                            rho);
    return cudaGetLastError();
}

// The Fock-side plane of a GGA potential in FP64: sum_d v_d X_d, one thread
// per AO and two points (HBM-bound: 32 bytes read and 8 written per element).
template<typename T, bool V>
__global__ void gga_aow_kernel(const double* __restrict__ X, const double* __restrict__ v,
                               int nao, int64_t ld, int64_t npts, T* __restrict__ G) {
    const int64_t g = 2 * ((int64_t)blockIdx.x * blockDim.x + threadIdx.x);
    if (g >= ld) return;
    const int64_t pl = (int64_t)nao * ld, o = (int64_t)blockIdx.y * ld + g;
    double a = 0.0, b = 0.0;
#pragma unroll
    for (int d = 0; d < 4; ++d) {
        const double2 x = load2<V>(X + d * pl + o);
        const double2 u = load2<V>(v + d * ld + g);
        a = fma(u.x, x.x, a);
        b = fma(u.y, x.y, b);
    }
    G[o] = (T)(g < npts ? a : 0.0);
    G[o + 1] = (T)(g + 1 < npts ? b : 0.0);
}

cudaError_t launch_gga_aow(const double* X, const double* v, int nao, int64_t ld,
                           int64_t npts, bool g32, void* G, cudaStream_t s) {
    if (ld <= 0 || nao <= 0) return cudaSuccess;
    const dim3 grid((unsigned)((ld / 2 + 255) / 256), (unsigned)nao);
    const bool al = pair_aligned(X, v, nullptr);
    if (g32)
        (al ? gga_aow_kernel<float, true> : gga_aow_kernel<float, false>)
            <<<grid, 256, 0, s>>>(X, v, nao, ld, npts, static_cast<float*>(G));
    else
        (al ? gga_aow_kernel<double, true> : gga_aow_kernel<double, false>)
            <<<grid, 256, 0, s>>>(X, v, nao, ld, npts, static_cast<double*>(G));
    return cudaGetLastError();
}

cudaError_t launch_gsum(const float* gc, const int4* src, int nao, int64_t ld,
                        float* G, cudaStream_t s) {
    if (nao <= 0 || ld <= 0) return cudaSuccess;
    const int64_t quads = ld / 4;
    dim3 grid((unsigned)((quads + 255) / 256), (unsigned)nao);
    gsum_kernel<<<grid, 256, 0, s>>>(gc, src, ld, G);
    return cudaGetLastError();
}

cudaError_t launch_gsum2(const GSum2& g, int nom, const int4* src, int nao, int64_t ld,
                         cudaStream_t s) {
    if (nao <= 0 || ld <= 0) return cudaSuccess;
    const int64_t quads = ld / 4;
    dim3 grid((unsigned)((quads + 255) / 256), (unsigned)nao, (unsigned)nom);
    gsum2_kernel<<<grid, 256, 0, s>>>(g, src, ld);
    return cudaGetLastError();
}

// -- FP64 AO evaluation (gpu/ao_eval.py:186-329, deriv 0 and 1) -------------
// One thread per (point, centre), threads of a block on consecutive points:
// every AO column is written coalesced, and r - A and r^2 serve all shells of
// the centre.  Bound by the FP64 pipe (2 lanes per clock and SM) where the
// writes alone would take a tenth of the time: the exponential runs on the
// integer pipe, the angular factors skip the zeros of the transform, and the
// gradient is rad1 S d + rad0 grad S from the solid harmonic S and its
// derivatives rather than from every Cartesian component.  648 AOs x 384,998
// points: 6.0 -> 1.4 ms; with gradients, 442 x 157,256: 3.5 -> 1.1 ms.
__constant__ double c_c2s0[1];
__constant__ double c_c2s1[9];
__constant__ double c_c2s2[30];
__constant__ double c_c2s3[70];

template<int L>
__device__ __forceinline__ const double* c2s_ptr() {
    if constexpr (L == 0) return c_c2s0;
    else if constexpr (L == 1) return c_c2s1;
    else if constexpr (L == 2) return c_c2s2;
    else return c_c2s3;
}

__constant__ unsigned long long c_exp2m[64];            // the table of exp_neg

// a < 70, on the integer pipe (a >= 0; false for a NaN of either sign): a
// primitive below exp(-70) ~ 4e-31 is zero at FP64 parity with any AO value of
// order one
__device__ __forceinline__ bool below70(const double a) {
    return (unsigned)__double2hiint(a) < 0x40518000u;
}

// The real solid harmonics S_m (NS) of a shell at (dx, dy, dz) and, with D,
// their derivatives G (3 x NS).
template<int L, bool D>
__device__ __forceinline__ void solid(const double dx, const double dy, const double dz,
                                      double* S, double* G) {
    using namespace f64;
    constexpr int NC = ncart_c(L), NS = 2 * L + 1;
    const double* c2s = c2s_ptr<L>();
    double p[3][L + 1];
    p[0][0] = p[1][0] = p[2][0] = 1.0;
#pragma unroll
    for (int e = 1; e <= L; ++e) {
        p[0][e] = e == 1 ? dx : p[0][e - 1] * dx;
        p[1][e] = e == 1 ? dy : p[1][e - 1] * dy;
        p[2][e] = e == 1 ? dz : p[2][e - 1] * dz;
    }
    auto mono = [&](int i, int j, int k) -> double {
        double v = 1.0;
        bool one = true;
        if (i) { v = p[0][i]; one = false; }
        if (j) { v = one ? p[1][j] : v * p[1][j]; one = false; }
        if (k) v = one ? p[2][k] : v * p[2][k];
        return v;
    };
    double t[4][NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const int e[3] = {cx(L, c), cy(L, c), cz(L, c)};
        t[3][c] = mono(e[0], e[1], e[2]);
        if constexpr (D) {
#pragma unroll
            for (int x = 0; x < 3; ++x)
                if (e[x]) {
                    const double v = mono(e[0] - (x == 0), e[1] - (x == 1), e[2] - (x == 2));
                    t[x][c] = e[x] == 1 ? v : (double)e[x] * v;
                }
        }
    }
#pragma unroll
    for (int m = 0; m < NS; ++m) {
        bool first = true, gfirst[3] = {true, true, true};
        S[m] = 0.0;
        if constexpr (D) G[m] = G[NS + m] = G[2 * NS + m] = 0.0;
#pragma unroll
        for (int c = 0; c < NC; ++c)
            if (c2s_nz(L, c, m)) {
                const double w = c2s[c * NS + m];
                S[m] = first ? w * t[3][c] : fma(w, t[3][c], S[m]);
                first = false;
                if constexpr (D) {
                    const int e[3] = {cx(L, c), cy(L, c), cz(L, c)};
#pragma unroll
                    for (int x = 0; x < 3; ++x)
                        if (e[x]) {
                            G[x * NS + m] = gfirst[x] ? w * t[x][c]
                                                      : fma(w, t[x][c], G[x * NS + m]);
                            gfirst[x] = false;
                        }
                }
            }
    }
}

// whether d S_m / d x_a vanishes identically (m and a known at compile time)
template<int L>
__device__ __forceinline__ constexpr bool solid_flat(const int m, const int a) {
    using namespace f64;
    for (int c = 0; c < ncart_c(L); ++c)
        if (c2s_nz(L, c, m) && (a == 0 ? cx(L, c) : a == 1 ? cy(L, c) : cz(L, c))) return false;
    return true;
}

// One shell at one point.  For R(r) S with R = sum c exp(-a r^2): the value
// rad0 S and, with D, the gradient rad1 S d + rad0 grad S, rad1 = sum c (-2 a)
// exp(-a r^2) (gpu/ao_eval.py:305-319).
template<int L, bool D>
__device__ __forceinline__ void ao_shell(const AoArgs& A, const int sh, const int64_t g,
                                         const double dx, const double dy, const double dz,
                                         const double r2, const float r2f,
                                         const unsigned long long* etab) {
    constexpr int NS = 2 * L + 1;
    const int np = A.sh_np[sh], nc = A.sh_nc[sh];
    const double* ex = A.exps + A.sh_eoff[sh];
    const double* co = A.coeffs + A.sh_coff[sh];
    const int ao0 = A.sh_ao0[sh];
    const int64_t plane = (int64_t)A.nao * A.ld;
    // the angular factors are formed on the first contraction with a live
    // primitive: at most points of a cluster a shell has none
    double S[NS], G[D ? 3 * NS : 1];
    bool have = false;
    for (int ci = 0; ci < nc; ++ci) {
        double rad0 = 0.0, rad1 = 0.0;
        bool live = false;
        for (int k = 0; k < np; ++k) {
            // far out: decided in FP32 (exp(-71) and below), no FP64 product
            const double exk = ex[k];
            if (f64::narrow(exk) * r2f > 71.0f) continue;
            const double a = exk * r2;
            if (!below70(a)) continue;
            const double e = f64::exp_neg(a, etab);
            if constexpr (D) {
                const double w = co[k * nc + ci] * e;
                rad0 += w;
                rad1 = fma(-f64::twice(exk), w, rad1);
            } else {
                rad0 = fma(co[k * nc + ci], e, rad0);
            }
            live = true;
        }
        double* out = A.X + (int64_t)(ao0 + ci * NS) * A.ld + g;
        if (!live) {
#pragma unroll
            for (int m = 0; m < NS; ++m)
#pragma unroll
                for (int p = 0; p < (D ? 4 : 1); ++p) out[p * plane + (int64_t)m * A.ld] = 0.0;
            continue;
        }
        if constexpr (L == 1) {
            // S_m = c d_m: fewer products than by S
            const double c = c_c2s1[0], d[3] = {dx, dy, dz}, v0 = rad0 * c;
#pragma unroll
            for (int m = 0; m < 3; ++m) out[(int64_t)m * A.ld] = v0 * d[m];
            if constexpr (D) {
                const double t = rad1 * c;
#pragma unroll
                for (int m = 0; m < 3; ++m) {
                    const double u = t * d[m];
#pragma unroll
                    for (int x = m; x < 3; ++x) {
                        const double g2 = x == m ? fma(u, d[x], v0) : u * d[x];
                        out[(x + 1) * plane + (int64_t)m * A.ld] = g2;
                        if (x != m) out[(m + 1) * plane + (int64_t)x * A.ld] = g2;
                    }
                }
            }
            continue;
        }
        if (!have) {
            solid<L, D>(dx, dy, dz, S, G);
            have = true;
        }
#pragma unroll
        for (int m = 0; m < NS; ++m) {
            double* o = out + (int64_t)m * A.ld;
            o[0] = rad0 * S[m];
            if constexpr (D) {
                const double rs = rad1 * S[m], d[3] = {dx, dy, dz};
#pragma unroll
                for (int x = 0; x < 3; ++x)
                    o[(x + 1) * plane] = solid_flat<L>(m, x)
                                             ? rs * d[x]
                                             : fma(rs, d[x], rad0 * G[x * NS + m]);
            }
        }
    }
}

template<bool D>
__global__ void __launch_bounds__(128) ao_eval_kernel(const AoArgs A) {
    __shared__ unsigned long long etab[64];
    if (threadIdx.x < 64) etab[threadIdx.x] = c_exp2m[threadIdx.x];
    __syncthreads();
    const int s0 = A.centre[blockIdx.y], s1 = A.centre[blockIdx.y + 1];
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= A.ld) return;
    if (g >= A.npts) {
        const int64_t plane = (int64_t)A.nao * A.ld;
        const int last = s1 - 1;
        const int end = A.sh_ao0[last] + A.sh_nc[last] * (2 * A.sh_l[last] + 1);
        for (int i = A.sh_ao0[s0]; i < end; ++i)
            for (int c = 0; c < (D ? 4 : 1); ++c) A.X[c * plane + (int64_t)i * A.ld + g] = 0.0;
        return;
    }
    const double dx = A.coords[g * 3] - A.sh_ctr[s0 * 3];
    const double dy = A.coords[g * 3 + 1] - A.sh_ctr[s0 * 3 + 1];
    const double dz = A.coords[g * 3 + 2] - A.sh_ctr[s0 * 3 + 2];
    const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
    const float r2f = f64::narrow(r2);
    for (int sh = s0; sh < s1; ++sh)
        switch (A.sh_l[sh]) {
        case 0: ao_shell<0, D>(A, sh, g, dx, dy, dz, r2, r2f, etab); break;
        case 1: ao_shell<1, D>(A, sh, g, dx, dy, dz, r2, r2f, etab); break;
        case 2: ao_shell<2, D>(A, sh, g, dx, dy, dz, r2, r2f, etab); break;
        default: ao_shell<3, D>(A, sh, g, dx, dy, dz, r2, r2f, etab); break;
        }
}

cudaError_t launch_ao_eval_d1(const AoArgs& a, cudaStream_t s) {
    if (a.ld <= 0 || a.ncentre <= 0) return cudaSuccess;
    dim3 grid((unsigned)((a.ld + 127) / 128), (unsigned)a.ncentre);
    ao_eval_kernel<true><<<grid, 128, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_ao_eval(const AoArgs& a, cudaStream_t s) {
    if (a.ld <= 0 || a.ncentre <= 0) return cudaSuccess;
    dim3 grid((unsigned)((a.ld + 127) / 128), (unsigned)a.ncentre);
    ao_eval_kernel<false><<<grid, 128, 0, s>>>(a);
    return cudaGetLastError();
}

// c2s tables filled by the host (same formula as the host pair builder)
cudaError_t upload_exp_table(const unsigned long long* t64) {
    return cudaMemcpyToSymbol(c_exp2m, t64, sizeof(unsigned long long) * 64);
}

cudaError_t upload_c2s_tables(const double* t0, const double* t1,
                              const double* t2, const double* t3) {
    cudaError_t e;
    if ((e = cudaMemcpyToSymbol(c_c2s0, t0, sizeof(double) * 1)) != cudaSuccess) return e;
    if ((e = cudaMemcpyToSymbol(c_c2s1, t1, sizeof(double) * 9)) != cudaSuccess) return e;
    if ((e = cudaMemcpyToSymbol(c_c2s2, t2, sizeof(double) * 30)) != cudaSuccess) return e;
    return cudaMemcpyToSymbol(c_c2s3, t3, sizeof(double) * 70);
}

// -- dense contracted spherical A (validation, gpu/int3c1e.py:230-271) -------
// One thread per (point, pair), run-time L, arrays in local memory.  Uses
// the same pair tables and the same Boys / R / E math as the fused kernels
// but forms the Cartesian block explicitly.
__constant__ float c_c2s_f[4][70];

__device__ void cart_comp(int l, int c, int* i, int* j, int* k) {
    int r = 0;
    while ((r + 1) * (r + 2) / 2 <= c) ++r;
    *i = l - r;
    *j = r - (c - r * (r + 1) / 2);
    *k = l - *i - *j;
}

__device__ int e_index(int la, int lb, int i, int j, int t) {
    // position of (i, j, t) in the packed per-axis list (E^{00}_0 excluded)
    int n = 0;
    for (int ii = 0; ii <= la; ++ii)
        for (int jj = 0; jj <= lb; ++jj)
            for (int tt = 0; tt <= ii + jj; ++tt) {
                if (ii == 0 && jj == 0) continue;
                if (ii == i && jj == j && tt == t) return n;
                ++n;
            }
    return -1;
}

__device__ float e_val(const float* Em, int cnt, int ax, int la, int lb,
                       int i, int j, int t) {
    if (i == 0 && j == 0) return t == 0 ? 1.0f : 0.0f;
    return Em[ax * cnt + e_index(la, lb, i, j, t)];
}

template<int LMAXC>
__device__ void boys_dyn(int L, float T, float* F, const float4* tab) {
    switch (L) {
    case 0: boys_fp32<0>(T, F, tab); break;
    case 1: boys_fp32<1>(T, F, tab); break;
    case 2: boys_fp32<2>(T, F, tab); break;
    case 3: boys_fp32<3>(T, F, tab); break;
    case 4: boys_fp32<4>(T, F, tab); break;
    case 5: boys_fp32<5>(T, F, tab); break;
    default: boys_fp32<6>(T, F, tab); break;
    }
}

struct DenseArgs {
    CosxArgs a;
    int npairs, nao;
    const int* pclass;
    const int* pl;          // (npairs, 2): la, lb
    const int* estride;     // per class, floats
    float* out;             // (npts, nao, nao)
};

__global__ void dense_kernel(const DenseArgs D) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t total = (int64_t)D.a.npts * D.npairs;
    if (idx >= total) return;
    const int64_t g = idx / D.npairs;
    const int k = (int)(idx - g * D.npairs);
    const CosxArgs& A = D.a;
    const int4 hdr = A.hdr[k];
    const int ia0 = hdr.x, ib0 = hdr.y, pp0 = hdr.z, npp = hdr.w & 0xffff;
    const int cls = D.pclass[k];
    const int la = D.pl[2 * k], lb = D.pl[2 * k + 1], L = la + lb;
    const int nca = (la + 1) * (la + 2) / 2, ncb = (lb + 1) * (lb + 2) / 2;
    int cnt = 0;
    for (int i = 0; i <= la; ++i)
        for (int j = 0; j <= lb; ++j) cnt += i + j + 1;
    cnt -= 1;
    const float gxh = A.gxyz_hi[g], gyh = A.gxyz_hi[A.ld + g], gzh = A.gxyz_hi[2 * A.ld + g];
    const float gxl = A.gxyz_lo[g], gyl = A.gxyz_lo[A.ld + g], gzl = A.gxyz_lo[2 * A.ld + g];
    float Ac[100];
    for (int i = 0; i < 100; ++i) Ac[i] = 0.0f;
    float R[7][7][7];
    for (int m = pp0; m < pp0 + npp; ++m) {
        const float4 ph = A.geo[2 * m], pl = A.geo[2 * m + 1];
        const float dx = (ph.x - gxh) + (pl.x - gxl);
        const float dy = (ph.y - gyh) + (pl.y - gyl);
        const float dz = (ph.z - gzh) + (pl.z - gzl);
        const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
        const float* o = (const float*)(A.om + 5 * (int64_t)m);
        const float T = fmaf(o[0], r2, o[1] * r2);
        float Fb[7];
        boys_dyn<6>(L, T, Fb, A.boys);
        for (int t = 0; t < 7; ++t)
            for (int u = 0; u < 7; ++u)
                for (int v = 0; v < 7; ++v) R[t][u][v] = 0.0f;
        for (int n = L; n >= 0; --n) {
            const int mm = L - n;
            for (int u = 0; u < mm; ++u)
                for (int v = 0; v < mm - u; ++v)
                    for (int t = mm - u - v; t >= 1; --t)
                        R[t][u][v] = (t == 1) ? dx * R[0][u][v]
                            : fmaf(dx, R[t - 1][u][v], (float)(t - 1) * R[t - 2][u][v]);
            for (int v = 0; v < mm; ++v)
                for (int u = mm - v; u >= 1; --u)
                    R[0][u][v] = (u == 1) ? dy * R[0][0][v]
                        : fmaf(dy, R[0][u - 1][v], (float)(u - 1) * R[0][u - 2][v]);
            for (int v = mm; v >= 1; --v)
                R[0][0][v] = (v == 1) ? dz * R[0][0][0]
                    : fmaf(dz, R[0][0][v - 1], (float)(v - 1) * R[0][0][v - 2]);
            R[0][0][0] = fmaf(o[2 + 2 * n], Fb[n], o[3 + 2 * n] * Fb[n]);
        }
        const float* Em = (const float*)A.Ecls[cls] +
                          (int64_t)(m - A.pp_begin[cls]) * D.estride[cls];
        for (int ca = 0; ca < nca; ++ca) {
            int i, j, kk;
            cart_comp(la, ca, &i, &j, &kk);
            for (int cb = 0; cb < ncb; ++cb) {
                int ip, jp, kp;
                cart_comp(lb, cb, &ip, &jp, &kp);
                float s = 0.0f;
                for (int t = 0; t <= i + ip; ++t) {
                    const float ex = e_val(Em, cnt, 0, la, lb, i, ip, t);
                    for (int u = 0; u <= j + jp; ++u) {
                        const float ey = e_val(Em, cnt, 1, la, lb, j, jp, u);
                        for (int v = 0; v <= kk + kp; ++v)
                            s += ex * ey * e_val(Em, cnt, 2, la, lb, kk, kp, v) * R[t][u][v];
                    }
                }
                Ac[ca * ncb + cb] += s;
            }
        }
    }
    const int na = 2 * la + 1, nb = 2 * lb + 1;
    float* row = D.out + g * (int64_t)D.nao * D.nao;
    for (int mu = 0; mu < na; ++mu)
        for (int nu = 0; nu < nb; ++nu) {
            float v = 0.0f;
            for (int ca = 0; ca < nca; ++ca) {
                const float cam = la <= 1 ? (ca == mu ? 1.0f : 0.0f)
                                          : c_c2s_f[la][ca * na + mu];
                if (cam == 0.0f) continue;
                for (int cb = 0; cb < ncb; ++cb) {
                    const float cbn = lb <= 1 ? (cb == nu ? 1.0f : 0.0f)
                                              : c_c2s_f[lb][cb * nb + nu];
                    v += cam * cbn * Ac[ca * ncb + cb];
                }
            }
            row[(int64_t)(ia0 + mu) * D.nao + ib0 + nu] = v;
            row[(int64_t)(ib0 + nu) * D.nao + ia0 + mu] = v;
        }
}

cudaError_t upload_c2s_f(const float* all /* 4 x 70 */) {
    return cudaMemcpyToSymbol(c_c2s_f, all, sizeof(float) * 4 * 70);
}

cudaError_t launch_dense_impl(const CosxArgs& a, int npairs, const int* pclass,
                              const int* pl, const int* estride, int nao,
                              float* out, cudaStream_t s) {
    DenseArgs D;
    D.a = a; D.npairs = npairs; D.nao = nao; D.pclass = pclass; D.pl = pl;
    D.estride = estride; D.out = out;
    const int64_t total = (int64_t)a.npts * npairs;
    if (total <= 0) return cudaSuccess;
    dense_kernel<<<(unsigned)((total + 63) / 64), 64, 0, s>>>(D);
    return cudaGetLastError();
}

// -- Boys batch (tests, gpu/boys.py:181-189) ---------------------------------
template<int L>
__global__ void boys_batch_kernel(const float* __restrict__ t, int64_t n,
                                  const float4* __restrict__ tab,
                                  float* __restrict__ out) {
    __shared__ float4 stab[145 * 5];
    for (int i = threadIdx.x; i < 145 * 5; i += blockDim.x) stab[i] = tab[i];
    __syncthreads();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float F[L + 1];
    boys_fp32<L>(t[i], F, stab);
#pragma unroll
    for (int m = 0; m <= L; ++m) out[m * n + i] = F[m];
}

cudaError_t launch_boys(const float* t, int64_t n, int nmax,
                        const float4* tab, float* out, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const unsigned blocks = (unsigned)((n + 255) / 256);
    switch (nmax) {
    case 0: boys_batch_kernel<0><<<blocks, 256, 0, s>>>(t, n, tab, out); break;
    case 1: boys_batch_kernel<1><<<blocks, 256, 0, s>>>(t, n, tab, out); break;
    case 2: boys_batch_kernel<2><<<blocks, 256, 0, s>>>(t, n, tab, out); break;
    case 3: boys_batch_kernel<3><<<blocks, 256, 0, s>>>(t, n, tab, out); break;
    case 4: boys_batch_kernel<4><<<blocks, 256, 0, s>>>(t, n, tab, out); break;
    case 5: boys_batch_kernel<5><<<blocks, 256, 0, s>>>(t, n, tab, out); break;
    case 6: boys_batch_kernel<6><<<blocks, 256, 0, s>>>(t, n, tab, out); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace wb

namespace wb {

// -- FP32 FMA throughput probe (the roofline denominator of the FP32-pipe
// kernels): 8 independent FMA chains per thread, nothing but FFMA in the
// loop; each thread writes one value so nothing is optimised away.
__global__ void fma_probe_kernel(int64_t iters, float* __restrict__ out) {
    float a0 = threadIdx.x * 1e-7f, a1 = a0 + 1e-7f, a2 = a0 + 2e-7f,
          a3 = a0 + 3e-7f, a4 = a0 + 4e-7f, a5 = a0 + 5e-7f, a6 = a0 + 6e-7f,
          a7 = a0 + 7e-7f;
    const float m = 0.999999f, c = 1e-7f;
    for (int64_t i = 0; i < iters; ++i) {
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            a0 = fmaf(a0, m, c); a1 = fmaf(a1, m, c); a2 = fmaf(a2, m, c);
            a3 = fmaf(a3, m, c); a4 = fmaf(a4, m, c); a5 = fmaf(a5, m, c);
            a6 = fmaf(a6, m, c); a7 = fmaf(a7, m, c);
        }
    }
    out[(int64_t)blockIdx.x * blockDim.x + threadIdx.x] =
        a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
}

// the same with packed FMAs (fma.rn.f32x2: two FP32 FMAs per instruction)
__global__ void fma2_probe_kernel(int64_t iters, float* __restrict__ out) {
    unsigned long long a[8];
    const float b0 = threadIdx.x * 1e-7f;
    for (int k = 0; k < 8; ++k) {
        const float lo = b0 + 2 * k * 1e-7f, hi = lo + 1e-7f;
        asm("mov.b64 %0, {%1, %2};" : "=l"(a[k]) : "f"(lo), "f"(hi));
    }
    unsigned long long m, c;
    asm("mov.b64 %0, {%1, %1};" : "=l"(m) : "f"(0.999999f));
    asm("mov.b64 %0, {%1, %1};" : "=l"(c) : "f"(1e-7f));
    for (int64_t i = 0; i < iters; ++i) {
#pragma unroll
        for (int k = 0; k < 16; ++k) {
#pragma unroll
            for (int r = 0; r < 8; ++r)
                asm volatile("fma.rn.f32x2 %0, %0, %1, %2;" : "+l"(a[r]) : "l"(m), "l"(c));
        }
    }
    float s = 0.0f;
    for (int k = 0; k < 8; ++k) {
        float lo, hi;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a[k]));
        s += lo + hi;
    }
    out[(int64_t)blockIdx.x * blockDim.x + threadIdx.x] = s;
}

cudaError_t launch_fma_probe(int64_t iters, int blocks, int threads,
                             float* out, cudaStream_t s, bool packed) {
    if (packed)
        fma2_probe_kernel<<<blocks, threads, 0, s>>>(iters, out);
    else
        fma_probe_kernel<<<blocks, threads, 0, s>>>(iters, out);
    return cudaGetLastError();
}

// -- screen mask (test aid) ---------------------------------------------------
// keep[blk * npairs + k] = 1 where the fused G kernels keep task (blk, k)
// at block level lv (blocks of 32 << lv points): the same screen_pair call,
// on the same block statistics and pair data, as the class kernels make.
__global__ void screen_mask_kernel(const CosxArgs A, const int lv, const int npairs,
                                   unsigned char* __restrict__ keep) {
    const int64_t total = (int64_t)A.nblk[lv] * npairs;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int blk = (int)(idx / npairs);
        const int k = (int)(idx - (int64_t)blk * npairs);
        int c = 0;
        while (c < kClasses - 1 && !(k >= A.cls_pb[c] && k < A.cls_pe[c])) ++c;
        bool kp = true;
        if (A.tol > 0.0f) {
            const int2 sh = A.pshell[k];
            const float* ms = A.blk_msh[lv] + (int64_t)blk * A.nvshell;
            kp = screen_pair(A.tol, A.bnd + A.pp_begin[c], A.bpref + A.pp_begin[c],
                             A.blk_cr[lv][blk], A.khdr[k], A.ptau[k],
                             max_nan(ms[sh.x], ms[sh.y]));
        }
        keep[idx] = kp ? 1 : 0;
    }
}

cudaError_t launch_screen_mask(const CosxArgs& a, int lv, int npairs,
                               unsigned char* keep, cudaStream_t s) {
    const int64_t total = (int64_t)a.nblk[lv] * npairs;
    if (total <= 0) return cudaSuccess;
    screen_mask_kernel<<<(unsigned)grid_stride_blocks(total, 256, 16), 256, 0, s>>>(
        a, lv, npairs, keep);
    return cudaGetLastError();
}

}  // namespace wb
