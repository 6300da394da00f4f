// Plain FP64 form of the fused screen + G kernels (templates shared by
// cosx_fp64.cu and cosx_fp64_f.cu): the same task set (the
// reference's locked bound on 32-point blocks, tol / 1.001) and the same
// McMurchie-Davidson algorithm as the FP32 class kernels, with every
// arithmetic step in FP64 and G accumulated in FP64.  It is the comparison
// point of the mixed-precision path and the operator of an FP64 tail; the
// reference runs that tail through stock PySCF on the CPU
// (staging/schedule.py:329-334).
//
// One warp owns one 32-point block (one point per lane) and walks its
// class's shell pairs in order; 32 pairs at a time each lane evaluates one
// pair's bound and a ballot keeps the warp on the kept ones.  Per task and
// point: the Boys values (fp64_boys.cuh), R_tuv in place, the Hermite sums
// axis by axis into the Cartesian block A_ab, summed over the primitive
// pairs; then G_A += c2s (A c2s^T F_B) and G_B += c2s (A^T c2s^T F_A)
// (diagonal pairs: G_A += c2s (A + A^T) / 2 c2s^T F_A).  F_A and the sums of
// G_A stay in registers over a run of pairs with one bra shell.  Each lane
// owns its point's column of its range's G and the classes run one after
// another on one stream, so every element has one writer and a fixed summation
// order; the ranges' G are added in order afterwards.
//
// What bounds it: the FP64 pipe, 2 lanes per clock and SM, 64 times below
// FP32.  Everything is arranged to spend few FP64 instructions, the other
// pipes being idle: factors that depend on the primitive pair alone come
// from a record formed once per omega (f64_records_kernel) instead of a
// division and a square root a lane, E^{00} = 1 and the zeros of the c2s
// tables are skipped, the block A is summed over the primitive pairs before
// F meets it, G_A and G_B are added by reductions in the L2 (no FP64
// instruction on the SM; one writer lane an element, so program order).
// Eight to sixteen warps an SM fill the pipe, so one CTA an SM with the
// whole register file and the Boys table in shared memory is enough.
// Measured on 8 waters (192 AOs, 70,478 points, both omegas), a whole K build:
// 180 -> 48.4 ms, the class kernels at 82-88 % of the FP64 pipe's issue rate.
#pragma once
#include <algorithm>
#include <cuda_runtime.h>

#include "cart.cuh"
#include "cosx_kernels.cuh"
#include "cosx_fp64.hpp"
#include "fp64_boys.cuh"

namespace wb {
namespace f64 {

constexpr __host__ __device__ int nr_c(int L) { return (L + 1) * (L + 2) * (L + 3) / 6; }
// packed index of R_tuv (t + u + v <= L): v-major, then u, then t
constexpr __host__ __device__ int ridx(int L, int t, int u, int v) {
    int k = 0;
    for (int vv = 0; vv < v; ++vv)
        for (int uu = 0; uu <= L - vv; ++uu) k += L - vv - uu + 1;
    for (int uu = 0; uu < u; ++uu) k += L - v - uu + 1;
    return k + t;
}
// offset of E^{i,j}_0 inside one axis block ([i][j][t], j <= lb)
constexpr __host__ __device__ int eoff(int lb, int i, int j) {
    int k = 0;
    for (int ii = 0; ii < i; ++ii)
        for (int jj = 0; jj <= lb; ++jj) k += ii + jj + 1;
    for (int jj = 0; jj < j; ++jj) k += i + jj + 1;
    return k;
}
constexpr __host__ __device__ int eaxis(int la, int lb) {
    return eoff(lb, la + 1, 0);
}

// c2s^T v (Cartesian components of a spherical vector) and c2s y
template<int L>
__device__ __forceinline__ void to_cart(const double* __restrict__ c2s,
                                        const double* s, double* c) {
#pragma unroll
    for (int i = 0; i < ncart_c(L); ++i) {
        if constexpr (L <= 1) {
            c[i] = s[i];
        } else {
            bool first = true;
            c[i] = 0.0;
#pragma unroll
            for (int m = 0; m < 2 * L + 1; ++m)
                if (c2s_nz(L, i, m)) {
                    const double t = c2s[(L - 2) * 30 + i * (2 * L + 1) + m];
                    c[i] = first ? t * s[m] : fma(t, s[m], c[i]);
                    first = false;
                }
        }
    }
}
template<int L>
__device__ __forceinline__ double to_sph(const double* __restrict__ c2s,
                                        const double* y, const int m) {
    if constexpr (L <= 1) {
        return y[m];
    } else {
        bool first = true;
        double a = 0.0;
#pragma unroll
        for (int i = 0; i < ncart_c(L); ++i)
            if (c2s_nz(L, i, m)) {
                const double t = c2s[(L - 2) * 30 + i * (2 * L + 1) + m];
                a = first ? t * y[i] : fma(t, y[i], a);
                first = false;
            }
        return a;
    }
}

// k r for a small k known at compile time
__device__ __forceinline__ double times(const int k, const double r) {
    return k == 1 ? r : (double)k * r;
}

// R_tuv (t + u + v <= L) at PC = (x, y, z) from r0[n] = R_000^(n), levels
// L .. 0 in place (each level reads only the level above)
template<int L>
__device__ __forceinline__ void fill_r64(const double* r0, const double x,
                                         const double y, const double z, double* R) {
#pragma unroll
    for (int n = L; n >= 0; --n) {
        const int m = L - n;
#pragma unroll
        for (int u = 0; u <= L; ++u)
#pragma unroll
            for (int v = 0; v <= L; ++v)
#pragma unroll
                for (int t = L; t >= 1; --t)
                    if (u < m && v < m - u && t <= m - u - v)
                        R[ridx(L, t, u, v)] =
                            t == 1 ? x * R[ridx(L, 0, u, v)]
                                   : fma(x, R[ridx(L, t - 1, u, v)],
                                         times(t - 1, R[ridx(L, t >= 2 ? t - 2 : 0, u, v)]));
#pragma unroll
        for (int v = 0; v <= L; ++v)
#pragma unroll
            for (int u = L; u >= 1; --u)
                if (v < m && u <= m - v)
                    R[ridx(L, 0, u, v)] =
                        u == 1 ? y * R[ridx(L, 0, 0, v)]
                               : fma(y, R[ridx(L, 0, u - 1, v)],
                                     times(u - 1, R[ridx(L, 0, u >= 2 ? u - 2 : 0, v)]));
#pragma unroll
        for (int v = L; v >= 1; --v)
            if (v <= m)
                R[ridx(L, 0, 0, v)] =
                    v == 1 ? z * R[0]
                           : fma(z, R[ridx(L, 0, 0, v - 1)],
                                 times(v - 1, R[ridx(L, 0, 0, v >= 2 ? v - 2 : 0)]));
        R[0] = r0[n];
    }
}

// A[a][b] += sum_tuv E^x_t E^y_u E^z_v R_tuv of one primitive pair, axis by
// axis: the x sums of one (i, i') serve every (j, j', k, k') with it
template<int LA, int LB>
__device__ __forceinline__ void hermite_block(const double* __restrict__ E,
                                              const double* R, double* A) {
    constexpr int L = LA + LB, NAX = eaxis(LA, LB), NCB = ncart_c(LB);
#pragma unroll
    for (int i = 0; i <= LA; ++i)
#pragma unroll
        for (int ip = 0; ip <= LB; ++ip) {
            const int M = L - i - ip;               // u + v <= M
            const double* ex = E + eoff(LB, i, ip);
            double h1[nr_c(L) > 1 ? (L + 1) * (L + 2) / 2 : 1];
#pragma unroll
            for (int u = 0; u <= L; ++u)
#pragma unroll
                for (int v = 0; v <= L; ++v)
                    if (u + v <= M) {
                        double s;
                        if (i + ip == 0) {
                            s = R[ridx(L, 0, u, v)];
                        } else {
                            s = ex[0] * R[ridx(L, 0, u, v)];
#pragma unroll
                            for (int t = 1; t <= L; ++t)
                                if (t <= i + ip) s = fma(ex[t], R[ridx(L, t, u, v)], s);
                        }
                        h1[u * (2 * M + 3 - u) / 2 + v] = s;
                    }
#pragma unroll
            for (int j = 0; j <= LA; ++j)
#pragma unroll
                for (int jp = 0; jp <= LB; ++jp)
                    if (j <= LA - i && jp <= LB - ip) {
                        const int k = LA - i - j, kp = LB - ip - jp;
                        const double* ey = E + NAX + eoff(LB, j, jp);
                        const double* ez = E + 2 * NAX + eoff(LB, k, kp);
                        const int ab = cidx(LA, i, j) * NCB + cidx(LB, ip, jp);
                        double s = A[ab];
                        if (k + kp == 0 && j + jp > 0) {
                            // one v: the y sum continues A
#pragma unroll
                            for (int u = 0; u <= L; ++u)
                                if (u <= j + jp)
                                    s = fma(ey[u], h1[u * (2 * M + 3 - u) / 2], s);
                            A[ab] = s;
                            continue;
                        }
                        if (j + jp + k + kp == 0 && i + ip > 0) {
                            // only this component uses the x sum
#pragma unroll
                            for (int t = 0; t <= L; ++t)
                                if (t <= i + ip) s = fma(ex[t], R[ridx(L, t, 0, 0)], s);
                            A[ab] = s;
                            continue;
                        }
#pragma unroll
                        for (int v = 0; v <= L; ++v)
                            if (v <= k + kp) {
                                double h2;
                                if (j + jp == 0) {
                                    h2 = h1[v];
                                } else {
                                    h2 = ey[0] * h1[v];
#pragma unroll
                                    for (int u = 1; u <= L; ++u)
                                        if (u <= j + jp)
                                            h2 = fma(ey[u], h1[u * (2 * M + 3 - u) / 2 + v], h2);
                                }
                                s = k + kp == 0 ? s + h2 : fma(ez[v], h2, s);
                            }
                        A[ab] = s;
                    }
        }
}

// pairs of one of nseg ranges, in whole units of align pairs.  The classes of
// d and f shells have few pairs and long tasks, so a range may be shorter than
// a screening chunk of 32 (C4H10 in TZVP has 10 pairs of f shells: its
// gradient 81.3 -> 74.4 ms against ranges of whole chunks).
__host__ __device__ constexpr int segment_pairs(int npairs, int nseg, int align = 1) {
    return ((npairs + nseg - 1) / nseg + align - 1) / align * align;
}

// threads of a CTA (one an SM): the light classes leave registers for
// sixteen warps, the others take 255 a thread
template<int LA, int LB, int NW>
struct F64Cta { static constexpr int kThreads = LA + LB <= (NW == 2 ? 1 : 2) ? 512 : 256; };

// NW = 2: two omegas in one pass (records rec and rec2, G and G2).  They share
// the screen, F, the distances and their square.  For the light classes, where
// those are a fifth to half of the work and the second block fits the
// registers: 8 waters (192 AOs, 70,478 points), a K build 58.1 -> 51.9 ms.
template<int LA, int LB, int NW>
__global__ void __launch_bounds__(F64Cta<LA, LB, NW>::kThreads, 1)
cosx_fp64_kernel(const CosxF64Args A, const int cls, const int pair_begin,
                 const int pair_end) {
    constexpr int L = LA + LB;
    constexpr int NCA = ncart_c(LA), NCB = ncart_c(LB);
    constexpr int NA = 2 * LA + 1, NB = 2 * LB + 1;
    constexpr int NAX = eaxis(LA, LB);
    extern __shared__ double stab[];
    load_boys<L>(A.boys, stab);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const long long ld = A.ld;
    const int pp_begin = A.pp_begin[cls];
    const float4* __restrict__ bnd = A.bnd + pp_begin;
    const float* __restrict__ bpref = A.bpref + pp_begin;
    const double* __restrict__ Ecls = A.E + A.e_base[cls];
    unsigned long long kept = 0, flops = 0, ints = 0;
    // An item is a block and one of nseg ranges of the pairs; each range adds
    // to a G of its own.  The first items go to the warps of all SMs in turn,
    // the others by the counter: a grid of few blocks still uses every SM's
    // pipe.
    const int nwarps = gridDim.x * (blockDim.x >> 5);
    const int nitem = A.nblk * A.nseg;
    const int seg_pairs = segment_pairs(pair_end - pair_begin, A.nseg);
    int item = (int)(threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    while (item < nitem) {
        const int seg = item / A.nblk, blk = item - seg * A.nblk;
        const int k0 = pair_begin + seg * seg_pairs;
        const int k1 = min(pair_end, k0 + seg_pairs);
        const int g0 = blk * 32 + lane;
        const bool ok = g0 < A.npts;
        const int g = ok ? g0 : A.npts - 1;
        const double gx = A.coords[3LL * g], gy = A.coords[3LL * g + 1],
                     gz = A.coords[3LL * g + 2];
        const double* __restrict__ Fp = A.F + g;
        double* const Gp[2] = {A.G + seg * A.gstride + g,
                               NW == 2 ? A.G2 + seg * A.gstride + g : nullptr};
        const float4 cr = A.blk_cr[blk];
        const float* __restrict__ ms = A.blk_msh + (long long)blk * A.nvshell;
        const int rem = A.npts - blk * 32;
        const int nvalid = rem < 32 ? rem : 32;
        int run = -1;                       // first AO of the bra shell held
        double fa[NCA], ya[NW][NCA];
        auto flush = [&]() {
            if (run < 0 || !ok) return;
#pragma unroll
            for (int w = 0; w < NW; ++w)
#pragma unroll
                for (int m = 0; m < NA; ++m)
                    atomicAdd(Gp[w] + (long long)(run + m) * ld, to_sph<LA>(A.c2s, ya[w], m));
        };
        for (int c0 = k0; c0 < k1; c0 += 32) {
            const int k = c0 + lane;
            bool keep = k < k1;
            if (keep && A.tol > 0.0f) {
                const int2 sh = A.pshell[k];
                keep = screen_pair(A.tol, bnd, bpref, cr, A.khdr[k], A.ptau[k],
                                   max_nan(ms[sh.x], ms[sh.y]));
            }
            unsigned mask = __ballot_sync(0xffffffffu, keep);
            if (keep) {
                flops += (unsigned long long)A.pflops[k] * nvalid * NW;
                ints += (unsigned long long)A.pnint[k] * nvalid * NW;
            }
            while (mask) {
                const int kk = c0 + __ffs(mask) - 1;
                mask &= mask - 1;
                kept += NW;
                const int4 hdr = A.khdr[kk];
                const int ia0 = hdr.x & 0xffff, ib0 = hdr.y & 0xffff;
                const int pp0 = pp_begin + hdr.z, npp = hdr.w & 0xffff;
                const bool diag = (hdr.w >> 16) != 0;
                if (ia0 != run) {
                    flush();
                    run = ia0;
                    double sa[NA];
#pragma unroll
                    for (int m = 0; m < NA; ++m) sa[m] = Fp[(long long)(ia0 + m) * ld];
                    to_cart<LA>(A.c2s, sa, fa);
#pragma unroll
                    for (int w = 0; w < NW; ++w)
#pragma unroll
                        for (int i = 0; i < NCA; ++i) ya[w][i] = 0.0;
                }
                double sb[NB], fb[NCB];
#pragma unroll
                for (int m = 0; m < NB; ++m) sb[m] = Fp[(long long)(ib0 + m) * ld];
                to_cart<LB>(A.c2s, sb, fb);
                double ab[NW][NCA * NCB];
#pragma unroll
                for (int w = 0; w < NW; ++w)
#pragma unroll
                    for (int i = 0; i < NCA * NCB; ++i) ab[w][i] = 0.0;
                for (int q = pp0; q < pp0 + npp; ++q) {
                    const double* __restrict__ rec = A.rec + (long long)q * kF64Rec;
                    const double X = rec[0] - gx, Y = rec[1] - gy, Z = rec[2] - gz;
                    const double rr = fma(X, X, fma(Y, Y, Z * Z));
#pragma unroll
                    for (int w = 0; w < NW; ++w) {
                        const double* __restrict__ rw =
                            w ? A.rec2 + (long long)q * kF64Rec : rec;
                        double r0[L + 1];
                        boys_fast<L>(rw[3] * rr, stab, r0);
                        if constexpr (L == 0) {
                            ab[w][0] = fma(rw[4], r0[0], ab[w][0]);
                        } else {
#pragma unroll
                            for (int n = 0; n <= L; ++n) r0[n] *= rw[4 + n];
                            double R[nr_c(L)];
                            fill_r64<L>(r0, X, Y, Z, R);
                            hermite_block<LA, LB>(
                                Ecls + (long long)(q - pp_begin) * 3 * NAX, R, ab[w]);
                        }
                    }
                }
#pragma unroll
                for (int w = 0; w < NW; ++w) {
                    if (diag) {
                        if constexpr (LA == LB) {
#pragma unroll
                            for (int a = 0; a < NCA; ++a)
#pragma unroll
                                for (int b = 0; b < NCB; ++b)
                                    ya[w][a] = fma(0.5 * (ab[w][a * NCB + b] + ab[w][b * NCB + a]),
                                                   fb[b], ya[w][a]);
                        }
                    } else {
                        double yb[NCB];
#pragma unroll
                        for (int b = 0; b < NCB; ++b) yb[b] = ab[w][b] * fa[0];
#pragma unroll
                        for (int a = 0; a < NCA; ++a)
#pragma unroll
                            for (int b = 0; b < NCB; ++b) {
                                ya[w][a] = fma(ab[w][a * NCB + b], fb[b], ya[w][a]);
                                if (a) yb[b] = fma(ab[w][a * NCB + b], fa[a], yb[b]);
                            }
                        if (ok) {
#pragma unroll
                            for (int m = 0; m < NB; ++m)
                                atomicAdd(Gp[w] + (long long)(ib0 + m) * ld,
                                          to_sph<LB>(A.c2s, yb, m));
                        }
                    }
                }
            }
        }
        flush();
        if (lane == 0) item = nwarps + atomicAdd(A.work + cls, 1);
        item = __shfl_sync(0xffffffffu, item, 0);
    }
    for (int o = 16; o > 0; o >>= 1) {
        flops += __shfl_xor_sync(0xffffffffu, flops, o);
        ints += __shfl_xor_sync(0xffffffffu, ints, o);
    }
    if (lane == 0 && kept) {
        atomicAdd(A.counters + 3 * cls + 0, kept);
        atomicAdd(A.counters + 3 * cls + 1, flops);
        atomicAdd(A.counters + 3 * cls + 2, ints);
    }
}

template<int LA, int LB, int NW = 1>
cudaError_t run64(const CosxF64Args& a, int cls, int pb, int pe, int nsm,
                  cudaStream_t s) {
    auto k = cosx_fp64_kernel<LA, LB, NW>;
    constexpr int smem = BoysTable<LA + LB>::kBytes;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         smem);
    if (e != cudaSuccess) return e;
    const int grid = std::max(1, std::min(nsm, a.nblk * a.nseg));
    k<<<grid, F64Cta<LA, LB, NW>::kThreads, smem, s>>>(a, cls, pb, pe);
    return cudaGetLastError();
}

}  // namespace f64
}  // namespace wb
