// Integral-derivative part of the COSX exchange nuclear gradient (grid
// response off), in FP64:
//
//   E_w = -1/4 sum_g w_g sum_{nu,lam} F_g,nu A^g_nu,lam(w) F_g,lam,
//   F = X D.
//
// Moving a nucleus moves its basis functions.  The part of dE/dR that
// differentiates A is
//
//   -1/2 sum_g w_g sum_{nu on C} sum_lam F_g,nu F_g,lam d(nu lam|g)/dR_nu.
//
// It is collected per unordered shell pair (A, B): the bra derivative goes
// to atom(A) and the ket derivative to atom(B); a diagonal pair (B = A)
// contributes its bra derivative only.  For a primitive pair,
//   d/dA_x (a b|g) = 2 alpha (a + 1_x, b|g) - a_x (a - 1_x, b|g),
// and the ket derivative follows from translational invariance,
//   d/dB = -d/dA - d/dC, with d/dC_x R_tuv(P - C) = -R_t+1,u,v.
// The X side of the gradient (d F / dR through the AO values) is formed
// from G and the AO gradients by the host (cosx.CosxEngine.k_grad).
//
// With P = (alpha A + beta B) / p and Q = A - B, d/dA = (alpha / p) d/dP +
// d/dQ and d/dB = (beta / p) d/dP - d/dQ; d/dP_x raises the Hermite index,
// R_tuv -> R_t+1,u,v, and d/dQ acts on the Hermite coefficients (tables formed
// once per call, grad_e_kernel) and on the prefactor exp(-mu Q^2).  So one pass
// over the primitive pair gives both centres:
//   S_x = sum_ab f_a f_b sum E^x_t E^y_u E^z_v R_t+1,u,v
//   e   = sum_ab f_a f_b sum E^x_t E^y_u E^z_v R_tuv
//   D_x = sum_ab f_a f_b sum (dE^x_t / dQ_x) E^y_u E^z_v R_tuv - 2 mu Q_x e
//   dA = (alpha / p) S + D,  dB = S - dA
// (dE^{ij}_t / dQ is zero for t >= i + j, so the three sums of D are short.)
// (differentiating the Gaussians themselves needs integrals of l + 1 and
// l - 1 for each of the three axes and each component).
//
// The screen, pair tables, Boys function and McMurchie-Davidson recurrence
// are those of the plain FP64 kernels (cosx_fp64.cuh), and so is the bound:
// the FP64 pipe.  One warp owns one 32-point block, one point a lane.  A
// lane adds its point's sums to its own column of its range's gpt (3 natm, ld) by
// reductions in the L2, dA once per run of pairs with one bra shell; a lane
// reduction in the task would cost 30 FP64 instructions.  The columns are
// weighted with -w_g / 2 and summed in a fixed order at the end, so the
// result is bitwise reproducible.  Measured (whole call): 8 waters, 36,369
// points 370 -> 54 ms; C4H10 in TZVP, 21,512 points 692 -> 70 ms.
#include "cosx_fp64.cuh"
#include "cosx_grad64.hpp"

namespace wb {
namespace {

using namespace f64;

// d/dQ of every Hermite coefficient, in the layout of E, and -2 mu Q into the
// records.  One thread per (shell pair, axis); E by its recurrence and its
// derivative along.
__global__ void grad_e_kernel(const GradEArgs A) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= A.npairs) return;
    const int x = blockIdx.y;
    const int cls = A.pclass[k];
    int la = 0;
    while ((la + 1) * (la + 2) / 2 <= cls) ++la;
    const int lb = cls - la * (la + 1) / 2;
    const int nax = eoff(lb, la + 1, 0);
    const int4 h = A.hdr[k];
    const int2 sh = A.pshell[k];
    const double Q = A.vs_xyz[3 * sh.x + x] - A.vs_xyz[3 * sh.y + x];
    double E[4][4][8], D[4][4][8];
    for (int q = h.z; q < h.z + (h.w & 0xffff); ++q) {
        const double p = A.p[q], al = A.alpha[q], be = p - al;
        const double hp = 0.5 / p, ka = -be / p, kb = al / p;
        A.rec[(int64_t)q * kF64Rec + 13 + x] = -2.0 * al * be / p * Q;
        for (int i = 0; i <= la; ++i)
            for (int j = 0; j <= lb; ++j)
                for (int t = 0; t <= i + j; ++t) {
                    if (i + j == 0) {
                        E[0][0][0] = 1.0;
                        D[0][0][0] = 0.0;
                        continue;
                    }
                    const double c = i ? ka : kb;
                    const int ii = i ? i - 1 : i, jj = i ? j : j - 1, n = ii + jj;
                    double e = 0.0, d = 0.0;
                    if (t <= n) {
                        e = c * Q * E[ii][jj][t];
                        d = c * (Q * D[ii][jj][t] + E[ii][jj][t]);
                    }
                    if (t > 0) {
                        e += hp * E[ii][jj][t - 1];
                        d += hp * D[ii][jj][t - 1];
                    }
                    if (t + 1 <= n) {
                        e += (t + 1) * E[ii][jj][t + 1];
                        d += (t + 1) * D[ii][jj][t + 1];
                    }
                    E[i][j][t] = e;
                    D[i][j][t] = d;
                }
        double* out = A.dE + A.e_base[cls] + ((int64_t)(q - A.pp_begin[cls]) * 3 + x) * nax;
        int n = 0;
        for (int i = 0; i <= la; ++i)
            for (int j = 0; j <= lb; ++j)
                for (int t = 0; t <= i + j; ++t)
                    out[n++] = D[i][j][t];
    }
}

// S (assigned) and D (added) of one primitive pair, for f_a f_b over the
// Cartesian components; m2 = -2 mu Q; R packed for order L + 1.  Per (i, i'): R
// contracted with E^x, dE^x and E^x at t + 1; f_a f_b spread over (u, v) with
// E^y E^z and their derivatives; then the two sides meet.
template<int LA, int LB>
__device__ __forceinline__ void grad_block(const double* __restrict__ E,
                                           const double* __restrict__ dE,
                                           const double* __restrict__ m2,
                                           const double* R, const double* fa,
                                           const double* fb, double* S, double* D) {
    constexpr int L = LA + LB, NAX = eaxis(LA, LB);
    constexpr int NUV = (L + 1) * (L + 2) / 2, NUV1 = (L + 2) * (L + 3) / 2;
    double en = 0.0;
    S[0] = S[1] = S[2] = 0.0;
#pragma unroll
    for (int i = 0; i <= LA; ++i)
#pragma unroll
        for (int ip = 0; ip <= LB; ++ip) {
            const int M = L - i - ip;
            const double* ex = E + eoff(LB, i, ip);
            const double* dx = dE + eoff(LB, i, ip);
            double h[NUV], hy[NUV], hz[NUV];
            bool seth[NUV], sethy[NUV], sethz[NUV];
#pragma unroll
            for (int n = 0; n < NUV; ++n) seth[n] = sethy[n] = sethz[n] = false;
#pragma unroll
            for (int j = 0; j <= LA; ++j)
#pragma unroll
                for (int jp = 0; jp <= LB; ++jp)
                    if (j <= LA - i && jp <= LB - ip) {
                        const int k = LA - i - j, kp = LB - ip - jp;
                        const double* ey = E + NAX + eoff(LB, j, jp);
                        const double* dy = dE + NAX + eoff(LB, j, jp);
                        const double* ez = E + 2 * NAX + eoff(LB, k, kp);
                        const double* dz = dE + 2 * NAX + eoff(LB, k, kp);
                        const double f = fa[cidx(LA, i, j)] * fb[cidx(LB, ip, jp)];
#pragma unroll
                        for (int v = 0; v <= L; ++v)
                            if (v <= k + kp) {
                                const double zv = k + kp == 0 ? f : ez[v] * f;
                                const double zd = v < k + kp ? dz[v] * f : 0.0;
#pragma unroll
                                for (int u = 0; u <= L; ++u)
                                    if (u <= j + jp) {
                                        const int n = u * (2 * M + 3 - u) / 2 + v;
                                        if (j + jp == 0)
                                            h[n] = seth[n] ? h[n] + zv : zv;
                                        else
                                            h[n] = seth[n] ? fma(ey[u], zv, h[n]) : ey[u] * zv;
                                        seth[n] = true;
                                        if (v < k + kp) {
                                            if (j + jp == 0)
                                                hz[n] = sethz[n] ? hz[n] + zd : zd;
                                            else
                                                hz[n] = sethz[n] ? fma(ey[u], zd, hz[n])
                                                                 : ey[u] * zd;
                                            sethz[n] = true;
                                        }
                                        if (u < j + jp) {
                                            hy[n] = sethy[n] ? fma(dy[u], zv, hy[n])
                                                             : dy[u] * zv;
                                            sethy[n] = true;
                                        }
                                    }
                            }
                    }
            double rx[NUV1];
#pragma unroll
            for (int u = 0; u <= L + 1; ++u)
#pragma unroll
                for (int v = 0; v <= L + 1; ++v)
                    if (u + v <= M + 1) {
                        double s = R[ridx(L + 1, 0, u, v)];
                        if (i + ip > 0) {
                            s *= ex[0];
#pragma unroll
                            for (int t = 1; t <= L; ++t)
                                if (t <= i + ip) s = fma(ex[t], R[ridx(L + 1, t, u, v)], s);
                        }
                        rx[u * (2 * M + 5 - u) / 2 + v] = s;
                    }
#pragma unroll
            for (int u = 0; u <= L; ++u)
#pragma unroll
                for (int v = 0; v <= L; ++v)
                    if (u + v <= M) {
                        const int n = u * (2 * M + 3 - u) / 2 + v;
                        double rp = R[ridx(L + 1, 1, u, v)];
                        if (i + ip > 0) {
                            double rd = dx[0] * R[ridx(L + 1, 0, u, v)];
                            rp *= ex[0];
#pragma unroll
                            for (int t = 1; t <= L; ++t)
                                if (t <= i + ip) {
                                    if (t < i + ip) rd = fma(dx[t], R[ridx(L + 1, t, u, v)], rd);
                                    rp = fma(ex[t], R[ridx(L + 1, t + 1, u, v)], rp);
                                }
                            D[0] = fma(rd, h[n], D[0]);
                        }
                        const double r = rx[u * (2 * M + 5 - u) / 2 + v];
                        S[0] = fma(rp, h[n], S[0]);
                        S[1] = fma(rx[(u + 1) * (2 * M + 4 - u) / 2 + v], h[n], S[1]);
                        S[2] = fma(rx[u * (2 * M + 5 - u) / 2 + v + 1], h[n], S[2]);
                        en = fma(r, h[n], en);
                        if (sethy[n]) D[1] = fma(r, hy[n], D[1]);
                        if (sethz[n]) D[2] = fma(r, hz[n], D[2]);
                    }
        }
#pragma unroll
    for (int x = 0; x < 3; ++x) D[x] = fma(m2[x], en, D[x]);
}

// threads of a CTA (one an SM), as for the FP64 class kernels
template<int LA, int LB>
struct GradCta { static constexpr int kThreads = LA + LB <= 1 ? 512 : 256; };

template<int LA, int LB>
__global__ void __launch_bounds__(GradCta<LA, LB>::kThreads, 1)
cosx_grad64_kernel(const CosxGradArgs A, const int cls, const int pair_begin,
                   const int pair_end) {
    constexpr int L = LA + LB;
    constexpr int NCA = ncart_c(LA), NCB = ncart_c(LB);
    constexpr int NA = 2 * LA + 1, NB = 2 * LB + 1;
    constexpr int NAX = eaxis(LA, LB);
    extern __shared__ double stab[];
    load_boys<L + 1>(A.boys, stab);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const long long ld = A.ld;
    const int pp_begin = A.pp_begin[cls];
    const float4* __restrict__ bnd = A.bnd + pp_begin;
    const float* __restrict__ bpref = A.bpref + pp_begin;
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
        double* __restrict__ out = A.gpt + seg * A.gstride + g;
        const float4 cr = A.blk_cr[blk];
        const float* __restrict__ ms = A.blk_msh + (long long)blk * A.nvshell;
        int run = -1;                       // bra virtual shell held
        double fa[NCA], ga[3] = {0.0, 0.0, 0.0};
        auto flush = [&]() {
            if (run < 0 || !ok) return;
            const int at = A.vs_atom[run];
#pragma unroll
            for (int x = 0; x < 3; ++x) atomicAdd(out + (3 * at + x) * ld, ga[x]);
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
            while (mask) {
                const int kk = c0 + __ffs(mask) - 1;
                mask &= mask - 1;
                const int4 hdr = A.khdr[kk];
                const int2 sh = A.pshell[kk];
                const int ia0 = hdr.x & 0xffff, ib0 = hdr.y & 0xffff;
                const int pp0 = pp_begin + hdr.z, npp = hdr.w & 0xffff;
                const bool diag = (hdr.w >> 16) != 0;
                if (sh.x != run) {
                    flush();
                    run = sh.x;
                    double sa[NA];
#pragma unroll
                    for (int m = 0; m < NA; ++m) sa[m] = Fp[(long long)(ia0 + m) * ld];
                    to_cart<LA>(A.c2s, sa, fa);
                    ga[0] = ga[1] = ga[2] = 0.0;
                }
                double sb[NB], fb[NCB];
#pragma unroll
                for (int m = 0; m < NB; ++m) sb[m] = Fp[(long long)(ib0 + m) * ld];
                to_cart<LB>(A.c2s, sb, fb);
                double dA[3] = {0.0, 0.0, 0.0}, tot[3] = {0.0, 0.0, 0.0};
                for (int q = pp0; q < pp0 + npp; ++q) {
                    const double* __restrict__ rec = A.rec + (long long)q * kF64Rec;
                    const double X = rec[0] - gx, Y = rec[1] - gy, Z = rec[2] - gz;
                    const double T = rec[3] * fma(X, X, fma(Y, Y, Z * Z));
                    double r0[L + 2], R[nr_c(L + 1)], S[3];
                    boys_fast<L + 1>(T, stab, r0);
#pragma unroll
                    for (int n = 0; n <= L + 1; ++n) r0[n] *= rec[4 + n];
                    fill_r64<L + 1>(r0, X, Y, Z, R);
                    const long long e = A.e_base[cls] + (long long)(q - pp_begin) * 3 * NAX;
                    grad_block<LA, LB>(A.E + e, A.dE + e, rec + 13, R, fa, fb, S, dA);
#pragma unroll
                    for (int x = 0; x < 3; ++x) {
                        dA[x] = fma(rec[12], S[x], dA[x]);
                        tot[x] += S[x];
                    }
                }
#pragma unroll
                for (int x = 0; x < 3; ++x) ga[x] += dA[x];
                // a diagonal pair contributes its bra derivative only
                if (!diag && ok) {
                    const int at = A.vs_atom[sh.y];
#pragma unroll
                    for (int x = 0; x < 3; ++x)
                        atomicAdd(out + (3 * at + x) * ld, tot[x] - dA[x]);
                }
            }
        }
        flush();
        if (lane == 0) item = nwarps + atomicAdd(A.work + cls, 1);
        item = __shfl_sync(0xffffffffu, item, 0);
    }
}

template<int LA, int LB>
cudaError_t run_grad(const CosxGradArgs& a, int cls, int pb, int pe, int nsm,
                     cudaStream_t s) {
    auto k = cosx_grad64_kernel<LA, LB>;
    constexpr int smem = BoysTable<LA + LB + 1>::kBytes;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         smem);
    if (e != cudaSuccess) return e;
    const int grid = std::max(1, std::min(nsm, a.nblk * a.nseg));
    k<<<grid, GradCta<LA, LB>::kThreads, smem, s>>>(a, cls, pb, pe);
    return cudaGetLastError();
}

// out[r] += -1/2 sum_g w_g gpt[r][g] over the ranges: one CTA a row, fixed order
__global__ void grad_points_sum_kernel(const double* __restrict__ gpt,
                                       const double* __restrict__ w, int64_t npts,
                                       int64_t ld, int nseg, int64_t gstride,
                                       double* __restrict__ out) {
    __shared__ double red[256];
    const double* row = gpt + (int64_t)blockIdx.x * ld;
    double s = 0.0;
    for (int q = 0; q < nseg; ++q, row += gstride)
        for (int64_t g = threadIdx.x; g < npts; g += 256) s = fma(w[g], row[g], s);
    red[threadIdx.x] = s;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[blockIdx.x] -= 0.5 * red[0];
}

}  // namespace

cudaError_t launch_grad_e(const GradEArgs& a, cudaStream_t s) {
    if (a.npairs <= 0) return cudaSuccess;
    grad_e_kernel<<<dim3((a.npairs + 63) / 64, 3), 64, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_cosx_grad64_class(int cls, const CosxGradArgs& a, int pb, int pe,
                                     int nsm, cudaStream_t s) {
    switch (cls) {
    case 0: return run_grad<0, 0>(a, cls, pb, pe, nsm, s);
    case 1: return run_grad<1, 0>(a, cls, pb, pe, nsm, s);
    case 2: return run_grad<1, 1>(a, cls, pb, pe, nsm, s);
    case 3: return run_grad<2, 0>(a, cls, pb, pe, nsm, s);
    case 4: return run_grad<2, 1>(a, cls, pb, pe, nsm, s);
    case 5: return run_grad<2, 2>(a, cls, pb, pe, nsm, s);
    case 6: return run_grad<3, 0>(a, cls, pb, pe, nsm, s);
    case 7: return run_grad<3, 1>(a, cls, pb, pe, nsm, s);
    case 8: return run_grad<3, 2>(a, cls, pb, pe, nsm, s);
    case 9: return run_grad<3, 3>(a, cls, pb, pe, nsm, s);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_grad_points_sum(const double* gpt, const double* w, int64_t npts,
                                   int64_t ld, int natm, int nseg, double* out,
                                   cudaStream_t s) {
    if (natm <= 0) return cudaSuccess;
    grad_points_sum_kernel<<<3 * natm, 256, 0, s>>>(gpt, w, npts, ld, nseg,
                                                    3 * (int64_t)natm * ld, out);
    return cudaGetLastError();
}

}  // namespace wb

namespace wb {
namespace {

__global__ void ao_dot_kernel(const double* __restrict__ dX, const double* __restrict__ H,
                              const double* __restrict__ w, int64_t npts, int64_t ld,
                              int nao, double* __restrict__ out) {
    __shared__ double red[3][256];
    const int mu = blockIdx.x;
    double s[3] = {0.0, 0.0, 0.0};
    const double* h = H + (int64_t)mu * ld;
    for (int64_t g = threadIdx.x; g < npts; g += blockDim.x) {
        const double wh = w[g] * h[g];
        for (int x = 0; x < 3; ++x)
            s[x] = fma(wh, dX[((int64_t)(1 + x) * nao + mu) * ld + g], s[x]);
    }
    for (int x = 0; x < 3; ++x) red[x][threadIdx.x] = s[x];
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o)
            for (int x = 0; x < 3; ++x) red[x][threadIdx.x] += red[x][threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int x = 0; x < 3; ++x) out[3 * mu + x] = red[x][0];
}

__global__ void atom_sum_kernel(const double* __restrict__ aodot,
                                const int* __restrict__ vs_ao0,
                                const int* __restrict__ vs_nf,
                                const int* __restrict__ vs_atom, int nvshell, int natm,
                                double scale, double* __restrict__ grad) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 3 * natm) return;
    const int at = i / 3, x = i % 3;
    double s = 0.0;
    for (int v = 0; v < nvshell; ++v)
        if (vs_atom[v] == at)
            for (int m = 0; m < vs_nf[v]; ++m) s += aodot[3 * (vs_ao0[v] + m) + x];
    grad[i] += scale * s;
}

}  // namespace

cudaError_t launch_ao_dot(const double* dX, const double* H, const double* w,
                          int64_t npts, int64_t ld, int nao, double* out,
                          cudaStream_t s) {
    ao_dot_kernel<<<nao, 256, 0, s>>>(dX, H, w, npts, ld, nao, out);
    return cudaGetLastError();
}

cudaError_t launch_atom_sum(const double* aodot, const int* vs_ao0, const int* vs_nf,
                            const int* vs_atom, int nvshell, int natm, double scale,
                            double* grad, cudaStream_t s) {
    const int n = 3 * natm;
    atom_sum_kernel<<<(n + 127) / 128, 128, 0, s>>>(aodot, vs_ao0, vs_nf, vs_atom,
                                                    nvshell, natm, scale, grad);
    return cudaGetLastError();
}

}  // namespace wb
