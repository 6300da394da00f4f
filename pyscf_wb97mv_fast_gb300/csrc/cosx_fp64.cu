// Plain FP64 form of the fused screen + G kernels: the s/p/d classes, the
// class dispatcher and the per-omega records (the kernel itself is in
// cosx_fp64.cuh).
#include "cosx_fp64.cuh"
#include "launch.hpp"

namespace wb {

cudaError_t launch_cosx_fp64_class(int cls, const CosxF64Args& a, int pb, int pe,
                                   int nsm, cudaStream_t s) {
    switch (cls) {
    case 0: return f64::run64<0, 0>(a, cls, pb, pe, nsm, s);
    case 1: return f64::run64<1, 0>(a, cls, pb, pe, nsm, s);
    case 2: return f64::run64<1, 1>(a, cls, pb, pe, nsm, s);
    case 3: return f64::run64<2, 0>(a, cls, pb, pe, nsm, s);
    case 4: return f64::run64<2, 1>(a, cls, pb, pe, nsm, s);
    case 5: return f64::run64<2, 2>(a, cls, pb, pe, nsm, s);
    default: return launch_cosx_fp64_f(cls, a, pb, pe, nsm, s);
    }
}

cudaError_t launch_cosx_fp64_dual(int cls, const CosxF64Args& a, int pb, int pe, int nsm,
                                  cudaStream_t s) {
    switch (cls) {
    case 0: return f64::run64<0, 0, 2>(a, cls, pb, pe, nsm, s);
    case 1: return f64::run64<1, 0, 2>(a, cls, pb, pe, nsm, s);
    case 2: return f64::run64<1, 1, 2>(a, cls, pb, pe, nsm, s);
    case 3: return f64::run64<2, 0, 2>(a, cls, pb, pe, nsm, s);
    default: return cudaErrorInvalidValue;
    }
}

namespace {

// the lane-independent factors of a primitive pair, once per omega: in the
// class kernels the division and the square root would take 30 FP64
// instructions of every (primitive pair, point)
__global__ void f64_records_kernel(const int npp, const double* __restrict__ P,
                                   const double* __restrict__ p,
                                   const double* __restrict__ pref,
                                   const double* __restrict__ alpha, const double om2,
                                   double* __restrict__ rec) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= npp) return;
    double* r = rec + (int64_t)q * kF64Rec;
    const double pq = p[q];
    double th = 1.0, sth = 1.0;
    if (om2 > 0.0) {
        th = om2 / (om2 + pq);
        sth = sqrt(th);
    }
    const double pth = pq * th;
    r[0] = P[3 * (int64_t)q];
    r[1] = P[3 * (int64_t)q + 1];
    r[2] = P[3 * (int64_t)q + 2];
    r[3] = pth;
    double c = pref[q] * sth;
    for (int n = 0; n < 8; ++n) {
        r[4 + n] = c;
        c *= -2.0 * pth;
    }
    r[12] = alpha[q] / pq;
}

__global__ void f64_segment_sum_kernel(double* __restrict__ G, const int64_t n,
                                       const int nseg) {
    for (int64_t i = 2 * (blockIdx.x * (int64_t)blockDim.x + threadIdx.x); i < n;
         i += 2 * (int64_t)gridDim.x * blockDim.x) {
        double2 a = *reinterpret_cast<const double2*>(G + i);
        for (int s = 1; s < nseg; ++s) {
            const double2 b = *reinterpret_cast<const double2*>(G + s * n + i);
            a.x += b.x;
            a.y += b.y;
        }
        *reinterpret_cast<double2*>(G + i) = a;
    }
}
}  // namespace

cudaError_t launch_f64_segment_sum(double* G, int64_t n, int nseg, cudaStream_t s) {
    if (nseg < 2 || n <= 0) return cudaSuccess;      // n is a multiple of 32
    f64_segment_sum_kernel<<<(unsigned)grid_stride_blocks((n + 1) / 2, 256, 8), 256, 0, s>>>(
        G, n, nseg);
    return cudaGetLastError();
}

cudaError_t launch_f64_records(int npp, const double* P, const double* p,
                               const double* pref, const double* alpha, double omega,
                               double* rec, cudaStream_t s) {
    if (npp <= 0) return cudaSuccess;
    f64_records_kernel<<<(npp + 127) / 128, 128, 0, s>>>(npp, P, p, pref, alpha,
                                                         omega * omega, rec);
    return cudaGetLastError();
}

}  // namespace wb
