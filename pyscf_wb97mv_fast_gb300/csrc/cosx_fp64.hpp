// Plain FP64 form of the fused screen + G kernels (cosx_fp64.cu): argument
// block and launchers.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace wb {

constexpr int kBoys64Nodes = 145;   // T_k = k / 4, k = 0..144
constexpr int kBoys64Cols = 20;     // F_m(T_k), m = 0..19 (L <= 6 + 11 Taylor terms)
constexpr int kBoysTaylor = 12;     // terms of the 1/4-node series

constexpr int kBoysFineNodes = 1153;    // T_k = k / 32, k = 0..1152
constexpr int kBoysFineCols = 14;       // F_m(T_k), m = 0..13 (orders to 7)
// doubles of a primitive pair's record: P (3), p theta, then c_n = prefactor
// sqrt(theta) (-2 p theta)^n (n <= 7), the bra exponent over p and, in the
// gradient, -2 mu Q (3)
constexpr int kF64Rec = 16;

struct CosxF64Args {
    const double* F;            // (nao, ld) AO-major, FP64
    double* G;                  // nseg x (nao, ld) AO-major, FP64, accumulated
    double* G2;                 // the second omega's, with two (launch_cosx_fp64_dual)
    long long gstride;          // nao ld
    int nseg;                   // ranges of a class's pairs (f64_segments)
    const double* coords;       // (npts, 3) molecule frame
    long long ld;
    int npts;
    // screening inputs of the FP32 path (32-point blocks)
    const int4* khdr;
    const int2* pshell;
    const float2* ptau;
    const float4* bnd;
    const float* bpref;
    const float4* blk_cr;
    const float* blk_msh;
    int nblk;
    int nvshell;
    float tol;                  // tile_tol / 1.001, <= 0 keeps every task
    int pp_begin[10];           // first primitive pair of each class
    // FP64 pair data: per primitive pair the record of this omega
    // (f64_records); per class the Hermite E block from e_base[c]
    const double* rec;
    const double* rec2;         // the second omega's
    const double* E;
    long long e_base[10];
    const double* boys;         // the tables of fp64_boys.cuh
    const double* c2s;          // l = 2 (6 x 5) at 0, l = 3 (10 x 7) at 30, row-major
    const long long* pflops;
    const int* pnint;
    unsigned long long* counters;   // per class: kept, flops, ints
    int* work;                      // per class block counter (zeroed)
};

// rec (npp, kF64Rec) of one omega from P, p, the folded prefactor and the bra
// exponent of every primitive pair
cudaError_t launch_f64_records(int npp, const double* P, const double* p,
                               const double* pref, const double* alpha, double omega,
                               double* rec, cudaStream_t s);
// Ranges that the pairs of a block are split into: some six items for each of
// an SM's 16 warps, so that neither a short grid nor the last items of a class
// leave warps without work.  FP64 K of 8 waters (192 AOs, 70,478 points) 2
// ranges 51.8 ms, 4 48.0, 7 46.7; gradient of 8 waters (36,369 points) 4 ranges
// 58.1 ms, 13 53.6, of C4H10 in TZVP (21,512) 6 73.8, 22 70.3.
inline int f64_segments(int64_t nblk, int nsm) {
    const int64_t n = (96 * (int64_t)nsm + nblk - 1) / (nblk > 0 ? nblk : 1);
    return (int)(n < 1 ? 1 : n > 32 ? 32 : n);
}
// G[0] += the other nseg - 1 ranges, in order; n elements each
cudaError_t launch_f64_segment_sum(double* G, int64_t n, int nseg, cudaStream_t s);
// one class launch for two omegas (classes with fp64_dual)
inline bool fp64_dual(int cls) { return cls <= 3; }        // la + lb <= 2
cudaError_t launch_cosx_fp64_dual(int cls, const CosxF64Args& a, int pb, int pe, int nsm,
                                  cudaStream_t s);
// one class launch (classes 0..9); the f classes live in cosx_fp64_f.cu
cudaError_t launch_cosx_fp64_class(int cls, const CosxF64Args& a, int pb, int pe,
                                   int nsm, cudaStream_t s);
cudaError_t launch_cosx_fp64_f(int cls, const CosxF64Args& a, int pb, int pe,
                               int nsm, cudaStream_t s);

}  // namespace wb
