// FP64-accurate GEMMs on bf16 tensor cores (Ozaki split), see ozaki.cu.
#pragma once
#include <cublas_v2.h>
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace wb {

constexpr int kOzWidth = 42;        // bits per operand: 7 digits of 6 or 6 of 7
constexpr int kOzKc = 2048;         // points of a K-GEMM chunk
constexpr int kOzKcSmall = 512;     // where 2048-point chunks would leave SMs idle

// The digits of the F product: 6 of 7 bits (21 slice products) where a level's
// (l + 1) nao terms of up to 2^12 stay within 2^24, exact in FP32, else 7 of 6
// bits (28), which holds to 7 nao < 2^14.  Both engines take the same, so their
// F agree bitwise.
inline bool ozaki_f_seven_bit(int nao) { return 6 * ((nao + 7) / 8 * 8) <= (1 << 12); }
inline bool ozaki_f_supported(int nao) { return 7 * nao < (1 << 14); }

size_t ozaki_f_bytes(int nao, int64_t ld);
// workspace of the K split for nrhs right-hand sides (w o G of several
// omegas against the same X)
size_t ozaki_k_bytes(int nao, int64_t ld, int nrhs = 1);

// F (nao, ld) FP32 AO-major = fl32(X QD); X (nao, ld) FP64 AO-major, QD
// (nao, nao) row-major FP64.  Returns 0, a cudaError_t, or 1000 + cuBLAS
// status.  status (optional, device): bit 0 is set when a wait of the
// tensor-core kernel gave up (the affected F entries are NaN).
int ozaki_f_gemm(cublasHandle_t hb, const double* X, const double* QD,
                 int nao, int64_t ld, float* F, void* ws, cudaStream_t s,
                 unsigned long long* status = nullptr);

// the same product with FP64 output: the combined level sums (42 bits
// relative to the per-point / per-column maxima) rounded once to FP64
int ozaki_f_gemm64(cublasHandle_t hb, const double* X, const double* QD,
                   int nao, int64_t ld, double* F, void* ws, cudaStream_t s,
                   unsigned long long* status = nullptr);

// K (+)= X^T (w o G) with G FP64 (w o G formed in FP64 before the split)
int ozaki_k_gemm64(cublasHandle_t hb, const double* X, const double* G,
                   const double* w, int nao, int64_t ld, int64_t npts,
                   int accumulate, double* K, void* ws, cudaStream_t s);

// the two engines of the F product (bitwise the same F): cuBLAS level
// GEMMs and this library's tcgen05 kernel; kOzEngineAuto takes the kernel where
// ozaki_f_small, the GEMMs elsewhere
constexpr int kOzEngineLibrary = 0;
constexpr int kOzEngineTc = 1;
constexpr int kOzEngineAuto = 2;        // the default
void ozaki_set_f_engine(int engine);
int ozaki_get_f_engine();
// One column of tiles of the tensor-core kernel (64 AOs) in one wave of CTAs:
// the level GEMMs are then shorter than the gaps between them.  An F product
// as called: 48 AOs, 9,928 points 76 -> 42 us, 24 AOs, 5,012 points 78 -> 36;
// past it the level GEMMs win (96 AOs, 19,325 points 78 us against 83; 192 AOs,
// 36,475 points 178 against 257).
bool ozaki_f_small(int nao, int64_t ld);
bool ozaki_f_on_tc(int nao, int64_t ld);        // under the current engine
// kernel launches of one F product under the current engine
inline int ozaki_f_launches(int nao, int64_t ld) {
    return ozaki_f_on_tc(nao, ld) ? 4 : 4 + (ozaki_f_seven_bit(nao) ? 6 : 7);
}
// the same of one K product
int ozaki_k_launches(int nao, int64_t ld);
int ozaki_f_gemm_cublas(cublasHandle_t hb, const double* X, const double* QD,
                        int nao, int64_t ld, float* F, void* ws, cudaStream_t s);
int ozaki_f_gemm_tc(const double* X, const double* QD, int nao, int64_t ld, float* F,
                    void* ws, cudaStream_t s, unsigned long long* status);
int ozaki_f_gemm_cublas64(cublasHandle_t hb, const double* X, const double* QD,
                          int nao, int64_t ld, double* F, void* ws, cudaStream_t s);
int ozaki_f_gemm_tc64(const double* X, const double* QD, int nao, int64_t ld, double* F,
                      void* ws, cudaStream_t s, unsigned long long* status);
size_t ozaki_f_tc_bytes(int nao, int64_t ld);
// exponent of max_l |X(l, g)| per point g (shared by both engines)
void f_rowmax(const double* X, int nao, int64_t ld, int* erow, cudaStream_t s);

// K (nao, nao) row-major (+)= X^T (w o G) over the npts valid points.
// x_sliced: ws already holds the slices of this X (an earlier call on the
// same X and workspace, e.g. another omega of the same tile), which are
// reused.
int ozaki_k_gemm(cublasHandle_t hb, const double* X, const float* G,
                 const double* w, int nao, int64_t ld, int64_t npts,
                 int accumulate, double* K, void* ws, cudaStream_t s,
                 bool x_sliced = false);

// K_r (+)= X^T (w o G_r) for r < nrhs (<= 8) in one split: X sliced once,
// the w o G_r side by side (N = nrhs nao per level GEMM), one combine.
int ozaki_k_gemm_multi(cublasHandle_t hb, const double* X, const float* const* G,
                       int nrhs, const double* w, int nao, int64_t ld,
                       int64_t npts, int accumulate, double* const* K, void* ws,
                       cudaStream_t s, bool x_sliced = false);

}  // namespace wb
