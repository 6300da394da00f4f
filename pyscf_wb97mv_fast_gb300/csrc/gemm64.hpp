// FP64 GEMMs on the bf16 tensor cores at FP64 accuracy (gemm64.cu).
#pragma once
#include <cublas_v2.h>
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace wb {

// bytes of either product for nao rows and ld columns
size_t gemm64_bytes(int nao, int64_t ld);

// F (nao, ld) FP64 = X QD in the AO-major layout: F[mu][g] = sum_l X[l][g]
// QD[l][mu]; X (nao, ld), QD (nao, nao) row-major, ld a multiple of 32.
// Returns 0, a cudaError_t, or 1000 + cuBLAS status.
int gemm64_f(cublasHandle_t hb, const double* X, const double* QD, int nao, int64_t ld,
             double* F, void* ws, cudaStream_t s);

// K (nao, nao) row-major (+)= sum_{g < npts} w_g X[mu][g] G[nu][g]
int gemm64_k(cublasHandle_t hb, const double* X, const double* G, const double* w, int nao,
             int64_t ld, int64_t npts, int accumulate, double* K, void* ws, cudaStream_t s);

// kernel launches of one product, the GEMMs among them
int gemm64_f_launches(int nao, int64_t ld);
int gemm64_k_launches(int nao, int64_t npts);

}  // namespace wb
