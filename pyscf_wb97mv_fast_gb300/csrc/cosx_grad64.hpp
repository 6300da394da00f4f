// Integral-derivative part of the COSX exchange gradient (cosx_grad64.cu):
// argument block and launchers.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace wb {

struct CosxGradArgs {
    const double* F;            // (nao, ld) AO-major, FP64: F = X D
    const double* coords;       // (npts, 3) molecule frame
    long long ld;
    int npts;
    // the screen of the FP64 kernels (32-point blocks)
    const int4* khdr;
    const int2* pshell;
    const float2* ptau;
    const float4* bnd;
    const float* bpref;
    const float4* blk_cr;
    const float* blk_msh;
    int nblk;
    int nvshell;
    float tol;
    int pp_begin[10];
    // FP64 pair data: the records of this omega (f64_records), the Hermite
    // coefficients and their d/dQ, per class from e_base[c]; per virtual shell
    // its atom
    const double* rec;
    const double* E;
    const double* dE;
    long long e_base[10];
    const int* vs_atom;
    const double* boys;         // the tables of fp64_boys.cuh
    const double* c2s;          // l = 2 at 0, l = 3 at 30
    double* gpt;                // nseg x (3 natm, ld) sums of each point, zeroed
    long long gstride;          // 3 natm ld
    int nseg;                   // ranges of a class's pairs (f64_segments)
    int* work;                  // per class block counter (zeroed)
};

// the d/dQ of the Hermite coefficients of every primitive pair (layout of E)
struct GradEArgs {
    int npairs;
    const int* pclass;
    const int4* hdr;            // per pair: ia0, ib0, pp0, npp | diag << 16
    const int2* pshell;
    const double* p;
    const double* alpha;
    const double* vs_xyz;       // per virtual shell its centre (3)
    long long e_base[10];
    int pp_begin[10];
    double* dE;
    double* rec;                // the records: -2 mu Q is added to each
};
cudaError_t launch_grad_e(const GradEArgs& a, cudaStream_t s);

cudaError_t launch_cosx_grad64_class(int cls, const CosxGradArgs& a, int pb, int pe,
                                     int nsm, cudaStream_t s);
// out (natm * 3) -= 1/2 sum_g w_g gpt (fixed-order block reductions)
cudaError_t launch_grad_points_sum(const double* gpt, const double* w, int64_t npts,
                                   int64_t ld, int natm, int nseg, double* out,
                                   cudaStream_t s);
// out (nao, 3): sum_g w_g dX[x][mu][g] H[mu][g] (fixed-order block reduction)
cudaError_t launch_ao_dot(const double* dX, const double* H, const double* w,
                          int64_t npts, int64_t ld, int nao, double* out,
                          cudaStream_t s);
// grad (natm, 3) += scale * sum over the AOs of each atom of aodot (virtual
// shells in order)
cudaError_t launch_atom_sum(const double* aodot, const int* vs_ao0, const int* vs_nf,
                            const int* vs_atom, int nvshell, int natm, double scale,
                            double* grad, cudaStream_t s);

}  // namespace wb
