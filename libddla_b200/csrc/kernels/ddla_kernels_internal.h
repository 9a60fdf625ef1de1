// Declarations shared between the kernel translation units (not part of the C ABI).
#pragma once
#include <cuda_runtime.h>
#include "common.cuh"

namespace ddlak {

// C(i,j) -= sum_{k0 <= c < k0+nbk} L(i,c) conj(L(j,c)) for the lower-triangle
// entries of the region rows [t0, n) x columns [t0, n) (cols == 0) or
// columns [t0, t0+cols) (cols > 0), in the L view of common.cuh.
template <class T, bool UP>
cudaError_t trailing_update(T* A, long long lda, int k0, int nbk, int n, long long t0, int cols, const int* dinfo,
                            cudaStream_t st);

// The diagonal block [k0, k0+nbk)^2 (nbk <= 128) of each matrix of a batch (astride
// elements and one info word apart), FP64 arithmetic for either storage (panel.cu).
template <class S, bool UP>
cudaError_t launch_potrf_diag(S* A, long long lda, long long astride, int batch, int k0, int nbk, int* dinfo,
                              cudaStream_t st);

// X * L11^T = A21 for the rows below that block (panel.cu).
template <class S, bool UP>
cudaError_t launch_trsm_panel_dmma(S* A, long long lda, long long astride, int batch, int k0, int nbk, int n,
                                   const int* dinfo, cudaStream_t st);

// The FP64 lower update of the region from row / column t0 (all of it, or its
// first cols columns when cols > 0) over a batch of equal-order matrices
// (astride elements apart, info per matrix), nbk a multiple of 32 (syrk.cu).
cudaError_t launch_syrk_batched(double* A, long long lda, long long astride, int batch, int k0, int nbk, int n,
                                long long t0, int cols, const int* dinfo, cudaStream_t st);

// The FP32 update of the region as trailing_update, nbk a multiple of 32 (sgemm.cu).
template <bool UP>
cudaError_t syrk_f32(float* A, long long lda, int k0, int nbk, int n, long long t0, int cols, const int* dinfo,
                     cudaStream_t st);

// W = L^-1 for one lower FP32 factor of any order; what W holds above its diagonal
// afterwards is unspecified; a wait that gives up leaves NaN in its tile and its code in *status
// (sgemm.cu).
cudaError_t trtri_large_f32(int n, const float* L, long long ldl, float* W, long long ldw, int* status, cudaStream_t st);

template <class T, bool UP>
cudaError_t trailing_update_simt(T* A, long long lda, int k0, int nbk, int n, long long t0, int cols,
                                 const int* dinfo, cudaStream_t st);

}  // namespace ddlak
