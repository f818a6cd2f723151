// dgemm.cuh -- grouped FP64 contraction of many small problems (dgemm.cu).
#pragma once
#include <cuda_runtime.h>
#include <vector>

#include "common.cuh"
#include "tc_gemm.cuh"

namespace tdscha {

// Rows 16-byte aligned (even leading dimensions and k offsets), K a multiple of 16.
bool dgemm_fits(const double *A, long long lda, const double *B, long long ldb, const std::vector<tc::GemmGroup> &gs);

// Scratch of the split contractions: the partial tiles of at most eight CTAs per SM (39 MB, any contents), and arrival
// counters (zero before the first launch, left at zero by every launch).  Both serve launches that follow one another on a stream.
constexpr int DGEMM_MAX_CTAS = 8 * 148;   // of a launch with split contractions
constexpr size_t DGEMM_COUNT_BYTES = DGEMM_MAX_CTAS * sizeof(unsigned);
size_t dgemm_part_bytes();

// C[d_off + m * ldc + n] (+)= sum_k A[a_row + m, a_k + k] B[b_row + n, b_k + k] for every group, one launch per 64
// groups.  part, count: scratch as above.
int dgemm_grouped(const double *A, long long lda, const double *B, long long ldb, const std::vector<tc::GemmGroup> &gs, double *C,
                  long long ldc, bool accumulate, double *part, unsigned *count, cudaStream_t st);

}  // namespace tdscha
