// tc_gemm.cuh -- interface of the tcgen05 contraction kernel (tc_gemm.cu).
#pragma once
#include <cuda_runtime.h>
#include <functional>
#include <vector>
#include "common.cuh"

namespace tdscha {
namespace tc {

// D (M x N, fp32) = A (M x K) . B (N x K)^T, both operands row-major with K contiguous.
// fmt FMT_BF16: bf16 elements; FMT_TF32: fp32 elements already rounded to tf32.
// nprod 3 uses A_lo/B_lo (hi.hi + hi.lo + lo.hi); nprod 1 ignores them.
struct GemmOperands {
    Format fmt;
    int nprod;
    const void *A_hi, *A_lo;
    long long lda;   // elements; lda * element size must be a multiple of 16 bytes
    const void *B_hi, *B_lo;
    long long ldb;
    int drain_kb = 0;   // k-blocks per TMEM chunk drained to fp32 registers (0 = library default)
    bool accumulate = false;   // D += A . B^T instead of D = A . B^T
    bool tile_sync = true;     // co-resident tiles may wait for one another (bounded) to share operand slices
    const std::function<int(int)> *planned = nullptr;   // called before each launch with its CTAs
};

// K must be a multiple of 64 (bf16) or 32 (tf32); operands must be readable up to K columns.
int gemm(const GemmOperands &op, int M, int N, int K, float *D, long long ldd, cudaStream_t st, unsigned *err);

// One sub-problem of a grouped launch: D[d_off + m * ldd + n] (+)= sum_k A[a_row + m, a_k + k] B[b_row + n, b_k + k]
// for m < M, n < N, k < K (K a multiple of the 128-byte k-block; a_k, b_k multiples of it too).
struct GemmGroup {
    int M, N, K;
    int a_row, a_k, b_row, b_k;
    long long d_off;
};

// Several sub-problems over the same A (a_rows x a_cols) and B (b_rows x b_cols) buffers in one
// persistent launch (every 64 groups one launch): the tiles of all groups share the machine, so
// groups of a few tiles each leave no SM idle.
int gemm_grouped(const GemmOperands &op, long long a_rows, long long a_cols, long long b_rows, long long b_cols,
                 const GemmGroup *groups, int n_groups, float *D, long long ldd, cudaStream_t st, unsigned *err);

// [a|b] of every group (columns 2Nc) taken straight to the averages' weights: c and d of the same rows and
// columns are one more short contraction of the tile (operands A_* (a_rows x ld) and B_* (2Nc x ld), columns
// col[g] .. col[g] + K[g] of group g; K[g] = 0: c = d = 0), and instead of a, b, c, d the weights
//   Cw = [rho (-d/3 + d4 b/4) / 2 | rho (-c/3 + d4 a/8)],   AB = [-rho a/6 | -rho b/3]
// are stored, split, in rows of N2pc columns (zero past 2Nc); a group's rows start at row d_off.  fp32
// arithmetic when Nc is a multiple of 4, FP64 otherwise.
struct WeightsOut {
    const void *A_hi, *A_lo, *B_hi, *B_lo;
    long long ld;
    std::vector<int> K, col;
    const double *rho;
    int Nc, N2pc, d4;
    void *cw_hi, *cw_lo, *ab_hi, *ab_lo;
};
bool weights_fit(Format fmt, int nprod, int K);   // K of [c|d] that the epilogue can take (two chunks)
int gemm_grouped_weights(const GemmOperands &op, long long a_rows, long long a_cols, long long b_rows, long long b_cols,
                         const GemmGroup *groups, int n_groups, const WeightsOut &wo, cudaStream_t st, unsigned *err);

// Budget of every bounded wait of later launches (default 4 s), and a one-shot request that the next
// launch's producers issue no copy (its MMA warps' first wait then runs out): the abort-path test.
void set_wait_budget_ns(unsigned long long ns);
unsigned long long wait_budget_ns();
void stall_next_launch();

}  // namespace tc
}  // namespace tdscha
