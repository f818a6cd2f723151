// dgemm.cu -- FP64 contraction C = A . B^T of many small sub-problems in one launch (both operands K-contiguous).
//
// The class contractions of a small system are eight or fourteen products of a few 0.1 GF each; one library call per
// class is bound by its launches (48 kernels per apply on 2x2x2, 8 to 14 us each, twice that where the library splits K).
// Here a CTA takes one 32- or 64-row x 16- or 64-column tile of any class, and a contraction over the configurations (few tiles,
// long K) is cut into slices of K whose partial tiles the last CTA to finish adds up in slice order (the result does not
// depend on which one that is).  Four warps, m8n8k4 FP64 tensor instructions, three stages of 16 k in shared memory with
// 20-double rows: the 8 x 4 fragment reads of a half warp fall on all banks.
// Measured, us, one library call per class -> this: 2 vectors on 2x2x2, N = 2000: [a|b] 86 -> 42, [c|d] 61 -> 17, Z 121 -> 46,
// F 101 -> 21; F of 2 vectors on 4x4x4, N = 10000: 912 -> 280.  Large classes come out at 30 TFLOP/s: the FP64 unit, with
// 10 % lost to what its warps wait for; 16x8x8 instructions and 96-row tiles of 8 warps were no faster.
#include <algorithm>
#include <cstdint>

#include "dgemm.cuh"

namespace tdscha {
namespace {

constexpr int MAX_G = 64, BK = 16, LDS = BK + 4, STAGES = 3, THREADS = 128;
constexpr int MAX_CTAS = DGEMM_MAX_CTAS;

struct DGroup {
    int M, N, K, a_row, a_k, b_row, b_k, tile0, tiles_m, pad;
    long long d_off;
};
struct DTable {
    int n, slices;
    DGroup g[MAX_G];
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const double *src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};" : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}

// BM = 32 or 64 rows; the warps form a 2 x 2 grid (4 x 1 for 16 columns)
template <int BM, int BN>
__global__ void __launch_bounds__(THREADS) dgemm_grouped_kernel(const double *__restrict__ A, long long lda, const double *__restrict__ B,
                                                                long long ldb, double *__restrict__ C, long long ldc,
                                                                const __grid_constant__ DTable t, double *__restrict__ part,
                                                                unsigned *__restrict__ count, int accumulate) {
    constexpr int WN = BN == 16 ? 1 : 2, WR = BM * WN / 4, WC = BN / WN, MI = WR / 8, NI = WC / 8;   // 8 x 8 tiles of a warp
    extern __shared__ __align__(16) double sm[];
    double *As = sm, *Bs = sm + STAGES * BM * LDS;
    int gi = 0;
    while (gi + 1 < t.n && t.g[gi + 1].tile0 <= (int)blockIdx.x) ++gi;
    const DGroup &G = t.g[gi];
    const int lt = blockIdx.x - G.tile0, m0 = (lt % G.tiles_m) * BM, n0 = (lt / G.tiles_m) * BN;
    const int kblocks = G.K / BK, per = (kblocks + t.slices - 1) / t.slices;
    const int kb0 = min(kblocks, (int)blockIdx.y * per), kb1 = min(kblocks, kb0 + per);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t as_u = static_cast<uint32_t>(__cvta_generic_to_shared(As)), bs_u = static_cast<uint32_t>(__cvta_generic_to_shared(Bs));

    // 8 chunks of 16 bytes per row: thread -> (row, chunk)
    const int lr = tid >> 3, lc = (tid & 7) * 2;
    auto issue = [&](int kb, int s) {
        const long long ka = G.a_k + (long long)kb * BK + lc, kc = G.b_k + (long long)kb * BK + lc;
#pragma unroll
        for (int r = 0; r < BM; r += THREADS / 8) {
            const bool v = m0 + r + lr < G.M;
            cp_async16(as_u + (uint32_t)(((s * BM + r + lr) * LDS + lc) * 8), A + (long long)(G.a_row + (v ? m0 + r + lr : 0)) * lda + ka, v);
        }
#pragma unroll
        for (int r = 0; r < BN; r += THREADS / 8) {
            const bool v = n0 + r + lr < G.N;
            cp_async16(bs_u + (uint32_t)(((s * BN + r + lr) * LDS + lc) * 8), B + (long long)(G.b_row + (v ? n0 + r + lr : 0)) * ldb + kc, v);
        }
    };
    double acc[MI][NI][2];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NI; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    const int nk = kb1 - kb0;
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < nk) issue(kb0 + s, s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    const int wm = warp / WN * WR, wn = warp % WN * WC;
    const int fr = lane >> 2, fk = lane & 3;
    for (int k = 0; k < nk; ++k) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();   // stage k is in, and stage k - 1 is no longer read
        if (k + STAGES - 1 < nk) issue(kb0 + k + STAGES - 1, (k + STAGES - 1) % STAGES);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const double *a = As + (k % STAGES) * BM * LDS + (wm + fr) * LDS + fk, *b = Bs + (k % STAGES) * BN * LDS + (wn + fr) * LDS + fk;
#pragma unroll
        for (int kk = 0; kk < BK; kk += 4) {
            double av[MI], bv[NI];
#pragma unroll
            for (int i = 0; i < MI; ++i) av[i] = a[i * 8 * LDS + kk];
#pragma unroll
            for (int j = 0; j < NI; ++j) bv[j] = b[j * 8 * LDS + kk];
#pragma unroll
            for (int i = 0; i < MI; ++i)
#pragma unroll
                for (int j = 0; j < NI; ++j) dmma(acc[i][j], av[i], bv[j]);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");

    if (t.slices > 1) {
        // partial tiles [tile][slice][register pair][thread]; the last CTA of the tile adds them in slice order
        double2 *mine = reinterpret_cast<double2 *>(part) + ((long long)blockIdx.x * t.slices + blockIdx.y) * (MI * NI * THREADS) + tid;
#pragma unroll
        for (int i = 0; i < MI; ++i)
#pragma unroll
            for (int j = 0; j < NI; ++j) mine[(i * NI + j) * THREADS] = make_double2(acc[i][j][0], acc[i][j][1]);
        __threadfence();
        __shared__ unsigned last;
        __syncthreads();
        if (tid == 0) {
            last = atomicAdd(&count[blockIdx.x], 1u);
            if (last == (unsigned)t.slices - 1) count[blockIdx.x] = 0;   // ready for the next launch
        }
        __syncthreads();
        if (last != (unsigned)t.slices - 1) return;
        __threadfence();
        const double2 *all = reinterpret_cast<const double2 *>(part) + (long long)blockIdx.x * t.slices * (MI * NI * THREADS) + tid;
#pragma unroll
        for (int i = 0; i < MI; ++i)
#pragma unroll
            for (int j = 0; j < NI; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
        for (int s = 0; s < t.slices; ++s)
#pragma unroll
            for (int i = 0; i < MI; ++i)
#pragma unroll
                for (int j = 0; j < NI; ++j) {
                    const double2 v = __ldcg(all + ((long long)s * MI * NI + i * NI + j) * THREADS);
                    acc[i][j][0] += v.x;
                    acc[i][j][1] += v.y;
                }
    }
#pragma unroll
    for (int i = 0; i < MI; ++i) {
        const int m = m0 + wm + i * 8 + fr;
        if (m >= G.M) continue;
        double *row = C + G.d_off + (long long)m * ldc;
#pragma unroll
        for (int j = 0; j < NI; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int n = n0 + wn + j * 8 + 2 * fk + e;
                if (n < G.N) row[n] = accumulate ? row[n] + acc[i][j][e] : acc[i][j][e];
            }
    }
}

template <int BM, int BN>
int launch(const double *A, long long lda, const double *B, long long ldb, const tc::GemmGroup *gs, int n, double *C, long long ldc,
           bool accumulate, double *part, unsigned *count, cudaStream_t st) {
    DTable t{};
    t.n = n;
    int tiles = 0, kmax = 0;
    for (int i = 0; i < n; ++i) {
        DGroup &d = t.g[i];
        d.M = gs[i].M; d.N = gs[i].N; d.K = gs[i].K;
        d.a_row = gs[i].a_row; d.a_k = gs[i].a_k; d.b_row = gs[i].b_row; d.b_k = gs[i].b_k;
        d.d_off = gs[i].d_off;
        d.tile0 = tiles;
        d.tiles_m = ceil_div(d.M, BM);
        tiles += d.tiles_m * ceil_div(d.N, BN);
        kmax = std::max(kmax, d.K);
    }
    // Slices of K (8 k-blocks at least): the machine takes ceil(CTAs / 148) rounds of one slice each, to which a CTA
    // adds about 14 k-blocks of start, write-out and adding up, and the last CTA the latency of its own slice.  Against
    // four CTAs per SM whatever the shape: F of 32 vectors on 2x2x2 276 -> 228 us, Z of 8 vectors 168 -> 130.
    t.slices = 1;
    double best = 1e300;
    for (int s = 1; s == 1 || (s * tiles <= MAX_CTAS && s <= kmax / BK / 8); ++s) {
        const double kb = (double)kmax / BK / s, cost = ceil_div(tiles * s, 148) * (kb + 14.0) + 2.0 * kb;
        if (cost < best) { best = cost; t.slices = s; }
    }
    constexpr int smem = STAGES * (BM + BN) * LDS * (int)sizeof(double);
    TD_TRY((allow_smem<dgemm_grouped_kernel<BM, BN>>(smem)));
    dgemm_grouped_kernel<BM, BN><<<dim3((unsigned)tiles, (unsigned)t.slices), THREADS, smem, st>>>(A, lda, B, ldb, C, ldc, t,
                                                                                                   part, count, accumulate ? 1 : 0);
    TD_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace

size_t dgemm_part_bytes() { return (size_t)MAX_CTAS * 64 * 64 * sizeof(double); }

bool dgemm_fits(const double *A, long long lda, const double *B, long long ldb, const std::vector<tc::GemmGroup> &gs) {
    bool ok = lda % 2 == 0 && ldb % 2 == 0 && (reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) % 16 == 0;
    for (const auto &g : gs) ok = ok && g.M > 0 && g.N > 0 && g.K > 0 && g.K % BK == 0 && g.a_k % 2 == 0 && g.b_k % 2 == 0;
    return ok;
}

int dgemm_grouped(const double *A, long long lda, const double *B, long long ldb, const std::vector<tc::GemmGroup> &gs, double *C,
                  long long ldc, bool accumulate, double *part, unsigned *count, cudaStream_t st) {
    // 64-row tiles move half the operand bytes per product of 32-row ones (4 % faster where neither pads: [a|b] of 2 vectors
    // on 3x3x3, N = 20000, 6.25 and 6.54 ms); 32 where 64 would compute 1.1 times the rows or more (2 vectors on 2x2x2:
    // Z 46 us, with 64 rows 56).
    long long w32 = 0, w64 = 0;
    for (const auto &g : gs) {
        w32 += round_up(g.M, 32) * g.N * g.K;
        w64 += round_up(g.M, 64) * g.N * g.K;
    }
    // columns per tile: the products over a class's modes (5 to 16 columns) are bound by the rows' stream, and with 64
    // columns by products that are thrown away (F of 24 vectors on 3x3x3, N = 1200: 350 -> 160 us; 2 vectors on 4x4x4,
    // N = 10000: 570 -> 280)
    int nmax = 0;
    for (const auto &g : gs) nmax = std::max(nmax, g.N);
    const bool m64 = w64 <= 1.1 * w32;
    const auto run = nmax <= 16 ? (m64 ? launch<64, 16> : launch<32, 16>) : (m64 ? launch<64, 64> : launch<32, 64>);
    for (size_t i = 0; i < gs.size(); i += MAX_G) {
        const int n = (int)std::min<size_t>(MAX_G, gs.size() - i);
        TD_TRY(run(A, lda, B, ldb, gs.data() + i, n, C, ldc, accumulate, part, count, st));
    }
    return 0;
}

}  // namespace tdscha
