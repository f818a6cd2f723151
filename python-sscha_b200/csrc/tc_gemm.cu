// tc_gemm.cu -- hand-written sm_100a tensor-core contraction D = A . B^T for the ensemble averages.
//
//   A (M x K), B (N x K): row-major, K contiguous ("K-major" for both UMMA operands), stored as
//   bf16 or tf32-rounded fp32; optionally as hi/lo splits so that three products
//   hi.hi + hi.lo + lo.hi recover ~16 (bf16) / ~21 (tf32) significant bits.
//   D (M x N): fp32, row-major, written with edge masking.
//
// Pipeline (persistent: one CTA per SM walks output tiles of up to 128 x 256; 12 warps):
//   warps 0, 10, 11 : TMA producers of the P tiles, the Q hi and the Q lo tiles (P = A, Q = B or the other
//                 way round) -- cp.async.bulk.tensor.2d into a ring of 128B-swizzled tiles, completion
//                 tracked by mbarrier transaction counts.  One thread issues a copy about every 100 ns,
//                 which bounds narrow tiles, so the copies of a k-block are shared out;
//   warp 1      : allocates 512 TMEM columns (two accumulator buffers); one elected thread issues
//                 tcgen05.mma (kind::f16 for bf16, kind::tf32) from shared-memory descriptors,
//                 accumulating in TMEM, and frees each ring slot with tcgen05.commit -> mbarrier;
//   warps 2..9  : epilogue -- tcgen05.ld 32x32b from TMEM (warp w reads lanes 32*(w%4)..+31, half of
//                 the columns), fp32 sums in registers, stores to global memory through a per-warp
//                 shared-memory block (full 128-byte lines per store instruction).
// Every mbarrier wait is bounded by a %globaltimer budget; on expiry the CTA raises ERR_TIMEOUT in
// the caller's error word, drains its own TMA copies (bounded), frees TMEM and returns.
#include <cuda.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <functional>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>
#include <utility>
#include <vector>

#include "common.cuh"
#include "tc_gemm.cuh"

namespace tdscha {
namespace tc {

constexpr int BM = 128;
constexpr int NUM_THREADS = 384;   // P producer, MMA, 8 epilogue warps, 2 Q producers
constexpr unsigned long long DEFAULT_WAIT_BUDGET_NS = 4000000000ull;   // 4 s per pipeline wait
constexpr unsigned long long DRAIN_BUDGET_NS = 4000000000ull;          // 4 s per wait of the abort path

// Budget of every pipeline wait of the next launches (tdscha_set_wait_budget), and a one-shot request
// that the next launch's producers issue no copy, so that the MMA warps' first wait can only end by
// running out (tdscha_debug_stall_next_contraction: a test of the abort path).
static std::atomic<unsigned long long> g_wait_budget_ns{DEFAULT_WAIT_BUDGET_NS};
static std::atomic<int> g_stall_next{0};

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ unsigned long long globaltimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait of a whole warp: true when the phase completed, false (for every lane alike) on timeout
// or when another role aborted.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag,
                                          unsigned long long budget_ns) {
    if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return true;
    unsigned long long t0 = 0;
    for (uint32_t it = 0;; ++it) {
        if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return true;
        if ((it & 255u) == 255u) {
            bool stop = *abort_flag != 0;
            const unsigned long long t = globaltimer();
            if (t0 == 0) t0 = t;
            else stop = stop || t - t0 > budget_ns;
            if (__any_sync(0xffffffffu, stop)) return false;
        }
    }
}
// The same for one thread (the abort path's drain).
__device__ __forceinline__ bool mbar_wait_thread(uint32_t bar, uint32_t parity, unsigned long long budget_ns) {
    const unsigned long long t0 = globaltimer();
    while (!mbar_try(bar, parity))
        if (globaltimer() - t0 > budget_ns) return false;
    return true;
}
// One lane of a converged warp.
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t e;
    asm volatile(
        "{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(e));
    return e;
}

__device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Loose alignment of the CTAs' tile starts.  Each producer counts its tile starts in a global
// counter; before loading its i-th tile it waits (at most `budget_ns`, then goes on regardless)
// until every CTA that has an i-th tile has started it.  CTAs then walk the K range of concurrent
// tiles together and the A / B panels they share are read from HBM once and hit in L2 afterwards;
// without it they drift apart over the long K loops and most panel reads miss.  Purely a
// performance hint: results never depend on it.
__device__ __forceinline__ void tile_start_sync(unsigned *counter, unsigned target, unsigned long long budget_ns) {
    atomicAdd(counter, 1u);
    if (budget_ns == 0) return;
    const unsigned long long t0 = globaltimer();
    while (ld_acquire_gpu(counter) < target) {
        if (globaltimer() - t0 > budget_ns) break;
        __nanosleep(128);
    }
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int c0, int c1, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(bar)
        : "memory");
}

// Shared-memory matrix descriptor of a K-major tile stored as rows of KBYTES (128 or 64) bytes with the
// swizzle of that width (what TMA writes with CU_TENSOR_MAP_SWIZZLE_128B / _64B): start address >> 4 in
// bits 0-13, leading byte offset (unused for swizzled K-major, 16 B) in bits 16-29, stride byte offset
// (one 8-row swizzle atom) in bits 32-45, descriptor version 1 in bits 46-47, swizzle mode (2: 128B,
// 4: 64B) in bits 61-63.  The high word is the same for every tile, and a step along K or to another
// tile only adds (bytes >> 4) to the low word (addresses stay below 256 KB).
template <int KBYTES>
constexpr uint32_t DESC_HI = ((8u * KBYTES) >> 4) | (1u << 14) | ((KBYTES == 128 ? 2u : 4u) << 29);
__device__ __forceinline__ uint32_t desc_lo(uint32_t saddr) { return (saddr >> 4) | (1u << 16); }

// Instruction descriptor for kind::f16 / kind::tf32 with fp32 accumulation, both operands K-major:
// D format (bits 4-5) = 1 (f32); A/B format (bits 7-9, 10-12) = 1 (bf16) or 2 (tf32);
// N >> 3 in bits 17-22; M >> 4 in bits 24-28.
__host__ __device__ constexpr uint32_t make_idesc(bool tf32, int m, int n) {
    return (1u << 4) | ((tf32 ? 2u : 1u) << 7) | ((tf32 ? 2u : 1u) << 10) |
           ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// issued by the lane whose `leader` is set; the others pass through (no divergent branch, so the
// descriptors stay in uniform registers)
template <bool TF32, int KBYTES>
__device__ __forceinline__ void umma(uint32_t tmem_d, uint32_t adesc, uint32_t bdesc, uint32_t idesc, uint32_t accum, uint32_t leader) {
    const uint64_t ad = ((uint64_t)DESC_HI<KBYTES> << 32) | adesc, bd = ((uint64_t)DESC_HI<KBYTES> << 32) | bdesc;
    if constexpr (TF32) {
        asm volatile(
            "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
            "@q tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(tmem_d), "l"(ad), "l"(bd), "r"(idesc), "r"(accum), "r"(leader));
    } else {
        asm volatile(
            "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
            "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(tmem_d), "l"(ad), "l"(bd), "r"(idesc), "r"(accum), "r"(leader));
    }
}

__device__ __forceinline__ void umma_commit(uint32_t bar, uint32_t leader) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
        ::"r"(bar), "r"(leader) : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Sub-problems of one launch (a single contraction is one group).  Each 128-row tile of the P operand
// meets tiles of `tn` rows of the Q operand: P = A, Q = B, or the other way round (swapped).
// tile0 = tiles of the groups before.
constexpr int MAX_GROUPS = 64;
struct DevGroup {
    int np, nq, K, p_row, p_k, q_row, q_k, tile0, num_p, num_q, tn;
    int kw, pw_k, qw_k;        // weights epilogue: K and columns of the [c|d] operands
    long long d_off;
};
struct GroupTable {
    int n, total_tiles;
    int p_rows;                // P rows of a tile: 128, or 64 (half the P fetch of an MMA, and more tiles)
    int p_box, q_box;          // rows of one TMA box of each operand
    int stages, stage_bytes;   // copy ring
    int q_off;                 // bytes of the stage in front of the Q tiles (hi, then lo)
    int q_bytes;               // bytes of one Q tile's slot
    DevGroup g[MAX_GROUPS];
};

__device__ __forceinline__ const DevGroup &group_of(const GroupTable &gt, int t) {
    int g = 0;
    while (g + 1 < gt.n && gt.g[g + 1].tile0 <= t) ++g;
    return gt.g[g];
}

// Tile order of the persistent schedule: groups of `gp` P-tiles, Q-tiles of a group in turn, P
// fastest inside a group.  The ~148 tiles in flight then form a gp x (148/gp) block that shares its
// P rows and Q rows through L2, instead of one Q column of tiles streaming all of P from HBM.
// Swapped launches keep a P tile's few Q tiles next to each other (gp = 1).
__device__ __forceinline__ void tile_coords(int t, int num_p, int num_q, int gp, int &p_blk, int &q_blk) {
    const int per_group = gp * num_q;
    const int g = t / per_group, rem = t % per_group;
    const int p_first = g * gp;
    const int rows = min(gp, num_p - p_first);
    q_blk = rem / rows;
    p_blk = p_first + rem % rows;
}

constexpr int MAX_STAGES = 12;
constexpr int EPI_WARPS = 8;                       // 2 warps per TMEM lane quadrant
constexpr int EPI_BUF_FLOATS = 32 * 32;            // one epilogue warp's 32 x 32 staging block
constexpr int SMEM_MAX = 227 * 1024;
constexpr int SMEM_FIXED = 1024 /*align*/ + 512 /*barriers*/;
constexpr int EPI_STAGING = EPI_WARPS * EPI_BUF_FLOATS * 4;
constexpr int epi_staging(bool swap, bool weights) { return swap ? (weights ? 2 * EPI_STAGING : 0) : EPI_STAGING; }
constexpr uint32_t TMEM_COLS = 512;                // two accumulator buffers of up to 256 columns

template <bool TF32, int KBYTES>
struct KBlock {
    static constexpr int ELEMS = KBYTES / (TF32 ? 4 : 2);   // K per stage
    static constexpr int UMMA_K = TF32 ? 8 : 16;   // K per instruction (32 bytes)
};

// What happens to a tile's sums.  EpiArgs<false>: stored to D.  EpiArgs<true>: the averages' weights.  The
// tile holds a (columns k < Nc) and b (k >= Nc) of its rows; one or two more chunks of the same tile
// over the rows' and configurations' mode components give c and d, and the stored values are
//   k < Nc:   Cw[Nc + k] = rho_k (-c/3 + d4 a/8),                AB[k] = -rho_k a/6
//   k >= Nc:  Cw[k - Nc] = rho_(k-Nc) (-d/3 + d4 b/4) / 2,       AB[k] = -rho_(k-Nc) b/3
// split into hi / lo, zero from column 2Nc to N2pc.
template <bool WEIGHTS>
struct EpiArgs {
    int unused;
};
template <>
struct EpiArgs<true> {
    CUtensorMap p_hi, p_lo, q_hi, q_lo;   // operands of [c|d]
    const double *rho;
    int Nc, N2pc, d4;
    int f64;                              // FP64 arithmetic (Nc not a multiple of 4), else fp32
    int drain_w;                          // stages per chunk of [c|d]
    void *cw_hi, *cw_lo, *ab_hi, *ab_lo;  // rows of N2pc columns; the group's d_off is its first row
};

// hi and lo of two weights in the storage format, as bits (bf16: packed into one word each).  Products and
// differences are rounded one by one.
template <bool TF32, typename T>
struct Split2 {
    uint32_t h0, h1, l0, l1;   // tf32: one word per weight; bf16: h0, l0 hold both
    __device__ __forceinline__ Split2(T x0, T x1) {
        if constexpr (TF32) {
            const float f0 = tf32_round((float)x0), f1 = tf32_round((float)x1);
            h0 = __float_as_uint(f0);
            h1 = __float_as_uint(f1);
            if constexpr (sizeof(T) == 8) {
                l0 = __float_as_uint(tf32_round((float)(x0 - (double)f0)));
                l1 = __float_as_uint(tf32_round((float)(x1 - (double)f1)));
            } else {
                l0 = __float_as_uint(tf32_round(__fsub_rn(x0, f0)));
                l1 = __float_as_uint(tf32_round(__fsub_rn(x1, f1)));
            }
        } else {
            h0 = pack((float)x0, (float)x1);
            const float f0 = __uint_as_float(h0 << 16), f1 = __uint_as_float(h0 & 0xffff0000u);
            if constexpr (sizeof(T) == 8) l0 = pack((float)(x0 - (double)f0), (float)(x1 - (double)f1));
            else l0 = pack(__fsub_rn(x0, f0), __fsub_rn(x1, f1));
            h1 = l1 = 0;
        }
    }
    static __device__ __forceinline__ uint32_t pack(float a, float b) {   // a in the low half
        uint32_t r;
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
        return r;
    }
};

// The factors of one configuration column (first: a and c, else b and d) and the weights of one element,
// v = a or b, w = c or d, in T = float or double arithmetic.
template <typename T>
struct WeightCol {
    T rc, ra, s;   // of Cw; of AB; of v in Cw (0 without d4)
    bool first;
    __device__ __forceinline__ WeightCol() {}
    __device__ __forceinline__ WeightCol(double rho, bool first_, int d4) : first(first_) {
        if constexpr (sizeof(T) == 8) {
            rc = first ? rho : 0.5 * rho;
            ra = -rho;
            s = d4 ? (first ? 0.125 : 0.25) : 0.0;
        } else {
            const float r = (float)rho;
            rc = first ? r : 0.5f * r;
            ra = -r;
            s = d4 ? (first ? 0.125f : 0.25f) : 0.f;
        }
    }
    __device__ __forceinline__ T cw(float v, float w) const {
        if constexpr (sizeof(T) == 8) return rc * (div_const<3>(-(double)w) + (s != 0.0 ? (double)v * s : 0.0));
        else return __fmul_rn(rc, __fmaf_rn(v, s, __fmul_rn(-w, 1.f / 3.f)));   // v s is exact: rounded once
    }
    __device__ __forceinline__ T ab(float v) const {
        if constexpr (sizeof(T) == 8) {
            const double y = ra * (double)v;
            return first ? div_const<6>(y) : div_const<3>(y);
        } else {
            return __fmul_rn(__fmul_rn(ra, v), first ? 1.f / 6.f : 1.f / 3.f);
        }
    }
};
// One weight, hi and lo, at element `i` of the output arrays
template <bool TF32, int NPROD>
__device__ __forceinline__ void store_weight(void *hi, void *lo, long long i, uint32_t h, uint32_t l) {
    if constexpr (TF32) {
        static_cast<uint32_t *>(hi)[i] = h;
        if (NPROD == 3) static_cast<uint32_t *>(lo)[i] = l;
    } else {
        static_cast<uint16_t *>(hi)[i] = (uint16_t)h;
        if (NPROD == 3) static_cast<uint16_t *>(lo)[i] = (uint16_t)l;
    }
}

// 32 rows x 16 columns of a tile: v in the first half of the warp's block, w in the second, 16-byte chunks
// XOR-swizzled (chunk j of row r at j ^ (r / 2 & 3)).
// fp32 arithmetic (Nc a multiple of 4): lane = (row of 8, chunk of 4 columns, all a or all b), vector stores.
template <bool TF32, int NPROD>
__device__ __forceinline__ void weights_block_f32(const EpiArgs<true> &ea, const float *wbuf, long long row0, int rows, int k0, int k_end) {
    const int lane = threadIdx.x & 31, rsub = lane >> 2, chk = lane & 3;
    const int k = k0 + 4 * chk, Nc = ea.Nc;
    if (k >= k_end) return;   // k_end is a multiple of 4 here
    WeightCol<float> col[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) col[e] = WeightCol<float>(__ldg(ea.rho + (k < Nc ? k + e : k + e - Nc)), k < Nc, ea.d4);
    using E = typename std::conditional<TF32, float, uint16_t>::type;
    const long long o = (row0 + rsub) * ea.N2pc, oc = o + (k < Nc ? Nc + k : k - Nc);
    E *ch = static_cast<E *>(ea.cw_hi) + oc, *cl = static_cast<E *>(ea.cw_lo) + oc;
    E *ah = static_cast<E *>(ea.ab_hi) + o + k, *al = static_cast<E *>(ea.ab_lo) + o + k;
#pragma unroll 2
    for (int i = rsub; i < rows; i += 8) {
        const int c = i * 16 + 4 * (chk ^ ((i >> 1) & 3));
        const float4 v = *reinterpret_cast<const float4 *>(wbuf + c), w = *reinterpret_cast<const float4 *>(wbuf + 512 + c);
        const Split2<TF32, float> c0(col[0].cw(v.x, w.x), col[1].cw(v.y, w.y)), c1(col[2].cw(v.z, w.z), col[3].cw(v.w, w.w));
        const Split2<TF32, float> a0(col[0].ab(v.x), col[1].ab(v.y)), a1(col[2].ab(v.z), col[3].ab(v.w));
        const long long d = (long long)(i - rsub) * ea.N2pc;
        if constexpr (TF32) {
            *reinterpret_cast<uint4 *>(ch + d) = make_uint4(c0.h0, c0.h1, c1.h0, c1.h1);
            *reinterpret_cast<uint4 *>(ah + d) = make_uint4(a0.h0, a0.h1, a1.h0, a1.h1);
            if (NPROD == 3) {
                *reinterpret_cast<uint4 *>(cl + d) = make_uint4(c0.l0, c0.l1, c1.l0, c1.l1);
                *reinterpret_cast<uint4 *>(al + d) = make_uint4(a0.l0, a0.l1, a1.l0, a1.l1);
            }
        } else {
            *reinterpret_cast<uint2 *>(ch + d) = make_uint2(c0.h0, c1.h0);
            *reinterpret_cast<uint2 *>(ah + d) = make_uint2(a0.h0, a1.h0);
            if (NPROD == 3) {
                *reinterpret_cast<uint2 *>(cl + d) = make_uint2(c0.l0, c1.l0);
                *reinterpret_cast<uint2 *>(al + d) = make_uint2(a0.l0, a1.l0);
            }
        }
    }
}
// FP64 arithmetic (any Nc): lane = (row of 2, column), so that 16 lanes store 16 neighbouring elements.
template <bool TF32, int NPROD>
__device__ __forceinline__ void weights_block_f64(const EpiArgs<true> &ea, const float *wbuf, long long row0, int rows, int k0, int k_end) {
    const int lane = threadIdx.x & 31, rsub = lane >> 4, c = lane & 15;
    const int k = k0 + c, Nc = ea.Nc;
    if (k >= k_end) return;
    const WeightCol<double> col(__ldg(ea.rho + (k < Nc ? k : k - Nc)), k < Nc, ea.d4);
    const int kc = k < Nc ? Nc + k : k - Nc;
#pragma unroll 1
    for (int i = rsub; i < rows; i += 4) {   // two rows of the lane at a time
        const int i1 = min(i + 2, rows - 1);
        const int c0 = i * 16 + 4 * ((c >> 2) ^ ((i >> 1) & 3)) + (c & 3), c1 = i1 * 16 + 4 * ((c >> 2) ^ ((i1 >> 1) & 3)) + (c & 3);
        const Split2<TF32, double> x(col.cw(wbuf[c0], wbuf[512 + c0]), col.cw(wbuf[c1], wbuf[512 + c1]));
        const Split2<TF32, double> y(col.ab(wbuf[c0]), col.ab(wbuf[c1]));
        const long long o = (row0 + i) * ea.N2pc, o1 = o + 2LL * ea.N2pc;
        store_weight<TF32, NPROD>(ea.cw_hi, ea.cw_lo, o + kc, x.h0, x.l0);
        store_weight<TF32, NPROD>(ea.ab_hi, ea.ab_lo, o + k, y.h0, y.l0);
        if (i + 2 < rows) {
            store_weight<TF32, NPROD>(ea.cw_hi, ea.cw_lo, o1 + kc, TF32 ? x.h1 : x.h0 >> 16, TF32 ? x.l1 : x.l0 >> 16);
            store_weight<TF32, NPROD>(ea.ab_hi, ea.ab_lo, o1 + k, TF32 ? y.h1 : y.h0 >> 16, TF32 ? y.l1 : y.l0 >> 16);
        }
    }
}

// `rows` rows of a swapped tile, this lane's configuration k: v (row, lane) in the first of the warp's two
// blocks, w in the second.
template <bool TF32, int NPROD, typename T>
__device__ __forceinline__ void weights_rows_of(const EpiArgs<true> &ea, const float *wbuf, long long row0, int rows, int k, double rho) {
    const int lane = threadIdx.x & 31;
    const WeightCol<T> col(rho, k < ea.Nc, ea.d4);
    const int kc = k < ea.Nc ? ea.Nc + k : k - ea.Nc;
#pragma unroll(sizeof(T) == 8 ? 1 : 2)
    for (int i = 0; i < rows; i += 2) {   // row i + 1 is in the block even where it is not stored
        const float v0 = wbuf[i * 32 + lane], v1 = wbuf[i * 32 + 32 + lane];
        const float w0 = wbuf[1024 + i * 32 + lane], w1 = wbuf[1024 + i * 32 + 32 + lane];
        const Split2<TF32, T> x(col.cw(v0, w0), col.cw(v1, w1)), y(col.ab(v0), col.ab(v1));
        const long long o = (row0 + i) * ea.N2pc, o1 = o + ea.N2pc;
        store_weight<TF32, NPROD>(ea.cw_hi, ea.cw_lo, o + kc, x.h0, x.l0);
        store_weight<TF32, NPROD>(ea.ab_hi, ea.ab_lo, o + k, y.h0, y.l0);
        if (i + 1 < rows) {
            store_weight<TF32, NPROD>(ea.cw_hi, ea.cw_lo, o1 + kc, TF32 ? x.h1 : x.h0 >> 16, TF32 ? x.l1 : x.l0 >> 16);
            store_weight<TF32, NPROD>(ea.ab_hi, ea.ab_lo, o1 + k, TF32 ? y.h1 : y.h0 >> 16, TF32 ? y.l1 : y.l0 >> 16);
        }
    }
}

// Persistent: CTA c processes tiles c, c + gridDim.x, ...  Each tile's K loop is split into chunks
// of `drain` k-blocks; a chunk accumulates from zero in one of two TMEM buffers (the MMA warp moves on
// to the other buffer) and the epilogue warps add it into round-to-nearest fp32 registers, which
// bounds the error of the tensor core's own fp32 accumulation to `drain` k-blocks.
//
// What bounds it: large tiles run at the tensor pipe (power-capped); narrow tiles (few output columns,
// long K) run at the cost of one k-block through the ring, so the MMA warp stays converged (elected
// issue, uniform descriptors whose low word only gets constants added) and the tile width is whatever
// the sub-problem needs, in steps of 16 columns, so that no copy, shared memory or MMA goes to padding.
//   MAXC: columns a tile may have (register accumulators of an epilogue thread = MAXC / 2);
//   KBYTES: bytes of K of a ring stage.  128, or 64 where stages of 128 would leave the ring two deep
//         (tiles wider than 192 columns in the split modes): half the shared memory then waits for copies
//         while the other half computes; four or five half stages keep three quarters of it in flight.
//         240 rows x 9998 x 512, tf32x3 (Z of five vectors on 3x3x3): 664 -> 596 us.
//   SWAP: P = B, so that a problem with few rows of A (one chain: 96 or 192 rows) puts them on the
//         MMA's N side, which steps by 16, instead of padding them to 128-row tiles.
// The three split products of a k-step are issued hi.hi, A_hi.B_lo, A_lo.B_hi in both orientations and
// for every width, so each output is the same sum in the same order whatever tile computes it.
template <int MAXC, bool TF32, int NPROD, bool SWAP, int KBYTES, bool WEIGHTS>
__global__ void __launch_bounds__(NUM_THREADS, 1)
tc_gemm_kernel(const __grid_constant__ CUtensorMap tmP_hi, const __grid_constant__ CUtensorMap tmP_lo,
               const __grid_constant__ CUtensorMap tmQ_hi, const __grid_constant__ CUtensorMap tmQ_lo,
               const __grid_constant__ GroupTable gt, int drain, int group_p, float *__restrict__ D, long long ldd, unsigned *err,
               unsigned *tile_sync, unsigned sync_ns, int accumulate, unsigned long long wait_ns, int stall,
               const __grid_constant__ EpiArgs<WEIGHTS> ea) {
    using KB = KBlock<TF32, KBYTES>;
    constexpr int EPI_COLS = MAXC / 2;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int S = gt.stages, stage_bytes = gt.stage_bytes;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + S * stage_bytes);
    // bars[0..MS) full, [MS..2MS) empty, then 2 accumulator full, 2 accumulator empty
    uint64_t *acc_full = bars + 2 * MAX_STAGES;
    uint64_t *acc_empty = bars + 2 * MAX_STAGES + 2;
    uint64_t *done_bar = bars + 2 * MAX_STAGES + 4;   // abort path: completion of every MMA issued
    volatile int *abort_flag = reinterpret_cast<volatile int *>(bars + 2 * MAX_STAGES + 5);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * MAX_STAGES + 6);
    float *epi_buf = reinterpret_cast<float *>(smem + S * stage_bytes + 512);   // epilogue staging blocks

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const int lane = threadIdx.x & 31;
    const int num_tiles = gt.total_tiles;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(smem_u32(&bars[s]), NPROD == 3 ? 3 : 2);   // one arrival per producer warp
            mbar_init(smem_u32(&bars[MAX_STAGES + s]), 1);
        }
        for (int x = 0; x < 2; ++x) {
            mbar_init(smem_u32(&acc_full[x]), 1);
            mbar_init(smem_u32(&acc_empty[x]), EPI_WARPS);
        }
        mbar_init(smem_u32(done_bar), 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t bar0 = smem_u32(bars), smem0 = smem_u32(smem);

    int issued = 0;      // k-blocks this producer handed to TMA (for the drain on abort)
    if ((warp == 0 || warp == 10 || (warp == 11 && NPROD == 3)) && !stall) {
        // ---------------- TMA producers: P (hi and lo), Q hi, Q lo ----------------
        const uint32_t leader = elect_one();
        const CUtensorMap *map0 = warp == 0 ? &tmP_hi : (warp == 10 ? &tmQ_hi : &tmQ_lo), *map = map0;
        if (leader) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
        const uint32_t dst0 = smem0 + (warp == 0 ? 0 : gt.q_off + (warp == 10 ? 0 : gt.q_bytes));
        int s = 0;
        uint32_t ph = 1;
        unsigned target = 0;   // tile starts of all CTAs up to and including this round
        bool ok = true;
        for (int t = blockIdx.x, round = 0; t < num_tiles && ok; t += gridDim.x, ++round) {
            target += (unsigned)min((int)gridDim.x, num_tiles - round * (int)gridDim.x);
            if (tile_sync && warp == 0) {
                if (leader) tile_start_sync(tile_sync, target, round > 0 ? sync_ns : 0ull);
                __syncwarp();
            }
            const DevGroup &G = group_of(gt, t);
            int pb, qb;
            tile_coords(t - G.tile0, G.num_p, G.num_q, group_p, pb, qb);
            const int num_kb = G.K / KB::ELEMS;
            int row, kc, nbox, box;
            if (warp == 0) {
                row = G.p_row + pb * gt.p_rows;
                kc = G.p_k;
                box = gt.p_box;
                nbox = 1;
            } else {
                row = G.q_row + qb * G.tn;
                kc = G.q_k;
                box = gt.q_box;
                nbox = (min(G.tn, G.nq - qb * G.tn) + box - 1) / box;
            }
            const uint32_t tx = (uint32_t)((warp == 0 && NPROD == 3 ? 2 : nbox) * box * KBYTES);
            int kb_all = num_kb;
            if constexpr (WEIGHTS) kb_all += G.kw / KB::ELEMS;
            const CUtensorMap *map_lo = &tmP_lo;
            map = map0;
            for (int kb = 0; kb < kb_all; ++kb, kc += KB::ELEMS) {
                if constexpr (WEIGHTS) {
                    if (kb == num_kb) {   // the [c|d] chunks of the tile
                        map = warp == 0 ? &ea.p_hi : (warp == 10 ? &ea.q_hi : &ea.q_lo);
                        map_lo = &ea.p_lo;
                        kc = warp == 0 ? G.pw_k : G.qw_k;
                    }
                }
                if (!mbar_wait(bar0 + 8 * (MAX_STAGES + s), ph, abort_flag, wait_ns)) { ok = false; break; }
                if (leader) {
                    const uint32_t dst = dst0 + s * stage_bytes, full = bar0 + 8 * s;
                    mbar_expect_tx(full, tx);
                    tma_load_2d(dst, map, kc, row, full);
                    if (warp == 0) {
                        if constexpr (NPROD == 3) tma_load_2d(dst + (gt.q_off >> 1), map_lo, kc, row, full);
                    } else {
                        for (int i = 1; i < nbox; ++i) tma_load_2d(dst + i * box * KBYTES, map, kc, row + i * box, full);
                    }
                }
                ++issued;
                if (++s == S) { s = 0; ph ^= 1u; }
            }
        }
        if (!ok) *abort_flag = 1;
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        const uint32_t leader = elect_one();
        const uint32_t desc0 = desc_lo(smem0), stage_d = (uint32_t)stage_bytes >> 4;
        const uint32_t d_plo = (uint32_t)gt.q_off >> 5, d_qhi = (uint32_t)gt.q_off >> 4;
        const uint32_t d_qlo = d_qhi + ((uint32_t)gt.q_bytes >> 4);
        int s = 0;
        uint32_t ph = 0, ch = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
            const DevGroup &G = group_of(gt, t);
            int pb, qb;
            tile_coords(t - G.tile0, G.num_p, G.num_q, group_p, pb, qb);
            const int ncol = (min(G.tn, G.nq - qb * G.tn) + 15) & ~15;
            const uint32_t idesc = make_idesc(TF32, gt.p_rows, ncol);
            const int num_kb = G.K / KB::ELEMS;
            int kb_all = num_kb;
            if constexpr (WEIGHTS) kb_all += G.kw / KB::ELEMS;
            for (int k0 = 0, k1; k0 < kb_all && ok; k0 = k1, ++ch) {
                k1 = min(num_kb, k0 + drain);
                if constexpr (WEIGHTS) {
                    if (k0 >= num_kb) k1 = min(kb_all, k0 + ea.drain_w);
                }
                const uint32_t X = ch & 1u;
                if (!mbar_wait(smem_u32(&acc_empty[X]), ((ch >> 1) & 1u) ^ 1u, abort_flag, wait_ns)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t dtm = tmem_base + X * 256u;
                uint32_t acc = 0;
                for (int kb = k0; kb < k1; ++kb) {
                    if (!mbar_wait(bar0 + 8 * s, ph, abort_flag, wait_ns)) { ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t d = desc0 + (uint32_t)s * stage_d;
#pragma unroll
                    for (int k = 0; k < KB::ELEMS / KB::UMMA_K; ++k) {
                        const uint32_t ko = k * 2;   // 32 bytes inside the swizzled row, >> 4
                        umma<TF32, KBYTES>(dtm, d + ko, d + d_qhi + ko, idesc, k > 0 ? 1u : acc, leader);
                        if constexpr (NPROD == 3) {
                            if constexpr (!SWAP) {
                                umma<TF32, KBYTES>(dtm, d + ko, d + d_qlo + ko, idesc, 1u, leader);
                                umma<TF32, KBYTES>(dtm, d + d_plo + ko, d + d_qhi + ko, idesc, 1u, leader);
                            } else {
                                umma<TF32, KBYTES>(dtm, d + d_plo + ko, d + d_qhi + ko, idesc, 1u, leader);
                                umma<TF32, KBYTES>(dtm, d + ko, d + d_qlo + ko, idesc, 1u, leader);
                            }
                        }
                    }
                    acc = 1;
                    umma_commit(bar0 + 8 * (MAX_STAGES + s), leader);   // slot s free once these MMAs retire
                    if (++s == S) { s = 0; ph ^= 1u; }
                }
                if (!ok) break;
                umma_commit(smem_u32(&acc_full[X]), leader);             // chunk accumulated in buffer X
            }
        }
        if (!ok) *abort_flag = 1;
    } else if (warp >= 2 && warp < 10) {
        // ---------------- epilogue: drain chunks into fp32 registers, store each tile ----------------
        const int ew = warp - 2;
        const int q = warp & 3;              // TMEM lane quadrant this warp may access
        const int half = ew >> 2;            // which half of the tile's columns this warp owns
        uint32_t ch = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
            const DevGroup &G = group_of(gt, t);
            int pb, qb;
            tile_coords(t - G.tile0, G.num_p, G.num_q, group_p, pb, qb);
            const int width = min(G.tn, G.nq - qb * G.tn);          // valid columns of this tile
            const int hw = ((width + 63) >> 6) << 5;                // columns of a half, a multiple of 32
            const int c_lo = half * hw;
            const int nsub = (min(hw, width - c_lo) + 31) >> 5;     // 32-column pieces of this warp
            const int rq = gt.p_rows >> 2;                          // P rows of a lane quadrant: 32, or 16 (lanes 0..15)
            const int num_kb = G.K / KB::ELEMS;
            float acc[EPI_COLS];
#pragma unroll
            for (int i = 0; i < EPI_COLS; ++i) acc[i] = 0.f;
            for (int k0 = 0; k0 < num_kb; k0 += drain, ++ch) {
                const uint32_t X = ch & 1u;
                if (!mbar_wait(smem_u32(&acc_full[X]), (ch >> 1) & 1u, abort_flag, wait_ns)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t tbase = tmem_base + ((uint32_t)(q * 32) << 16) + X * 256u + (uint32_t)c_lo;
#pragma unroll
                for (int sub = 0; sub < EPI_COLS / 32; ++sub) {
                    if (sub >= nsub) break;
                    uint32_t r[32];
                    tmem_ld32(tbase + (uint32_t)(sub * 32), r);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 32; ++i) acc[sub * 32 + i] += __uint_as_float(r[i]);
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acc_empty[X])) : "memory");
            }
            if (!ok) break;
            if constexpr (WEIGHTS) {
                // [c|d]: none, one or two chunks, summed in fp32 as the others
                const int nw = (G.kw / KB::ELEMS + ea.drain_w - 1) / ea.drain_w;
                for (int x = 0; x < nw && ok; ++x)
                    ok = mbar_wait(smem_u32(&acc_full[(ch + x) & 1u]), ((ch + x) >> 1) & 1u, abort_flag, wait_ns);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t tq = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)c_lo;
                const uint32_t t0 = tq + (ch & 1u) * 256u, t1 = tq + ((ch + 1) & 1u) * 256u;
                const int p0 = pb * gt.p_rows + q * rq, q0 = qb * G.tn + c_lo;
                float *wbuf = epi_buf + ew * EPI_BUF_FLOATS * (SWAP ? 2 : 1);
                auto release = [&]() {   // after the last read of the buffers
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    for (int x = 0; x < nw; ++x)
                        if (lane == 0)
                            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acc_empty[(ch + x) & 1u])) : "memory");
                };
                auto load_w = [&](int col, float (&w)[16]) {   // c or d of 16 columns, summed over its chunks
#pragma unroll
                    for (int i = 0; i < 16; ++i) w[i] = 0.f;
                    if (nw > 0) {
                        uint32_t r[16];
                        tmem_ld16(t0 + (uint32_t)col, r);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; ++i) w[i] += __uint_as_float(r[i]);
                        if (nw > 1) {
                            tmem_ld16(t1 + (uint32_t)col, r);
                            tmem_ld_wait();
#pragma unroll
                            for (int i = 0; i < 16; ++i) w[i] += __uint_as_float(r[i]);
                        }
                    }
                };
                // The sums leave the registers through the warp's 4 KB block and are worked on in small
                // loops: unrolled over all 128 registers the arithmetic overran the instruction cache
                // (about 120 us a tile instead of 16).
                if constexpr (SWAP) {
                    // lane = configuration, block row = output row: a store of the warp is a row's 64 or 128
                    // contiguous bytes
                    const int k = p0 + lane;
                    const bool mine = lane < rq && k < G.np;
                    const double rho = mine ? __ldg(ea.rho + (k < ea.Nc ? k : k - ea.Nc)) : 0.0;
#pragma unroll
                    for (int sub = 0; sub < EPI_COLS / 32; ++sub) {
                        if (sub >= nsub) break;
#pragma unroll
                        for (int i = 0; i < 32; ++i) wbuf[i * 32 + lane] = acc[sub * 32 + i];
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            float w[16];
                            load_w(sub * 32 + j * 16, w);
#pragma unroll
                            for (int i = 0; i < 16; ++i) wbuf[1024 + (j * 16 + i) * 32 + lane] = w[i];
                        }
                        if (sub + 1 == nsub) release();
                        const int rows = min(32, width - c_lo - sub * 32);
                        if (mine) {   // every lane reads only what it wrote
                            if (ea.f64) weights_rows_of<TF32, NPROD, double>(ea, wbuf, G.d_off + q0 + sub * 32, rows, k, rho);
                            else weights_rows_of<TF32, NPROD, float>(ea, wbuf, G.d_off + q0 + sub * 32, rows, k, rho);
                        }
                        __syncwarp();
                    }
                } else {
                    // lane = row, register = configuration column: 16 columns at a time, transposed in the block
                    // so that a store covers 32 (bf16) or 64 contiguous bytes of each of 8 rows
#pragma unroll
                    for (int p = 0; p < EPI_COLS / 16; ++p) {
                        if (p * 16 >= min(hw, width - c_lo)) break;
                        float w[16];
                        load_w(p * 16, w);
                        if ((p + 1) * 16 >= min(hw, width - c_lo)) release();
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const int c = 4 * (j ^ ((lane >> 1) & 3));
                            *reinterpret_cast<float4 *>(wbuf + lane * 16 + c) =
                                make_float4(acc[p * 16 + 4 * j], acc[p * 16 + 4 * j + 1], acc[p * 16 + 4 * j + 2], acc[p * 16 + 4 * j + 3]);
                            *reinterpret_cast<float4 *>(wbuf + 512 + lane * 16 + c) = make_float4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
                        }
                        __syncwarp();
                        if (ea.f64) weights_block_f64<TF32, NPROD>(ea, wbuf, G.d_off + p0, min(rq, G.np - p0), q0 + p * 16, qb * G.tn + width);
                        else weights_block_f32<TF32, NPROD>(ea, wbuf, G.d_off + p0, min(rq, G.np - p0), q0 + p * 16, qb * G.tn + width);
                        __syncwarp();   // the block is rewritten by the next 16 columns
                    }
                }
                if (nsub <= 0) release();
                ch += nw;
                // zero columns past 2Nc, by the tile that ends there
                const int rows = SWAP ? width : min(gt.p_rows, G.np - pb * gt.p_rows);
                const bool last = SWAP ? (pb + 1) * gt.p_rows >= G.np : qb * G.tn + width >= G.nq;
                if (last)
                    for (int i = ew; i < rows; i += EPI_WARPS) {
                        const long long o = (G.d_off + (SWAP ? qb * G.tn : pb * gt.p_rows) + i) * (long long)ea.N2pc;
                        for (int k = 2 * ea.Nc + lane; k < ea.N2pc; k += 32) {
                            store_weight<TF32, NPROD>(ea.cw_hi, ea.cw_lo, o + k, 0u, 0u);
                            store_weight<TF32, NPROD>(ea.ab_hi, ea.ab_lo, o + k, 0u, 0u);
                        }
                    }
            } else if constexpr (SWAP) {
                // lane = output column (P row), register = output row (Q row): each register is one
                // coalesced 128-byte store of the warp
                const int m = pb * gt.p_rows + q * rq + lane;
                if (lane < rq && m < G.np) {
                    float *dcol = D + G.d_off + (long long)(qb * G.tn + c_lo) * ldd + m;
#pragma unroll
                    for (int sub = 0; sub < EPI_COLS / 32; ++sub) {
                        if (sub >= nsub) break;
                        const int left = width - c_lo - sub * 32;
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (i < left) {
                                float *d = dcol + (long long)(sub * 32 + i) * ldd;
                                *d = accumulate ? *d + acc[sub * 32 + i] : acc[sub * 32 + i];
                            }
                    }
                }
            } else {
                // Store through this warp's 32 x 32 staging block: each lane writes its row's 32 columns, then
                // lanes 8i..8i+7 store 128 contiguous bytes of one row each, so one store instruction covers
                // four full 128-byte lines instead of 16 bytes of 32 rows.  16-byte chunks are XOR-swizzled by
                // row (chunk j of row r at j ^ (r & 7)), which keeps both phases free of bank conflicts.
                const int m0 = pb * gt.p_rows + q * rq, cb0 = qb * G.tn + c_lo, c_end = qb * G.tn + width;
                float *wbuf = epi_buf + ew * EPI_BUF_FLOATS;
                const bool vec = ((ldd & 3) == 0) && ((G.d_off & 3) == 0);
                const int rsub = lane >> 3, chk = lane & 7;
#pragma unroll
                for (int sub = 0; sub < EPI_COLS / 32; ++sub) {
                    if (sub >= nsub) break;
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        *reinterpret_cast<float4 *>(wbuf + lane * 32 + 4 * (j ^ (lane & 7))) =
                            make_float4(acc[sub * 32 + 4 * j], acc[sub * 32 + 4 * j + 1], acc[sub * 32 + 4 * j + 2],
                                        acc[sub * 32 + 4 * j + 3]);
                    __syncwarp();
                    const int cb = cb0 + sub * 32 + 4 * chk;
#pragma unroll 1
                    for (int i0 = 0; i0 < rq; i0 += 4) {
                        const int i = i0 + rsub;
                        const float4 v = *reinterpret_cast<const float4 *>(wbuf + i * 32 + 4 * (chk ^ (i & 7)));
                        const long long grow = (long long)m0 + i;
                        if (grow >= G.np) continue;
                        float *drow = D + G.d_off + grow * ldd;
                        if (vec && cb + 4 <= c_end) {
                            float4 o = v;
                            if (accumulate) {
                                const float4 old = *reinterpret_cast<const float4 *>(drow + cb);
                                o.x += old.x; o.y += old.y; o.z += old.z; o.w += old.w;
                            }
                            *reinterpret_cast<float4 *>(drow + cb) = o;
                        } else {
                            const float vv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                            for (int e = 0; e < 4; ++e)
                                if (cb + e < c_end) drow[cb + e] = accumulate ? drow[cb + e] + vv[e] : vv[e];
                        }
                    }
                    __syncwarp();   // the block is rewritten by the next 32 columns
                }
            }
        }
        if (!ok) *abort_flag = 1;
    }

    // ---------------- teardown ----------------
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*abort_flag) {
        if (threadIdx.x == 0) atomicOr(err, ERR_TIMEOUT);
        if ((warp == 0 || warp >= 10) && lane == 0) {
            // drain the TMA copies this CTA still has in flight (bounded; copies older than the last
            // `stages` completed before their slots were handed back)
            for (int g = (issued > S ? issued - S : 0); g < issued; ++g)
                mbar_wait_thread(bar0 + 8 * (g % S), (uint32_t)(g / S) & 1u, DRAIN_BUDGET_NS);
        }
        if (warp == 1) {
            // every MMA the elected lane issued has retired before the accumulator columns are released
            const uint32_t leader = elect_one();
            umma_commit(smem_u32(done_bar), leader);
            if (leader) mbar_wait_thread(smem_u32(done_bar), 0u, DRAIN_BUDGET_NS);
            __syncwarp();
        }
        __syncthreads();
    }
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                   const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

// rows x K operand, leading dimension ld (elements), box = box_rows x (kbytes of K)
static int make_map(CUtensorMap *map, const void *base, bool tf32, long long rows, long long K, long long ld, int box_rows, int kbytes) {
    EncodeTiledFn enc = get_encode();
    TD_CHECK(enc != nullptr, TDSCHA_ECUDA, "cuTensorMapEncodeTiled entry point unavailable");
    const size_t es = tf32 ? 4 : 2;
    TD_CHECK((reinterpret_cast<uintptr_t>(base) & 15) == 0, TDSCHA_EINVAL, "operand base not 16-byte aligned");
    TD_CHECK(((ld * es) & 15) == 0, TDSCHA_EINVAL, "operand row stride not a multiple of 16 bytes");
    cuuint64_t gdim[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t gstride[1] = {(cuuint64_t)(ld * es)};
    cuuint32_t box[2] = {(cuuint32_t)(kbytes / es), (cuuint32_t)box_rows};
    cuuint32_t estride[2] = {1, 1};
    CUresult r = enc(map, tf32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                     const_cast<void *>(base), gdim, gstride, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     kbytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    TD_CHECK(r == CUDA_SUCCESS, TDSCHA_ECUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return 0;
}

// k-blocks accumulated in TMEM before the epilogue drains them.  Split modes drain every k-block:
// their error is otherwise dominated by the tensor core's own fp32 accumulation; single-product
// modes are limited by operand rounding and drain every 16.  TDSCHA_DRAIN_KB overrides (tuning).
static int default_drain(int nprod) {
    static int env_d = -2;
    if (env_d == -2) {
        const char *env = getenv("TDSCHA_DRAIN_KB");
        env_d = env ? std::max(1, atoi(env)) : -1;
    }
    if (env_d > 0) return env_d;
    return nprod == 3 ? 1 : 16;
}

// Autotuner key: one choice per (format, products, M, N, K, device).
struct TuneKey {
    int tf32, nprod, M, N, K, dev;
    unsigned long long shape;   // hash of the sub-problems' shapes of a grouped launch (0: one problem)
    bool operator<(const TuneKey &o) const {
        return std::tie(tf32, nprod, M, N, K, dev, shape) < std::tie(o.tf32, o.nprod, o.M, o.N, o.K, o.dev, o.shape);
    }
};
static std::mutex g_tune_mutex;

// One tile-start counter per (device, stream), zeroed on the stream before every launch, so that
// contractions running concurrently on different streams never share one.  A counter (256 bytes)
// is allocated on a stream's first launch outside graph capture and kept for the process.
static std::mutex g_sync_mutex;
static std::map<std::pair<int, cudaStream_t>, unsigned *> g_sync_counter;

static int tile_sync_counter(int dev, cudaStream_t st, bool capturing, unsigned **out) {
    std::lock_guard<std::mutex> lock(g_sync_mutex);
    TD_CHECK(dev >= 0 && dev < 64, TDSCHA_EINVAL, "device index %d out of range", dev);
    auto it = g_sync_counter.find({dev, st});
    if (it != g_sync_counter.end()) { *out = it->second; return 0; }
    if (capturing) { *out = nullptr; return 0; }   // no allocation inside a capture: no alignment
    void *slab = nullptr;
    TD_CUDA(cudaMalloc(&slab, 256));
    g_sync_counter[{dev, st}] = static_cast<unsigned *>(slab);
    *out = static_cast<unsigned *>(slab);
    return 0;
}

// Budget of one tile-start wait (TDSCHA_TILE_SYNC_US, 0 disables the alignment).
static unsigned tile_sync_budget_ns() {
    static long long v = -1;
    if (v < 0) {
        const char *env = getenv("TDSCHA_TILE_SYNC_US");
        v = env ? std::max(0, atoi(env)) * 1000LL : 50000LL;
    }
    return (unsigned)v;
}

// Extents of the two operand buffers and the sub-problems of one contraction.
struct Problem {
    long long a_rows, a_cols, b_rows, b_cols;
    std::vector<GemmGroup> groups;
};

// A tile shape: orientation and the widest tile along the MMA's N side.
struct TileShape {
    bool swap = false;   // the 128-row side of a tile is B (output columns) instead of A (output rows)
    int cap = 256;       // columns of a tile at most
    int p_rows = BM;     // P rows of a tile (128 or 64)
};

// Width of the tiles that cover n columns in pieces of at most cap: equal pieces, a multiple of 16.
static int tile_width(int n, int cap) { return (int)round_up(ceil_div(n, ceil_div(n, cap)), 16); }

struct TilePlan {
    long long tiles = 0;
    int p_box = 128, q_box = 0, q_rows = 0, max_p = 1;
    double cycles = 0;   // estimated SM cycles of the launch
};

// Tiles, TMA boxes and estimated time of groups [g0, g1) with one tile shape.  The estimate (SM cycles
// of a k-block: the largest of its MMA time, its copy time and the ring's latency) only has to order
// the shapes; measured on this GPU with one tile per SM: an MMA instruction takes half a cycle per
// column but no less than 68 cycles for its 128 P rows (34 for 64), copies 60 B per cycle and SM.
static TilePlan plan_tiles(const Problem &pb, size_t g0, size_t g1, TileShape sh, int kelems, int nprod, int drain, int sms) {
    TilePlan pl;
    const int nops = nprod == 3 ? 2 : 1;
    int pmax = 1;
    for (size_t i = g0; i < g1; ++i) pmax = std::max(pmax, sh.swap ? pb.groups[i].N : pb.groups[i].M);
    pl.p_box = (int)std::min<long long>(sh.p_rows, round_up(pmax, 8));
    // one Q box height for every group: the least rows copied, fewer boxes on a tie
    double best = 1e300;
    for (int q = 16; q <= 256; q += 16) {
        double cost = 0;
        int rows_max = 0;
        for (size_t i = g0; i < g1 && rows_max <= 256; ++i) {
            const GemmGroup &G = pb.groups[i];
            const int nq = sh.swap ? G.M : G.N, np = sh.swap ? G.N : G.M;
            const int tn = tile_width(nq, sh.cap), boxes = ceil_div(tn, q);
            rows_max = std::max(rows_max, boxes * q);
            cost += (double)ceil_div(nq, tn) * ceil_div(np, sh.p_rows) * G.K * (boxes * q + 8.0 * boxes);
        }
        if (rows_max > 256) continue;
        if (cost < best) { best = cost; pl.q_box = q; pl.q_rows = rows_max; }
    }
    double total = 0, longest = 0;
    for (size_t i = g0; i < g1; ++i) {
        const GemmGroup &G = pb.groups[i];
        const int nq = sh.swap ? G.M : G.N, np = sh.swap ? G.N : G.M;
        const int tn = tile_width(nq, sh.cap);
        const int num_p = ceil_div(np, sh.p_rows), num_q = ceil_div(nq, tn), nkb = G.K / kelems;
        const double mma = 4.0 * nprod * std::max(tn * 0.5, sh.p_rows * 0.53);
        const double copy = nops * 128.0 * (pl.p_box + ceil_div(tn, pl.q_box) * pl.q_box) / 60.0;
        const double lat = 400.0 + 150.0 / drain;
        const double tile = nkb * std::max(mma, std::max(copy, lat)) + 1500.0 + (sh.swap ? 40.0 : 16.0) * tn;
        pl.tiles += (long long)num_p * num_q;
        pl.max_p = std::max(pl.max_p, num_p);
        total += tile * num_p * num_q;
        longest = std::max(longest, tile);
    }
    const double per_sm = total / sms, waves = (double)((pl.tiles + sms - 1) / sms) * (total / pl.tiles);
    pl.cycles = std::max(longest, 0.5 * (per_sm + std::max(per_sm, waves)));
    return pl;
}

// One tile shape of a contraction, ready to launch with a tile-group size.
struct Prepared {
    std::function<void(int)> launch;
    int num_p = 0;
    TileShape shape;
    long long tiles = 0;
};

template <int MAXC, bool TF32, int NPROD, bool SWAP, int KBYTES, bool WEIGHTS>
static int prepare_cfg(const GemmOperands &op, const WeightsOut *wo, const Problem &pb, size_t g0, size_t g1, TileShape sh, const TilePlan &pl, float *D,
                       long long ldd, cudaStream_t st, unsigned *err, unsigned *counter, int stall, int sms, Prepared *out) {
    CUtensorMap p_hi, p_lo, q_hi, q_lo;
    const int a_box = SWAP ? pl.q_box : pl.p_box, b_box = SWAP ? pl.p_box : pl.q_box;
    CUtensorMap *a_maps[2] = {SWAP ? &q_hi : &p_hi, SWAP ? &q_lo : &p_lo}, *b_maps[2] = {SWAP ? &p_hi : &q_hi, SWAP ? &p_lo : &q_lo};
    TD_TRY(make_map(a_maps[0], op.A_hi, TF32, pb.a_rows, pb.a_cols, op.lda, a_box, KBYTES));
    TD_TRY(make_map(b_maps[0], op.B_hi, TF32, pb.b_rows, pb.b_cols, op.ldb, b_box, KBYTES));
    if (NPROD == 3) {
        TD_TRY(make_map(a_maps[1], op.A_lo, TF32, pb.a_rows, pb.a_cols, op.lda, a_box, KBYTES));
        TD_TRY(make_map(b_maps[1], op.B_lo, TF32, pb.b_rows, pb.b_cols, op.ldb, b_box, KBYTES));
    } else {
        p_lo = p_hi;
        q_lo = q_hi;
    }
    constexpr int NOPS = NPROD == 3 ? 2 : 1;
    GroupTable gt{};
    gt.n = (int)(g1 - g0);
    gt.p_rows = sh.p_rows;
    gt.p_box = pl.p_box;
    gt.q_box = pl.q_box;
    gt.q_off = NOPS * sh.p_rows * KBYTES;
    gt.q_bytes = pl.q_rows * KBYTES;
    gt.stage_bytes = gt.q_off + NOPS * gt.q_bytes;
    const int staging = epi_staging(SWAP, WEIGHTS);
    gt.stages = std::min(MAX_STAGES, (SMEM_MAX - SMEM_FIXED - staging) / gt.stage_bytes);
    TD_CHECK(gt.stages >= 2, TDSCHA_EINVAL, "tc::gemm: tile of %d rows does not fit", pl.q_rows);
    const int smem = gt.stages * gt.stage_bytes + SMEM_FIXED + staging;
    long long tiles = 0;
    for (size_t i = g0; i < g1; ++i) {
        const GemmGroup &g = pb.groups[i];
        DevGroup &d = gt.g[i - g0];
        d.np = SWAP ? g.N : g.M;
        d.nq = SWAP ? g.M : g.N;
        d.K = g.K;
        d.p_row = SWAP ? g.b_row : g.a_row;
        d.p_k = SWAP ? g.b_k : g.a_k;
        d.q_row = SWAP ? g.a_row : g.b_row;
        d.q_k = SWAP ? g.a_k : g.b_k;
        d.d_off = g.d_off;
        if (WEIGHTS) {
            d.kw = wo->K[i];
            d.pw_k = d.qw_k = wo->col[i];
        }
        d.tn = tile_width(d.nq, sh.cap);
        d.num_p = ceil_div(d.np, sh.p_rows);
        d.num_q = ceil_div(d.nq, d.tn);
        d.tile0 = (int)tiles;
        tiles += (long long)d.num_p * d.num_q;
    }
    TD_CHECK(tiles < (1LL << 31), TDSCHA_EINVAL, "tc::gemm: %lld tiles exceed the schedule", tiles);
    gt.total_tiles = (int)tiles;
    constexpr auto kern = tc_gemm_kernel<MAXC, TF32, NPROD, SWAP, KBYTES, WEIGHTS>;
    TD_TRY(allow_smem<kern>(SMEM_MAX));
    const int drain = (op.drain_kb > 0 ? op.drain_kb : default_drain(NPROD)) * (128 / KBYTES);   // in stages
    const dim3 grid((unsigned)std::min<long long>(tiles, sms));
    const unsigned sync_ns = tile_sync_budget_ns();
    const int accumulate = op.accumulate ? 1 : 0;
    const unsigned long long wait_ns = g_wait_budget_ns.load();
    // Tile starts are aligned only where K is long: the panels of one tile then outgrow L2 and CTAs that
    // drift apart re-read them.  Below that the wait and its counter's memset only cost: [a|b] of 192
    // rows x 20000, K <= 2432: 1623 us aligned, 1564 us not; Z (K = 20032) the same either way.
    int k_max = 0;
    for (size_t i = g0; i < g1; ++i) k_max = std::max(k_max, pb.groups[i].K);
    unsigned *cnt = (sync_ns > 0 && counter && tiles > grid.x && k_max >= 32768) ? counter : nullptr;
    EpiArgs<WEIGHTS> ea{};
    if constexpr (WEIGHTS) {
        CUtensorMap *wa[2] = {SWAP ? &ea.q_hi : &ea.p_hi, SWAP ? &ea.q_lo : &ea.p_lo}, *wb[2] = {SWAP ? &ea.p_hi : &ea.q_hi, SWAP ? &ea.p_lo : &ea.q_lo};
        if (wo->ld > 0) {
            for (int x = 0; x < (NPROD == 3 ? 2 : 1); ++x) {
                TD_TRY(make_map(wa[x], x ? wo->A_lo : wo->A_hi, TF32, pb.a_rows, wo->ld, wo->ld, a_box, KBYTES));
                TD_TRY(make_map(wb[x], x ? wo->B_lo : wo->B_hi, TF32, pb.b_rows, wo->ld, wo->ld, b_box, KBYTES));
            }
        }
        ea.rho = wo->rho;
        ea.Nc = wo->Nc;
        ea.N2pc = wo->N2pc;
        ea.d4 = wo->d4;
        ea.f64 = wo->Nc % 4 != 0;
        ea.drain_w = default_drain(NPROD) * (128 / KBYTES);
        ea.cw_hi = wo->cw_hi; ea.cw_lo = wo->cw_lo; ea.ab_hi = wo->ab_hi; ea.ab_lo = wo->ab_lo;
    }
    out->num_p = pl.max_p;
    out->shape = sh;
    out->tiles = tiles;
    out->launch = [=](int gp) {
        if (cnt) cudaMemsetAsync(cnt, 0, sizeof(unsigned), st);
        kern<<<grid, NUM_THREADS, smem, st>>>(p_hi, p_lo, q_hi, q_lo, gt, drain, gp, D, ldd, err, cnt, sync_ns, accumulate, wait_ns,
                                              stall, ea);
    };
    return 0;
}

template <bool TF32, int NPROD>
static int prepare(const GemmOperands &op, const WeightsOut *wo, const Problem &pb, size_t g0, size_t g1, TileShape sh, const TilePlan &pl, float *D,
                   long long ldd, cudaStream_t st, unsigned *err, unsigned *counter, int stall, int sms, Prepared *out) {
    const int c = sh.cap <= 64 ? 64 : (sh.cap <= 128 ? 128 : 256);
    // half stages where full ones would leave the ring two deep
    constexpr int NOPS = NPROD == 3 ? 2 : 1;
    const int room = SMEM_MAX - SMEM_FIXED - epi_staging(sh.swap, wo != nullptr);
    const bool half = c == 256 && room / (NOPS * 128 * (sh.p_rows + pl.q_rows)) < 3;
#define TD_PREP(C, SW, KBY, W) prepare_cfg<C, TF32, NPROD, SW, KBY, W>(op, wo, pb, g0, g1, sh, pl, D, ldd, st, err, counter, stall, sms, out)
    if (wo) {
        if (sh.swap) return half ? TD_PREP(256, true, 64, true) : TD_PREP(256, true, 128, true);
        return half ? TD_PREP(256, false, 64, true) : TD_PREP(256, false, 128, true);
    }
    if (sh.swap) {
        if (half) return TD_PREP(256, true, 64, false);
        return c == 64 ? TD_PREP(64, true, 128, false) : (c == 128 ? TD_PREP(128, true, 128, false) : TD_PREP(256, true, 128, false));
    }
    if (half) return TD_PREP(256, false, 64, false);
    return c == 64 ? TD_PREP(64, false, 128, false) : (c == 128 ? TD_PREP(128, false, 128, false) : TD_PREP(256, false, 128, false));
#undef TD_PREP
}

// ---- tile-order autotuner ---------------------------------------------------------------------------
// On the first call for a (format, products, M, N, K) with many tiles (8 per SM and more) and more than
// 24 P tiles, the launcher times the tile-group sizes on the caller's stream and remembers the winner
// (with fewer P tiles every order is within 3 %: the class contractions of 768 to 3072 rows):
// the candidates run in turn, twice round (every run writes the same D), and each keeps its faster run,
// so that the clock drift of a power-capped GPU over the trials does not favour the candidates timed
// first.  TDSCHA_AUTOTUNE_VERBOSE=1 prints every trial and the choice to stderr.  Swapped launches,
// small problems, launches that accumulate or are being captured, and TDSCHA_AUTOTUNE=0 use the
// P-fastest order; TDSCHA_GROUP_M fixes the choice.
static std::map<TuneKey, int> g_tune_gp;

static int choose_order(const TuneKey &key, const Prepared &cfg, int sms, cudaStream_t st, bool allow_trials, int *gp_out) {
    *gp_out = cfg.shape.swap ? 1 : cfg.num_p;
    if (cfg.shape.swap) return 0;
    if (const char *env_gm = getenv("TDSCHA_GROUP_M")) {
        *gp_out = std::max(1, std::min(cfg.num_p, atoi(env_gm)));
        return 0;
    }
    if (cfg.tiles < 8LL * sms || cfg.num_p <= 24) return 0;
    {
        std::lock_guard<std::mutex> lock(g_tune_mutex);
        auto it = g_tune_gp.find(key);
        if (it != g_tune_gp.end()) { *gp_out = it->second; return 0; }
    }
    const char *env = getenv("TDSCHA_AUTOTUNE");
    if (!allow_trials || (env && atoi(env) == 0)) return 0;
    const char *env_v = getenv("TDSCHA_AUTOTUNE_VERBOSE");
    const bool verbose = env_v && atoi(env_v) == 1;
    std::vector<int> cands;
    for (int cand : {cfg.num_p, 48, 24, 12, 6})
        if (cand <= cfg.num_p && std::find(cands.begin(), cands.end(), cand) == cands.end()) cands.push_back(cand);
    cudaEvent_t e0, e1;
    TD_CUDA(cudaEventCreate(&e0));
    TD_CUDA(cudaEventCreate(&e1));
    std::vector<float> t_min(cands.size(), 1e30f);
    for (int round = 0; round < 2 && cands.size() > 1; ++round)
        for (size_t i = 0; i < cands.size(); ++i) {
            TD_CUDA(cudaEventRecord(e0, st));
            cfg.launch(cands[i]);
            TD_CUDA(cudaGetLastError());
            TD_CUDA(cudaEventRecord(e1, st));
            TD_CUDA(cudaEventSynchronize(e1));
            float ms = 0.f;
            TD_CUDA(cudaEventElapsedTime(&ms, e0, e1));
            t_min[i] = std::min(t_min[i], ms);
            if (verbose)
                fprintf(stderr, "[tc autotune] M=%d N=%d K=%d nprod=%d tile_n=%d group=%d round %d: %.3f ms\n", key.M, key.N, key.K,
                        key.nprod, cfg.shape.cap, cands[i], round, ms);
        }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    size_t bi = 0;
    for (size_t i = 1; i < cands.size(); ++i)
        if (t_min[i] < t_min[bi]) bi = i;
    if (verbose)
        fprintf(stderr, "[tc autotune] M=%d N=%d K=%d nprod=%d -> tile_n=%d group=%d\n", key.M, key.N, key.K, key.nprod,
                cfg.shape.cap, cands[bi]);
    std::lock_guard<std::mutex> lock(g_tune_mutex);
    g_tune_gp[key] = cands[bi];
    *gp_out = cands[bi];
    return 0;
}

// The tile shape with the least estimated time (plan_tiles), remembered per problem shape.
// TDSCHA_TILE_N (256 | 128 | 64) forces tiles of that many output columns with A on the 128-row side.
static std::map<std::pair<TuneKey, int>, std::pair<TileShape, TilePlan>> g_tune_shape;

static TileShape choose_shape(const Problem &pb, size_t g0, size_t g1, const TuneKey &key, int kelems, int nprod, int drain, int sms,
                              bool stall, TilePlan *plan) {
    TileShape best;
    const char *env = getenv("TDSCHA_TILE_N");
    if (env || stall) {   // abort-path test: the wide tile
        if (env && (atoi(env) == 128 || atoi(env) == 64)) best.cap = atoi(env);
        *plan = plan_tiles(pb, g0, g1, best, kelems, nprod, drain, sms);
        return best;
    }
    std::lock_guard<std::mutex> lock(g_tune_mutex);
    auto it = g_tune_shape.find({key, drain});
    if (it != g_tune_shape.end()) {
        *plan = it->second.second;
        return it->second.first;
    }
    plan->cycles = 1e300;
    for (int swap = 0; swap < 2; ++swap)
        for (int cap : {256, 192, 128, 96, 64, 48, 32, 16})
            for (int p_rows : {128, 64}) {
                const TileShape sh{swap != 0, cap, p_rows};
                const TilePlan pl = plan_tiles(pb, g0, g1, sh, kelems, nprod, drain, sms);
                if (pl.cycles < plan->cycles) { *plan = pl; best = sh; }
            }
    const char *env_v = getenv("TDSCHA_AUTOTUNE_VERBOSE");
    if (env_v && atoi(env_v) == 1)
        fprintf(stderr, "[tc shape] %zu groups, first M=%d N=%d K=%d: %s cap %d, %d P rows, q box %d, %lld tiles, %.0f cycles\n", g1 - g0,
                pb.groups[g0].M, pb.groups[g0].N, pb.groups[g0].K, best.swap ? "swapped" : "normal", best.cap, best.p_rows,
                plan->q_box, plan->tiles, plan->cycles);
    g_tune_shape[{key, drain}] = {best, *plan};
    return best;
}

template <bool TF32, int NPROD>
static int launch_tuned(const GemmOperands &op, const WeightsOut *wo, const Problem &pb, float *D, long long ldd, cudaStream_t st, unsigned *err) {
    int dev = 0, sms = 148;
    TD_CUDA(cudaGetDevice(&dev));
    TD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    TD_CUDA(cudaStreamIsCapturing(st, &cap));
    const bool capturing = cap != cudaStreamCaptureStatusNone;
    unsigned *counter = nullptr;
    if (op.tile_sync && tile_sync_budget_ns() > 0) TD_TRY(tile_sync_counter(dev, st, capturing, &counter));
    const int stall = g_stall_next.exchange(0);
    const int drain = op.drain_kb > 0 ? op.drain_kb : default_drain(NPROD);
    for (size_t g0 = 0; g0 < pb.groups.size(); g0 += MAX_GROUPS) {
        const size_t g1 = std::min(pb.groups.size(), g0 + MAX_GROUPS);
        // tuning key: the one problem's shape, or the groups' shapes hashed (FNV-1a)
        TuneKey key{TF32 ? 1 : 0, NPROD, pb.groups[g0].M, pb.groups[g0].N, pb.groups[g0].K, dev, 0ull};
        if (g1 - g0 > 1) {
            key.shape = 1469598103934665603ull;
            for (size_t i = g0; i < g1; ++i)
                for (long long v : {(long long)pb.groups[i].M, (long long)pb.groups[i].N, (long long)pb.groups[i].K}) {
                    key.shape ^= (unsigned long long)v;
                    key.shape *= 1099511628211ull;
                }
            key.M = (int)(g1 - g0);
        }
        TilePlan pl;
        const TileShape sh = choose_shape(pb, g0, g1, key, KBlock<TF32, 128>::ELEMS, NPROD, drain, sms, stall != 0, &pl);
        if (op.planned) TD_TRY((*op.planned)((int)std::min<long long>(pl.tiles, sms)));
        Prepared cfg;
        TD_TRY((prepare<TF32, NPROD>(op, wo, pb, g0, g1, sh, pl, D, ldd, st, err, counter, stall, sms, &cfg)));
        int gp = cfg.num_p;
        // trial runs write D, so an accumulating launch only reuses a choice tuned earlier (and a launch
        // being captured into a CUDA graph runs nothing, so it cannot time trials); the abort-path
        // test runs one launch without trials
        if (!stall) TD_TRY(choose_order(key, cfg, sms, st, !op.accumulate && !capturing, &gp));
        cfg.launch(gp);
        TD_CUDA(cudaGetLastError());
    }
    return 0;
}

void set_wait_budget_ns(unsigned long long ns) { g_wait_budget_ns.store(ns); }
unsigned long long wait_budget_ns() { return g_wait_budget_ns.load(); }
void stall_next_launch() { g_stall_next.store(1); }

static int dispatch(const GemmOperands &op, const WeightsOut *wo, const Problem &pb, float *D, long long ldd, cudaStream_t st,
                    unsigned *err) {
    if (op.fmt == FMT_TF32) {
        if (op.nprod == 3) return launch_tuned<true, 3>(op, wo, pb, D, ldd, st, err);
        return launch_tuned<true, 1>(op, wo, pb, D, ldd, st, err);
    }
    if (op.nprod == 3) return launch_tuned<false, 3>(op, wo, pb, D, ldd, st, err);
    return launch_tuned<false, 1>(op, wo, pb, D, ldd, st, err);
}

int gemm(const GemmOperands &op, int M, int N, int K, float *D, long long ldd, cudaStream_t st, unsigned *err) {
    TD_CHECK(M > 0 && N > 0 && K > 0, TDSCHA_EINVAL, "tc::gemm: empty problem %d x %d x %d", M, N, K);
    const bool tf32 = op.fmt == FMT_TF32;
    TD_CHECK(op.fmt == FMT_TF32 || op.fmt == FMT_BF16, TDSCHA_EINVAL, "tc::gemm: operand format must be bf16 or tf32");
    TD_CHECK(K % (tf32 ? 32 : 64) == 0, TDSCHA_EINVAL, "tc::gemm: K=%d not a multiple of the 128-byte K block", K);
    TD_CHECK(op.nprod == 1 || op.nprod == 3, TDSCHA_EINVAL, "tc::gemm: nprod must be 1 or 3");
    constexpr long long LD_MAX = 1LL << 31;
    TD_CHECK(op.lda >= K && op.ldb >= K && ldd >= N && op.lda < LD_MAX && op.ldb < LD_MAX && ldd < LD_MAX, TDSCHA_EINVAL,
             "tc::gemm: leading dimensions lda=%lld ldb=%lld ldd=%lld inconsistent with K=%d N=%d", op.lda, op.ldb, ldd, K, N);
    TD_CHECK(op.A_hi && op.B_hi && D && (op.nprod == 1 || (op.A_lo && op.B_lo)), TDSCHA_EINVAL, "tc::gemm: NULL operand");
    Problem pb{M, K, N, K, {GemmGroup{M, N, K, 0, 0, 0, 0, 0}}};
    return dispatch(op, nullptr, pb, D, ldd, st, err);
}

static int check_groups(const GemmOperands &op, long long a_rows, long long a_cols, long long b_rows, long long b_cols,
                        const GemmGroup *groups, int n_groups, long long ldd, Problem *out) {
    TD_CHECK(n_groups > 0 && groups, TDSCHA_EINVAL, "tc::gemm_grouped: no groups");
    const bool tf32 = op.fmt == FMT_TF32;
    TD_CHECK(op.fmt == FMT_TF32 || op.fmt == FMT_BF16, TDSCHA_EINVAL, "tc::gemm_grouped: operand format must be bf16 or tf32");
    TD_CHECK(op.nprod == 1 || op.nprod == 3, TDSCHA_EINVAL, "tc::gemm_grouped: nprod must be 1 or 3");
    const int kblk = tf32 ? 32 : 64;
    constexpr long long LD_MAX = 1LL << 31;
    TD_CHECK(op.lda >= a_cols && op.ldb >= b_cols && op.lda < LD_MAX && op.ldb < LD_MAX && ldd < LD_MAX && a_rows < LD_MAX &&
                 b_rows < LD_MAX && a_cols < LD_MAX && b_cols < LD_MAX,
             TDSCHA_EINVAL, "tc::gemm_grouped: operand extents inconsistent with their leading dimensions");
    TD_CHECK(op.A_hi && op.B_hi && (op.nprod == 1 || (op.A_lo && op.B_lo)), TDSCHA_EINVAL, "tc::gemm_grouped: NULL operand");
    Problem &pb = *out;
    pb = Problem{a_rows, a_cols, b_rows, b_cols, {}};
    for (int i = 0; i < n_groups; ++i) {
        const GemmGroup &g = groups[i];
        TD_CHECK(g.M > 0 && g.N > 0 && g.K > 0 && g.K % kblk == 0 && g.a_k % kblk == 0 && g.b_k % kblk == 0, TDSCHA_EINVAL,
                 "tc::gemm_grouped: group %d: M=%d N=%d K=%d a_k=%d b_k=%d (K and offsets multiples of %d)", i, g.M, g.N, g.K,
                 g.a_k, g.b_k, kblk);
        TD_CHECK(g.a_row >= 0 && g.b_row >= 0 && g.a_row < a_rows && g.b_row < b_rows && g.a_k + (long long)g.K <= a_cols &&
                     g.b_k + (long long)g.K <= b_cols && g.N <= ldd && g.d_off >= 0,
                 TDSCHA_EINVAL, "tc::gemm_grouped: group %d outside its operands", i);
        pb.groups.push_back(g);
    }
    return 0;
}

int gemm_grouped(const GemmOperands &op, long long a_rows, long long a_cols, long long b_rows, long long b_cols,
                 const GemmGroup *groups, int n_groups, float *D, long long ldd, cudaStream_t st, unsigned *err) {
    TD_CHECK(D != nullptr, TDSCHA_EINVAL, "tc::gemm_grouped: NULL output");
    Problem pb;
    TD_TRY(check_groups(op, a_rows, a_cols, b_rows, b_cols, groups, n_groups, ldd, &pb));
    return dispatch(op, nullptr, pb, D, ldd, st, err);
}

bool weights_fit(Format fmt, int nprod, int K) {
    return ceil_div(K, (fmt == FMT_TF32 ? 32 : 64) * default_drain(nprod)) <= 2;
}

int gemm_grouped_weights(const GemmOperands &op, long long a_rows, long long a_cols, long long b_rows, long long b_cols,
                         const GemmGroup *groups, int n_groups, const WeightsOut &wo, cudaStream_t st, unsigned *err) {
    Problem pb;
    TD_TRY(check_groups(op, a_rows, a_cols, b_rows, b_cols, groups, n_groups, wo.N2pc, &pb));
    TD_CHECK(wo.rho && wo.cw_hi && wo.ab_hi && (op.nprod == 1 || (wo.cw_lo && wo.ab_lo)) && (int)wo.K.size() == n_groups &&
                 (int)wo.col.size() == n_groups && b_rows == 2LL * wo.Nc && wo.N2pc >= 2 * wo.Nc,
             TDSCHA_EINVAL, "tc::gemm_grouped_weights: bad arguments");
    const int kblk = op.fmt == FMT_TF32 ? 32 : 64;
    for (int i = 0; i < n_groups; ++i) {
        TD_CHECK(groups[i].N == b_rows && groups[i].b_row == 0 && wo.K[i] >= 0 && wo.K[i] % kblk == 0 && wo.col[i] % kblk == 0 &&
                     wo.col[i] + (long long)wo.K[i] <= wo.ld && weights_fit(op.fmt, op.nprod, wo.K[i]),
                 TDSCHA_EINVAL, "tc::gemm_grouped_weights: group %d: K=%d at column %d of %lld", i, wo.K[i], wo.col[i], wo.ld);
        TD_CHECK(wo.K[i] == 0 || (wo.A_hi && wo.B_hi && (op.nprod == 1 || (wo.A_lo && wo.B_lo))), TDSCHA_EINVAL,
                 "tc::gemm_grouped_weights: NULL [c|d] operand");
    }
    return dispatch(op, &wo, pb, nullptr, wo.N2pc, st, err);
}

}  // namespace tc
}  // namespace tdscha
