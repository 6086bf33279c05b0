// Products of one to eight tokens of 4-bit matrices (Q4_K, the repacked MLX-4) and Q8_0 on the fifth-generation tensor cores: the role of dmv_* and dmvk_*
// in the reference (src/cuda_decode.cu:139-232). The arithmetic is that of gemv_mma.cuh: the packed integers of the weights times
// signed digits of the activations (split.cuh: 23 to 24 bits of every value), summed exactly, scaled by 32 values in integers (Q4_K) or by
// 64 in f32 (MLX-4). Here tcgen05.mma.kind::i8 makes the sums: A = 128 weight rows, a byte a weight, in tensor memory; B = the digits in
// shared memory (three columns a token), 32 k an instruction, summed per 32 (Q4_K) or per 64 (MLX-4).
//
// A cluster of four CTAs takes tiles of 128 rows, CTA q the blocks q n / 4 .. of K, so the order of a row's sum depends on K alone: a
// row shard and every row of a step of several tokens have the bits of the one-token product. A CTA:
//   warp 0        : copies packed rows (128 x 144 bytes a block of 256 k) into a ring, filled before the kernel waits for the one ahead.
//   warps 2 .. 17 : four sets of four, a thread a row; set s takes the blocks s, s + 4, .. of those that the CTA has of all its tiles: nibbles to
//                   bytes in tensor memory, the instructions, the sums back and times the scales. At the end of a tile its sums go to the CTA of
//                   the cluster that owns the rows.
//   warp 1        : adds the sixteen sums of its rows in pairs, applies the norm's factor and the output mode, and stores.
// All but warp 0 split the CTA's part of the activations first (an RMS norm's weights multiply before the split, its factor the results).
// Five to eight tokens: every other cluster has those from the fifth on, and the second reading of the weights comes from L2.
// Q8_0 rows are bytes already: the instructions read them where the copies put them (two swizzled tiles of 128 k and the rows' scales), and a set's warps
// only scale the sums (f32, per 32). Eight tokens are 32 columns then: read twice, the bytes would pass at L2's rate.
//
// What bounds it: HBM on large matrices, the start on small ones. The form on mma.sync (gemv_mma.cu) was bound by instructions: 393 of a warp
// for 4096 weights (Q4_K 14336 x 4096, one token, ncu, everything counted); here it is 225, of which the bytes, the sums and the scales are about
// 110. Of the 4.7 us of 4096 x 4096, 0.5 pass before the first copy is issued, 1.5 until activations and weights are there, and 2 between them and
// the result, most of it the first fetch of each line of code: hence short code, no divisions, a pass of the results' loop that stores nothing. Four
// sets and the whole of tensor memory: two sets in half of an SM (two CTAs) left 4096 x 14336, four tokens, at 21 us.
// One launch after another in a stream, us, one / two / four / eight tokens, on mma.sync and here:
//   Q4_K  4096 x 4096    5.2 / 8.8 / 11.0 / 16.1   5.1 / 5.5 / 6.1 / 7.9
//         4096 x 14336  12.8 / 21.7 / 25.7 / 41.1  9.6 / 11.2 / 14.2 / 19.6
//         32064 x 4096  17.7 / 24.8 / 27.0 / 49.8  16.0 / 17.2 / 19.0 / 32.8
//   MLX-4 4096 x 4096    4.9 / 8.6 / 9.8 / 14.9    5.2 / 5.5 / 6.0 / 7.7
//         4096 x 14336  11.7 / 20.3 / 23.8 / 36.9  9.5 / 11.3 / 13.5 / 18.3
//         32064 x 4096  15.9 / 22.8 / 24.9 / 45.6  15.9 / 16.7 / 18.5 / 31.8
//   Q8_0  4096 x 4096    6.3 / 8.7 / 9.6 / 16.9    5.2 / 5.6 / 8.0 / 9.2
//         4096 x 14336  15.0 / 24.3 / 28.4 / 42.1  13.0 / 14.6 / 16.2 / 24.5
//         32064 x 4096  23.9 / 27.0 / 28.1 / 54.5  23.3 / 24.6 / 24.6 / 28.0
// (6144 x 4096, MLX-4, one token: 5.9 and 6.3: its 48 tiles take two rounds of 24 clusters. In a graph 4096 x 4096 takes 4.5 and 4.4. K of 1024 and
// less: gemv_tc_supports.)
// Largest error of a result against 64 bits, in parts of the row's norm, N(0, 1) activations, K = 1024 / 4096 / 14336:
// Q4_K 1.60 / 1.70 / 1.71e-7 on mma.sync, 1.60 / 1.65 / 1.66e-7 here; MLX-4, unsigned there, 1.78 / 2.07 / 2.39e-7 and 1.57 / 1.65 / 1.59e-7;
// Q8_0 1.67 / 1.72 / 1.79e-7 and 1.67 / 1.69 / 1.73e-7.
#include <cuda.h>

#include <algorithm>
#include <climits>
#include <map>
#include <mutex>
#include <tuple>

#include "gemm_wt.h"
#include "split.cuh"
#include "tcgen05.cuh"

namespace b2 {

namespace {

constexpr int GT_CTAS = 4, GT_ROWS = 128, GT_SETS = 4, GT_WARPS = 2 + 4 * GT_SETS, GT_THREADS = GT_WARPS * 32;
constexpr int GT_MOST_SLOTS = 8, GT_TOKENS = 4, GT_MOST_JOBS = GEMV_TC_JOBS;
__host__ __device__ constexpr uint32_t gt_raw(int fmt) { return GT_ROWS * (fmt == B2_FMT_Q8_0 ? 272 : 144); }  // a slot: a block of 256 k of 128 rows
constexpr uint32_t GT_TMEM_COLS = 512, GT_SET_COLS = 128;  // of a set: 64 of weights, 64 of sums
constexpr uint32_t GT_AM = 0, GT_DM = 16, GT_D = 64;       // (the minimums and their sums lie where weights were)

struct GtArgs {
    const float* x;
    size_t x_stride;
    const float* nw;
    float pre;
    int norm;
    float eps;
    const uint8_t* rec;
    size_t rec_stride;
    float* y;
    size_t y_stride;
    const float* gate;
    size_t gate_stride;
    int fast, mode, T, two, n_in, tiles, rounds, slots, zero;  // two: groups of four tokens; rounds: tiles a cluster
    size_t n_out;
    uint32_t b_off, min_off, sum_off, xs_off;  // shared memory
    uint32_t* status;
};

// The matrices: one, a pair, or up to GT_MOST_JOBS with results of their own (JOBS), whose tiles follow one another.
template <bool JOBS, bool Q8>
struct GtMats {
    CUtensorMap m[Q8 ? 4 : 2];  // (Q8_0: of bytes, then of scales)
};
template <>
struct GtMats<true, false> {
    CUtensorMap m[GT_MOST_JOBS];
    float* y[GT_MOST_JOBS];
    size_t n_out[GT_MOST_JOBS];
    int first[GT_MOST_JOBS];  // tile; behind the last matrix: no tile
};

template <int TP>
struct __align__(16) GtShared {
    float in[2][GT_SETS * GT_CTAS][32][TP];   // tiles in turn: a set's sums of this CTA's 32 rows
    float ssq_in[GT_CTAS][TP == 8 ? 8 : GT_TOKENS];  // the parts' sums of squares
    // A set's copies have barriers of their own, in the order of its blocks: a slot passes from set to set, and one that waited on a slot's barrier
    // could be two uses ahead of it, where a parity says nothing. (At most GT_MOST_SLOTS blocks are in flight, so eight are enough.)
    uint64_t raw_full[GT_SETS][GT_MOST_SLOTS], raw_empty[GT_MOST_SLOTS];
    uint64_t d_full[GT_SETS];
    uint64_t in_full[2], in_free[GT_CTAS][2], ssq_full;  // in_free: CTA w's places are free again
    uint32_t tmem_base;
    volatile uint32_t abort_flag;
};

// CLUSTER: what the barrier counts comes from the cluster's other CTAs.
template <bool CLUSTER = false, class Sh>
__device__ __forceinline__ bool gt_wait(uint64_t* bar, uint32_t parity, Sh* sh, uint32_t* status, bool heed_abort = true) {
    auto test = [&] { return CLUSTER ? mbar_try_wait_cluster(bar, parity) : mbar_try_wait(bar, parity); };
    if (test()) return true;
    const long long t0 = clock64();
    for (uint32_t spin = 1;; spin++) {
        if (test()) return true;
        if ((spin & 255) == 0) {
            if (heed_abort && sh->abort_flag) return false;
            if (clock64() - t0 > WAIT_LIMIT_CYCLES) {
                *(volatile uint32_t*)status = 2u;  // (may be the host's memory)
                __threadfence_system();
                sh->abort_flag = 1;
                return false;
            }
        }
    }
}
__device__ __forceinline__ void gt_mma(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, int add) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
        "r"(a), "l"(bdesc), "r"(idesc), "r"(add)
        : "memory");
}
__device__ __forceinline__ void gt_mma_ss(uint32_t d, uint64_t adesc, uint64_t bdesc, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(0)
        : "memory");
}
__device__ __forceinline__ void gt_st32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, "
        "%21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]),
        "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]),
        "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
__device__ __forceinline__ void gt_st2(uint32_t taddr, uint32_t a, uint32_t b) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(taddr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void gt_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void gt_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void gt_ld(uint32_t taddr, int (&v)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(taddr));
}
__device__ __forceinline__ void gt_ld(uint32_t taddr, int (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr));
}
__device__ __forceinline__ void gt_ld(uint32_t taddr, int (&v)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
                   "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(taddr));
}
__device__ __forceinline__ void gt_ld(uint32_t taddr, int (&v)[24]) {
    gt_ld(taddr, *(int(*)[16]) & v[0]);
    gt_ld(taddr + 16, *(int(*)[8]) & v[16]);
}
// Into a CTA of the cluster, counted on its barrier.
__device__ __forceinline__ void gt_send(uint32_t a, const float (&v)[1], uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(a), "f"(v[0]), "r"(bar) : "memory");
}
__device__ __forceinline__ void gt_send(uint32_t a, const float (&v)[2], uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(a), "f"(v[0]), "f"(v[1]), "r"(bar) : "memory");
}
__device__ __forceinline__ void gt_send(uint32_t a, const float (&v)[4], uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(a), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void gt_send(uint32_t a, const float (&v)[8], uint32_t bar) {
    const float lo[4] = {v[0], v[1], v[2], v[3]}, hi[4] = {v[4], v[5], v[6], v[7]};
    gt_send(a, lo, bar);
    gt_send(a + 16, hi, bar);
}
__device__ __forceinline__ void gt_arrive(uint32_t cluster_bar) { asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory"); }
__device__ __forceinline__ float gt_half(uint32_t w, int hi) { return __half2float(__ushort_as_half((unsigned short)(hi ? w >> 16 : w & 0xffffu))); }
// Byte k of row n in a 128-byte swizzled tile of 16 rows.
__device__ __forceinline__ uint32_t gt_at(uint32_t n, uint32_t k) { return (n >> 3) * 1024 + (n & 7) * 128 + (((k >> 4) ^ (n & 7)) << 4) + (k & 15); }
__device__ __forceinline__ float gt_silu(float a) { return a / (1.0f + __expf(-a)); }
__device__ __forceinline__ float gt_gelu(float a) { return 0.5f * a * (1.0f + tanhf(0.7978845608f * (a + 0.044715f * a * a * a))); }

template <int FMT, bool PAIR, int TP, bool JOBS>
__global__ void __launch_bounds__(GT_THREADS, 1)
gemv_tc_kernel(const __grid_constant__ GtMats<JOBS, FMT == B2_FMT_Q8_0> mats, const __grid_constant__ GtArgs a) {
    constexpr bool MLX = FMT == B2_FMT_MLX4, Q8 = FMT == B2_FMT_Q8_0;
    constexpr int MOST = TP == 8 ? 8 : GT_TOKENS;     // tokens of a cluster
    constexpr uint32_t NB = TP == 8 ? 32 : 16;        // columns of an instruction
    constexpr uint32_t RAW = gt_raw(FMT);
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    extern __shared__ uint8_t smem_raw[];
    uint8_t* const smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ GtShared<TP> shared;
    GtShared<TP>* const sh = &shared;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // (five to eight tokens: every other cluster has those from the fifth on)
    const int rank = (int)cluster_rank(), t0 = a.two ? (int)(blockIdx.x / GT_CTAS & 1) * GT_TOKENS : 0;
    const int cluster = (int)(blockIdx.x / GT_CTAS) >> a.two, clusters = (int)(gridDim.x / GT_CTAS) >> a.two;
    const int T = min(a.T - t0, MOST);
    const int nb = a.n_in / 256, b0 = rank * nb / GT_CTAS, nbq = (rank + 1) * nb / GT_CTAS - b0;  // this CTA's blocks of K
    const int my_tiles = a.rounds - (cluster + (a.rounds - 1) * clusters >= a.tiles);  // (no divisions here and below: they are a third of the time to the first copy)
    const int total = my_tiles * nbq;  // blocks to copy
    constexpr uint32_t IN_BYTES = GT_SETS * GT_CTAS * 32 * TP * 4;
    if (warp == 0) {
        if (lane < (JOBS ? GT_MOST_JOBS : Q8 ? 4 : PAIR ? 2 : 1)) asm volatile("prefetch.tensormap [%0];" ::"l"(&mats.m[lane]) : "memory");
        mbar_init(&sh->raw_full[lane / GT_MOST_SLOTS][lane % GT_MOST_SLOTS], 1);
        if (lane < GT_MOST_SLOTS) mbar_init(&sh->raw_empty[lane], 4);
        if (lane < GT_SETS) mbar_init(&sh->d_full[lane], 1);
        if (lane < 2 * GT_CTAS) mbar_init(&sh->in_free[lane >> 1][lane & 1], 1);
        if (lane < 2) mbar_init(&sh->in_full[lane], 1);
        if (lane == 2) mbar_init(&sh->ssq_full, 1);
        if (lane == 3) sh->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (lane < 2) mbar_arrive_expect_tx(&sh->in_full[lane], IN_BYTES);
        if (lane == 2) mbar_arrive_expect_tx(&sh->ssq_full, GT_CTAS * MOST * 4);
        __syncwarp();
    } else if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh->tmem_base)), "r"(GT_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        tc_fence_before();
    }
    auto job_of = [&](int tile) {
        int j = 0;
        if constexpr (JOBS)
#pragma unroll
            for (int k = 1; k < GT_MOST_JOBS; k++) j += tile >= mats.first[k];
        return j;
    };
    // warp 0: the next block goes to slot c_slot: block c_blk of tile c_tile
    int c_slot = 0, c_blk = 0, c_tile = cluster, c_n = 0;
    auto full_of = [&](int n) { return &sh->raw_full[n & 3][(n >> 2) & (GT_MOST_SLOTS - 1)]; };  // block n: set n % 4, its n / 4th
    auto full_parity = [&](int n) { return (uint32_t)(n >> 5) & 1; };
    static_assert(GT_SETS == 4 && GT_MOST_SLOTS == 8, "full_of, full_parity");
    auto copy = [&] {
        if (elect_one()) {
            const int x = (b0 + c_blk) * (Q8 ? 256 : 144);
            uint8_t* dst = smem + (size_t)c_slot * RAW;
            uint64_t* const full = full_of(c_n);
            mbar_arrive_expect_tx(full, RAW);
            if constexpr (Q8) {  // two swizzled tiles of 128 k and the rows' eight scales; a pair's matrices 64 rows each
#pragma unroll
                for (int u = 0; u < (PAIR ? 2 : 1); u++) {
                    const int y = c_tile * (PAIR ? 64 : GT_ROWS);
                    tma_load_2d(dst + u * 64 * 128, &mats.m[u], full, x, y);
                    tma_load_2d(dst + GT_ROWS * 128 + u * 64 * 128, &mats.m[u], full, x + 128, y);
                    tma_load_2d(dst + GT_ROWS * 256 + u * 64 * 16, &mats.m[2 + u], full, (b0 + c_blk) * 8, y);
                }
            } else if constexpr (PAIR) {  // 64 rows of either matrix
                tma_load_2d(dst, &mats.m[0], full, x, c_tile * 64);
                tma_load_2d(dst + 64 * 144, &mats.m[1], full, x, c_tile * 64);
            } else if constexpr (JOBS) {
                const int j = job_of(c_tile);
                tma_load_2d(dst, &mats.m[j], full, x, (c_tile - mats.first[j]) * GT_ROWS);
            } else {
                tma_load_2d(dst, &mats.m[0], full, x, c_tile * GT_ROWS);
            }
        }
        __syncwarp();
        c_n++;
        if (++c_slot == a.slots) c_slot = 0;
        if (++c_blk == nbq) {
            c_blk = 0;
            c_tile += clusters;
        }
    };
    const int first = min(total, a.slots);
    if (warp == 0)
        for (int n = 0; n < first; n++) copy();  // (the weights do not wait for the kernel ahead)
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");

    // ---------------- this part's activations: digits, scales, chunk sums ----------------
    uint8_t* const b_s = smem + a.b_off;
    uint8_t* const min_s = smem + a.min_off;
    float* const sum_s = (float*)(smem + a.sum_off);  // MLX: sums of 64 times the block's scale [block][TP][4]
    float* const xs_s = (float*)(smem + a.xs_off);    // [block][TP]
    float* const ssq_s = xs_s + nbq * TP;
    const int items = nbq * T;
    auto block_of = [&](int i) {  // i / T (i < 512: times ceil(2^16 / T) where T is no power of two)
        if constexpr (TP == 1) return i;
        if constexpr (TP == 2) return i >> 1;
        return T == 4   ? i >> 2
               : T == 3 ? (i * 21846) >> 16
               : T == 2 ? i >> 1
               : T == 1 ? i
               : T == 8 ? i >> 3
               : T == 7 ? (i * 9363) >> 16
               : T == 6 ? (i * 10923) >> 16
                        : (i * 13108) >> 16;
    };
    auto load = [&](int i) {
        const int lb = block_of(i), tk = i - lb * T, blk = b0 + lb;
        return split_load(a.x + (size_t)(t0 + tk) * a.x_stride + (size_t)blk * 256, a.nw ? a.nw + (size_t)blk * 256 : nullptr, 256, lane);
    };
    const int w0 = warp == 1 ? GT_WARPS - 2 : warp - 2;  // (warp 0 is busy with the copies)
    SplitIn next;
    if (warp > 0 && !a.rec && w0 < items) next = load(w0);
    for (int i = warp > 0 ? w0 : items; i < items; i += GT_WARPS - 1) {
        const int lb = block_of(i), tk = i - lb * T, blk = b0 + lb;
        SplitDigits<3> d;
        int s;  // lanes 0 .. 7: the sum of chunk `lane`
        if (a.rec) {
            const uint8_t* r = a.rec + (size_t)(t0 + tk) * a.rec_stride + (size_t)blk * SPLIT_DIGITS;
            const uint8_t* aux = a.rec + (size_t)(t0 + tk) * a.rec_stride + (size_t)nb * SPLIT_DIGITS + (size_t)blk * SPLIT_AUX;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                int pair, in16;
                split_digit_at(h, lane, pair, in16);
#pragma unroll
                for (int p = 0; p < 3; p++) d.d[h][p] = __ldcg((const uint32_t*)(r + pair * 192 + p * 64 + in16));
            }
            const float2 h0 = __ldcg((const float2*)aux);
            d.xs = h0.x;
            d.ssq = h0.y;
            s = __ldcg((const int*)(aux + 16) + (lane & 7));
        } else {
            const SplitIn in = next;
            if (i + GT_WARPS - 1 < items) next = load(i + GT_WARPS - 1);
            d = split_digits<3>(in, a.pre, a.fast);
            const int from = (lane & 3) * 8, sl = __shfl_sync(0xffffffffu, d.s[0], from), su = __shfl_sync(0xffffffffu, d.s[1], from);
            s = (lane & 4) ? su : sl;
        }
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int p = 0; p < 3; p++) *(uint32_t*)(b_s + lb * (NB * 256) + h * (NB * 128) + gt_at(3 * tk + p, 4 * lane)) = d.d[h][p];
        if constexpr (Q8) {  // (no offsets: the sums are not needed)
        } else if constexpr (MLX) {
            const int o = __shfl_xor_sync(0xffffffffu, s, 1);
            if (lane < 8 && (lane & 1) == 0) sum_s[(lb * TP + tk) * 4 + (lane >> 1)] = d.xs * (float)(s + o);
        } else {  // four signed digits (|s| < 2^28), eight bytes of a block's 32; the others are zeros
            const uint32_t v = lane < 8 ? (uint32_t)(s + (int)0x80808080u) ^ 0x80808080u : 0u;
#pragma unroll
            for (int p = 0; p < 4; p++) min_s[(lb >> 2) * 2048 + gt_at(4 * tk + p, 32 * (lb & 3) + lane)] = (uint8_t)(v >> (8 * p));
        }
        if (lane == 0) {
            xs_s[lb * TP + tk] = d.xs;
            ssq_s[lb * TP + tk] = d.ssq;
        }
    }
    fence_proxy_async();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh->tmem_base;

    if (warp > 1) {
        // ---------------- bytes in, sums out ----------------
        constexpr uint32_t idesc = (2u << 4) | (MLX || Q8 ? 1u << 7 : 0u) | (1u << 10) | ((NB >> 3) << 17) | ((128u >> 4) << 24);  // s32 = u8 or s8 x s8, 128 x 16 or 32
        const int set = (warp - 2) >> 2, w = warp & 3, r = 32 * w + lane;
        const uint32_t at = tmem + ((uint32_t)(32 * w) << 16) + set * GT_SET_COLS;
        const uint32_t base = tmem + set * GT_SET_COLS;
        const uint64_t bd = smem_desc_sw128(smem_u32(b_s)), md = smem_desc_sw128(smem_u32(min_s));
        uint32_t phase = 0;
        int s = 0, at_n = 0;  // the slot of block at_n
        bool ok = true;
        // How often the set's warps have met, MEETS times a block. (MLX-4 works it out where a wait gives up: counted, four tokens took 1 % longer.)
        int met = 0;
        constexpr int MEETS = MLX || (Q8 && NB == 16) ? 1 : 2;
        for (int i = 0; i < my_tiles && ok; i++) {
            float acc[TP], low[TP];  // the third digit's share, the others'
#pragma unroll
            for (int t = 0; t < TP; t++) acc[t] = low[t] = 0.0f;
            // Block n of the CTA belongs to set n % 4, so that short parts of K keep all four busy (28672 x 2048, one token, Q4_K: by the block in the tile
            // 12.5 us, this way 10.3); the sums go by the block in the tile.
            const int share = (set - i * nbq) & 3;
            for (int lb = share; lb < nbq && ok; lb += GT_SETS) {
                const int n = i * nbq + lb;
                for (s += n - at_n, at_n = n; s >= a.slots;) s -= a.slots;
                ok = __all_sync(0xffffffffu, gt_wait(full_of(n), full_parity(n), sh, a.status));
                if (!ok) {
                    if constexpr (MLX) met = n >> 2;
                    break;
                }
                const uint8_t* const slot = smem + (size_t)s * RAW;
                const uint4 hd = *(const uint4*)(slot + (Q8 ? GT_ROWS * 256 + r * 16 : r * 144));  // (Q8_0: eight scales)
                uint4 q[8];
                if constexpr (!Q8) {
                    uint32_t words = hd.x;
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        q[k] = *(const uint4*)(slot + r * 144 + 16 + 16 * k);
                        words |= q[k].x;
                    }
                    release_raw(&sh->raw_empty[s], words, a.zero, lane);
                }
                int p[TP][3];
                float f[TP], fl[TP];
#pragma unroll
                for (int t = 0; t < TP; t++) {
                    p[t][0] = p[t][1] = p[t][2] = 0;
                    f[t] = fl[t] = 0.0f;
                }
                constexpr uint32_t LOW = 0x0F0F0F0Fu;
                auto expand = [&](int h) {  // 128 values
                    uint32_t o[32];
#pragma unroll
                    for (int j = 0; j < 2; j++) {  // 64 values: the low nibbles of 32 bytes, the high ones
                        const uint32_t v[8] = {q[4 * h + 2 * j].x, q[4 * h + 2 * j].y, q[4 * h + 2 * j].z, q[4 * h + 2 * j].w,
                                               q[4 * h + 2 * j + 1].x, q[4 * h + 2 * j + 1].y, q[4 * h + 2 * j + 1].z, q[4 * h + 2 * j + 1].w};
#pragma unroll
                        for (int k = 0; k < 8; k++) {
                            // MLX: 16 (n - 8) as signed bytes
                            o[16 * j + k] = MLX ? ((v[k] << 4) & 0xF0F0F0F0u) ^ 0x80808080u : v[k] & LOW;
                            o[16 * j + 8 + k] = MLX ? (v[k] & 0xF0F0F0F0u) ^ 0x80808080u : (v[k] >> 4) & LOW;
                        }
                    }
                    gt_st32(at + 32 * h, o);
                };
                auto multiply = [&](auto issue) {  // what the set's warps have stored, by one thread
                    gt_st_wait();
                    tc_fence_before();
                    asm volatile("bar.sync %0, 128;" ::"r"(1 + set) : "memory");
                    if constexpr (!MLX) met++;
                    if (w == 0) {
                        tc_fence_after();
                        if (elect_one()) {
                            issue(bd + (uint64_t)((lb * (NB * 256)) >> 4));
                            mma_commit(&sh->d_full[set]);
                        }
                        __syncwarp();
                    }
                };
                auto sums = [&] {
                    ok = __all_sync(0xffffffffu, gt_wait(&sh->d_full[set], phase, sh, a.status));
                    phase ^= 1;
                    tc_fence_after();
                };
                constexpr int AT_ONCE = TP == 8 ? 1 : TP == 4 ? 2 : 4;  // sums of three digits a token that registers hold at once
                constexpr int CW = TP == 8 ? 24 : 4 * TP;
                if constexpr (Q8) {  // a sum per 32, the bytes from where they were copied; 128 columns of sums at a time
                    constexpr int CHUNKS = NB == 16 ? 8 : 4;
                    const uint64_t ad = smem_desc_sw128(smem_u32(slot));
#pragma unroll
                    for (int k0 = 0; k0 < 8; k0 += CHUNKS) {
                        multiply([&](uint64_t b) {
#pragma unroll
                            for (int k = k0; k < k0 + CHUNKS; k++)
                                gt_mma_ss(base + NB * (k - k0), ad + (k >> 2) * (GT_ROWS * 128 >> 4) + 2 * (k & 3), b + (k >> 2) * (NB * 128 >> 4) + 2 * (k & 3), idesc);
                        });
                        sums();
                        if (!ok) break;
                        if (k0 + CHUNKS == 8) release_raw(&sh->raw_empty[s], hd.x, a.zero, lane);
#pragma unroll
                        for (int k1 = 0; k1 < CHUNKS; k1 += AT_ONCE) {
                            int c[AT_ONCE][CW];
#pragma unroll
                            for (int k = 0; k < AT_ONCE; k++) gt_ld(at + NB * (k1 + k), c[k]);
                            gt_ld_wait();
#pragma unroll
                            for (int k = 0; k < AT_ONCE; k++) {
                                const int g = k0 + k1 + k;
                                const float d = gt_half(g < 2 ? hd.x : g < 4 ? hd.y : g < 6 ? hd.z : hd.w, g & 1);
#pragma unroll
                                for (int t = 0; t < TP; t++) {
                                    f[t] = fmaf(d, (float)c[k][3 * t + 2], f[t]);
                                    fl[t] = fmaf(d, (float)(256 * c[k][3 * t + 1] + c[k][3 * t]), fl[t]);
                                }
                            }
                        }
                    }
                    if (!ok) break;
                } else if constexpr (MLX) {  // a sum per 64 values
                    expand(0);
                    expand(1);
                    multiply([&](uint64_t b) {
#pragma unroll
                        for (int k = 0; k < 8; k++) gt_mma(base + GT_D + 16 * (k >> 1), base + 8 * k, b + (k >> 2) * 128 + 2 * (k & 3), idesc, k & 1);
                    });
                    sums();
                    if (!ok) {
                        met = (n >> 2) + 1;
                        break;
                    }
#pragma unroll
                    for (int g0 = 0; g0 < 4; g0 += AT_ONCE) {
                        int c[AT_ONCE][CW];
#pragma unroll
                        for (int g = 0; g < AT_ONCE; g++) gt_ld(at + GT_D + 16 * (g0 + g), c[g]);
                        gt_ld_wait();
#pragma unroll
                        for (int g = 0; g < AT_ONCE; g++) {
                            const float d = gt_half(g0 + g < 2 ? hd.x : hd.y, (g0 + g) & 1);
#pragma unroll
                            for (int t = 0; t < TP; t++) {
                                f[t] = fmaf(d, (float)c[g][3 * t + 2], f[t]);
                                fl[t] = fmaf(d, fmaf((float)c[g][3 * t + 1], 256.0f, (float)c[g][3 * t]), fl[t]);
                            }
                        }
                    }
                } else {  // a sum per 32; the second half's bytes are stored while the first is multiplied
                    auto scaled = [&](uint32_t sc) {
#pragma unroll
                        for (int k0 = 0; k0 < 4; k0 += AT_ONCE) {
                            int c[AT_ONCE][CW];
#pragma unroll
                            for (int k = 0; k < AT_ONCE; k++) gt_ld(at + GT_D + 16 * (k0 + k), c[k]);
                            gt_ld_wait();
#pragma unroll
                            for (int k = 0; k < AT_ONCE; k++) {
                                const int sk = (int)((sc >> (8 * (k0 + k))) & 0xffu);
#pragma unroll
                                for (int t = 0; t < TP; t++)
#pragma unroll
                                    for (int e = 0; e < 3; e++) p[t][e] += sk * c[k][3 * t + e];
                            }
                        }
                    };
                    expand(0);
                    multiply([&](uint64_t b) {
#pragma unroll
                        for (int k = 0; k < 4; k++) gt_mma(base + GT_D + 16 * k, base + 8 * k, b + 2 * k, idesc, 0);
                    });
                    expand(1);
                    sums();
                    if (!ok) break;
                    scaled(hd.y & 0x3f3f3f3fu);
                    // (the minimums take the first half's columns; of their 32 values eight are set, the others meet zeros)
                    gt_st2(at + GT_AM, hd.z & 0x3f3f3f3fu, ((hd.w >> 4) & LOW) | ((hd.z >> 2) & 0x30303030u));  // (get_scale_min_k4, src/ggml.rs:501-509)
                    multiply([&](uint64_t b) {
#pragma unroll
                        for (int k = 0; k < 4; k++) gt_mma(base + GT_D + 16 * k, base + 32 + 8 * k, b + 128 + 2 * k, idesc, 0);
                        gt_mma(base + GT_DM, base + GT_AM, md + (uint64_t)(((lb >> 2) * 2048 + (lb & 3) * 32) >> 4), idesc, 0);
                    });
                    sums();
                    if (!ok) break;
                    scaled((hd.w & LOW) | ((hd.y >> 2) & 0x30303030u));
                }
                if constexpr (Q8) {
#pragma unroll
                    for (int t = 0; t < TP; t++) {
                        const float xs = xs_s[lb * TP + t];
                        acc[t] = fmaf(xs * 65536.0f, f[t], acc[t]);
                        low[t] = fmaf(xs, fl[t], low[t]);
                    }
                } else if constexpr (MLX) {  // w = (n - 8) d + off per 64: off times the sums of 64
#pragma unroll
                    for (int t = 0; t < TP; t++) {
                        const float xs = 0.0625f * xs_s[lb * TP + t];
                        acc[t] = fmaf(xs * 65536.0f, f[t], acc[t]);
                        low[t] = fmaf(xs, fl[t], low[t]);
#pragma unroll
                        for (int g = 0; g < 4; g++) {
                            const uint32_t ow = g < 2 ? hd.z : hd.w;
                            low[t] = fmaf(__uint_as_float((g & 1) ? ow & 0xffff0000u : ow << 16), sum_s[(lb * TP + t) * 4 + g], low[t]);
                        }
                    }
                } else {
                    int m[4 * TP];
                    gt_ld(at + GT_DM, m);
                    gt_ld_wait();
                    const float d = gt_half(hd.x, 0), dm = gt_half(hd.x, 1);
#pragma unroll
                    for (int t = 0; t < TP; t++) {
                        // (the third digit's products and the minimums' upper two by themselves: their integers are exact as floats)
                        const float xs = xs_s[lb * TP + t];
                        const float up = fmaf(d, (float)p[t][2], -(dm * (float)(256 * m[4 * t + 3] + m[4 * t + 2])));
                        const float dn = fmaf(d, fmaf((float)p[t][1], 256.0f, (float)p[t][0]), -(dm * (float)(256 * m[4 * t + 1] + m[4 * t])));
                        acc[t] = fmaf(xs * 65536.0f, up, acc[t]);
                        low[t] = fmaf(xs, dn, low[t]);
                    }
                }
            }
            if (!ok) break;
            // To the CTA that has the row: 32 of them each; of a pair, 16 of either matrix (rows 0 .. 63 of the tile are the first one's).
#pragma unroll
            for (int t = 0; t < TP; t++) acc[t] += low[t];
            const int buf = i & 1, to = PAIR ? 2 * (w & 1) + (lane >> 4) : w, row = PAIR ? 16 * (w >> 1) + (lane & 15) : lane;
            if (i >= 2) ok = __all_sync(0xffffffffu, gt_wait<true>(&sh->in_free[to][buf], (uint32_t)(((i >> 1) - 1) & 1), sh, a.status));
            if (!ok) {
                if constexpr (MLX) met = (i * nbq + nbq - set + 3) >> 2;
                break;
            }
            gt_send(cluster_addr(&sh->in[buf][GT_SETS * rank + share][row][0], to), acc, cluster_addr(&sh->in_full[buf], to));
        }
        // A warp whose wait gave up still meets the others wherever they will be waiting for it, in all of the set's blocks; and the one that issues stays
        // until the last instructions have ended.
        if (!ok) {
            if (w == 0 && met > 0) gt_wait(&sh->d_full[set], (uint32_t)(met - 1) & 1, sh, a.status, false);
            const int meets = MEETS * ((total - set + 3) >> 2);
            for (; met < meets; met++) asm volatile("bar.sync %0, 128;" ::"r"(1 + set) : "memory");
        }
    } else if (warp == 0) {
        // ---------------- packed weights ----------------
        int issued = first;
        uint32_t round = 0;  // (parity of the slots' last use)
        for (int n = first; n < total; n++) {
            if (c_slot == 0 && n > first) round ^= 1;
            if (!__all_sync(0xffffffffu, gt_wait(&sh->raw_empty[c_slot], round, sh, a.status))) break;
            issued = n + 1;
            copy();
        }
        if (sh->abort_flag)  // copies in flight land before the shared memory goes away
            for (int n = max(0, issued - a.slots); n < issued; n++) gt_wait(full_of(n), full_parity(n), sh, a.status, false);
    } else if (warp == 1) {
        // ---------------- results ----------------
        float factor[TP];
#pragma unroll
        for (int t = 0; t < TP; t++) factor[t] = 1.0f;
        bool ok = true;
        if (a.norm) {
            if (lane < GT_CTAS) {  // this part's sums of squares, to every CTA
                float q[MOST] = {};
#pragma unroll
                for (int t = 0; t < TP; t++)
                    for (int lb = 0; lb < nbq && t < T; lb++) q[t] += ssq_s[lb * TP + t];
                gt_send(cluster_addr(sh->ssq_in[rank], lane), q, cluster_addr(&sh->ssq_full, lane));
            }
            __syncwarp();
            ok = __all_sync(0xffffffffu, gt_wait<true>(&sh->ssq_full, 0, sh, a.status));
#pragma unroll
            for (int t = 0; t < TP; t++) {
                const float sq = sh->ssq_in[0][t] + sh->ssq_in[1][t] + sh->ssq_in[2][t] + sh->ssq_in[3][t];
                factor[t] = 1.0f / sqrtf(sq / (float)a.n_in + a.eps);
            }
        }
#pragma unroll 1
        for (int i = -1; i < my_tiles && ok; i++) {  // (the first pass fetches the code and stores nothing)
            const int buf = i & 1;
            int tile = cluster + i * clusters;
            float* y = a.y;
            size_t n_out = a.n_out;
            if constexpr (JOBS) {
                const int j = job_of(max(tile, 0));
                y = mats.y[j];
                n_out = mats.n_out[j];
                tile -= mats.first[j];
            }
            const size_t y_stride = JOBS ? n_out : a.y_stride;
            const size_t row = i < 0 ? n_out : PAIR ? (size_t)tile * 64 + 16 * rank + (lane & 15) : (size_t)tile * GT_ROWS + 32 * rank + lane;
            float old[TP], times[TP];  // what the results are added to, read while the products run
            if (!PAIR) {
#pragma unroll
                for (int t = 0; t < TP; t++) {
                    old[t] = a.mode != B2_MODE_STORE && t < T && row < n_out ? y[(size_t)(t0 + t) * y_stride + row] : 0.0f;
                    times[t] = a.mode != B2_MODE_STORE && a.mode != B2_MODE_ADD && t < T ? 1.0f / (1.0f + __expf(-a.gate[(size_t)(t0 + t) * a.gate_stride])) : 1.0f;
                }
            }
            if (i >= 0) ok = __all_sync(0xffffffffu, gt_wait<true>(&sh->in_full[buf], (uint32_t)((i >> 1) & 1), sh, a.status));
            if (!ok) break;
            float v[TP];
#pragma unroll
            for (int t = 0; t < TP; t++) {
                float u[GT_SETS * GT_CTAS];
#pragma unroll
                for (int p = 0; p < GT_SETS * GT_CTAS; p++) u[p] = sh->in[buf][p][lane][t];
#pragma unroll
                for (int n = GT_SETS * GT_CTAS / 2; n > 0; n /= 2)  // in pairs: a row of sixteen additions rounded off 4 % more
#pragma unroll
                    for (int p = 0; p < n; p++) u[p] = u[2 * p] + u[2 * p + 1];
                v[t] = u[0];
                v[t] *= factor[t];
            }
#pragma unroll
            for (int t = 0; t < TP; t++) {
                const float up = PAIR ? __shfl_xor_sync(0xffffffffu, v[t], 16) : 0.0f;
                if (t >= T || row >= n_out || (PAIR && lane >= 16)) continue;
                float* o = y + (size_t)(t0 + t) * y_stride + row;
                if (PAIR) *o = (a.mode == B2_MODE_SILU_PAIR ? gt_silu(v[t]) : gt_gelu(v[t])) * up;
                else *o = a.mode == B2_MODE_STORE ? v[t] : old[t] + v[t] * times[t];
            }
            if (i >= 0 && i + 2 < my_tiles) {
                if (lane == 0) mbar_arrive_expect_tx(&sh->in_full[buf], IN_BYTES);
                // (relaxed: with release at cluster scope an arrival takes 1500 cycles; what every lane has loaded enters its address, by a vote: an
                // OR over the words took
                // 1 % of a launch)
                uint32_t words = __float_as_uint(v[0]);
#pragma unroll
                for (int t = 1; t < TP; t++) words |= __float_as_uint(v[t]);
                words = __ballot_sync(0xffffffffu, words == 0x7fc0dead) & (uint32_t)a.zero;
                if (lane < GT_CTAS) gt_arrive(cluster_addr(&sh->in_free[rank][buf], lane) + words);
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    asm volatile("barrier.cluster.arrive.relaxed.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");  // (no CTA ends before its peers have stored and arrived)
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(GT_TMEM_COLS) : "memory");
    }
}

bool gt_encode(CUtensorMap* m, CUtensorMapDataType type, const void* p, size_t width, size_t rows, size_t bytes, uint32_t bw, uint32_t bh, CUtensorMapSwizzle sw) {
    TensorMapEncodeFn enc = tensor_map_encode();
    if (!enc) return false;
    cuuint64_t dims[2] = {width, rows}, strides[1] = {bytes};
    cuuint32_t box[2] = {bw, bh}, estr[2] = {1, 1};
    return enc(m, type, 2, (void*)p, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
bool gt_map(CUtensorMap* m, const WeightDev& w, uint32_t rows) {
    const size_t row = w.n_in / 256 * 144;
    return gt_encode(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, w.p0, row, w.n_out, row, 144, rows, CU_TENSOR_MAP_SWIZZLE_NONE);
}
bool gt_map_bytes(CUtensorMap* m, const WeightDev& w, uint32_t rows) {
    return gt_encode(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, w.p0, w.n_in, w.n_out, w.n_in, 128, rows, CU_TENSOR_MAP_SWIZZLE_128B);
}
bool gt_map_scales(CUtensorMap* m, const WeightDev& w, uint32_t rows) {
    return gt_encode(m, CU_TENSOR_MAP_DATA_TYPE_UINT16, w.p1, w.n_in / 32, w.n_out, w.n_in / 16, 8, rows, CU_TENSOR_MAP_SWIZZLE_NONE);
}

constexpr size_t gt_smem(int tp) { return tp == 8 ? 190 * 1024 : 208 * 1024; }  // of an SM (beside the static part)
size_t gt_fixed(int fmt, size_t K, int tp) {  // shared memory beside the ring
    const size_t nbq = (K / 256 + GT_CTAS - 1) / GT_CTAS;
    return 1024 + nbq * (tp == 8 ? 8192 : 4096) + (fmt == B2_FMT_Q4_K ? (nbq + 3) / 4 * 2048 : 0) + nbq * (tp == 8 ? 8 : GT_TOKENS) * 4 * 6;
}

template <int FMT, bool PAIR, int TP, bool JOBS>
cudaError_t gt_launch(const WeightDev& w, const WeightDev* up, const GemvTcJob* jobs, int n_jobs, GtArgs a, int sm_count, cudaStream_t st, bool pdl) {
    constexpr bool Q8 = FMT == B2_FMT_Q8_0;
    constexpr uint32_t ROWS = PAIR ? 64 : GT_ROWS;
    GtMats<JOBS, Q8> mats;
    if constexpr (JOBS) {
        a.tiles = 0;
        for (int j = 0; j < GT_MOST_JOBS; j++) {
            const GemvTcJob& job = jobs[std::min(j, n_jobs - 1)];
            if (!gt_map(&mats.m[j], *job.w, GT_ROWS)) return cudaErrorInvalidValue;
            mats.y[j] = job.y;
            mats.n_out[j] = job.w->n_out;
            mats.first[j] = j < n_jobs ? a.tiles : INT_MAX;
            if (j < n_jobs) a.tiles += (int)((job.w->n_out + GT_ROWS - 1) / GT_ROWS);
        }
    } else {
        for (int u = 0; u < 2; u++) {
            const WeightDev& m = u && PAIR ? *up : w;
            if constexpr (Q8) {
                if (!gt_map_bytes(&mats.m[u], m, ROWS) || !gt_map_scales(&mats.m[2 + u], m, ROWS)) return cudaErrorInvalidValue;
            } else {
                if (!gt_map(&mats.m[u], m, ROWS)) return cudaErrorInvalidValue;
            }
        }
        a.tiles = (int)((w.n_out + ROWS - 1) / ROWS);
    }
    const size_t nbq = (w.n_in / 256 + GT_CTAS - 1) / GT_CTAS, fixed = gt_fixed(FMT, w.n_in, TP);
    a.slots = (int)std::min<size_t>(GT_MOST_SLOTS, (gt_smem(TP) - fixed) / gt_raw(FMT));
    a.b_off = (uint32_t)a.slots * gt_raw(FMT);
    a.min_off = a.b_off + (uint32_t)nbq * (TP == 8 ? 8192 : 4096);
    a.sum_off = a.min_off + (uint32_t)(FMT == B2_FMT_Q4_K ? (nbq + 3) / 4 * 2048 : 0);
    a.xs_off = a.sum_off + (uint32_t)(nbq * TP * 16);
    const size_t smem = std::max(fixed + (size_t)a.slots * gt_raw(FMT), TMEM_512_SMEM);
    auto kern = gemv_tc_kernel<FMT, PAIR, TP, JOBS>;
    if (cudaError_t e = ensure_dynamic_smem((const void*)kern, smem, 0); e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(GT_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = GT_CTAS;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    // as many clusters as run at once (groups of SMs that are no multiple of four leave some out), a CTA an SM
    int most = 0;
    {
        static std::mutex mu_;
        static std::map<std::tuple<const void*, int, size_t>, int> known;
        int dev = 0;
        if (cudaError_t e = cudaGetDevice(&dev); e != cudaSuccess) return e;
        std::lock_guard<std::mutex> lock(mu_);
        int& m = known[std::make_tuple((const void*)kern, dev, smem)];
        if (m == 0) {
            cfg.gridDim = dim3(GT_CTAS);
            cfg.numAttrs = 1;
            if (cudaError_t e = cudaOccupancyMaxActiveClusters(&m, kern, &cfg); e != cudaSuccess) return e;
            m = std::max(1, m);
        }
        most = std::min(m, sm_count / GT_CTAS);
    }
    most >>= a.two;
    if (most < 1) return cudaErrorInvalidValue;
    a.rounds = (a.tiles + most - 1) / most;
    cfg.gridDim = dim3((unsigned)((a.tiles + a.rounds - 1) / a.rounds * GT_CTAS << a.two));
    cfg.numAttrs = pdl ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kern, mats, a);
}

template <int FMT, bool PAIR, bool JOBS = false>
cudaError_t gt_tokens(const WeightDev& w, const WeightDev* up, GtArgs a, int sm_count, cudaStream_t st, bool pdl, const GemvTcJob* jobs = nullptr, int n_jobs = 0) {
    if constexpr (FMT == B2_FMT_Q8_0) {  // (twice the bytes: a second reading costs more than columns for eight tokens)
        a.two = 0;
        if (a.T > GT_TOKENS) return gt_launch<FMT, PAIR, 8, JOBS>(w, up, jobs, n_jobs, a, sm_count, st, pdl);
    }
    if (a.T == 1) return gt_launch<FMT, PAIR, 1, JOBS>(w, up, jobs, n_jobs, a, sm_count, st, pdl);
    if (a.T == 2) return gt_launch<FMT, PAIR, 2, JOBS>(w, up, jobs, n_jobs, a, sm_count, st, pdl);
    return gt_launch<FMT, PAIR, 4, JOBS>(w, up, jobs, n_jobs, a, sm_count, st, pdl);
}

GtArgs gt_args(const WeightDev& w, const GemvIn& in, int T) {
    GtArgs a{};
    a.x = in.x;
    a.x_stride = in.x_stride;
    a.nw = in.norm_w;
    a.pre = in.pre;
    a.norm = in.norm;
    a.eps = in.eps;
    a.rec = in.rec;
    a.rec_stride = in.rec_stride;
    a.fast = in.fast;
    a.T = T;
    a.two = T > GT_TOKENS;
    a.n_in = (int)w.n_in;
    a.status = in.status;
    return a;
}

}  // namespace

// By format and K alone: all of a matrix's rows, whatever shard or token they belong to, have to take the same form. (Q8_0 up to 14336 values a row: two
// slots beside the digits of eight tokens. Q4_K up to 36864, MLX-4 to 41984.) Up to 1024 values a row the form on mma.sync is faster, by itself, where
// it splits the activations (us in a graph, one / two / four / eight tokens, on mma.sync and here: Q4_K 1024 x 1024 2.54 / 2.72 / 3.14 / 4.26 and 3.35 /
// 3.49 / 3.82 / 3.88, 14336 x 1024 5.00 / 5.46 / 5.60 / 8.03 and 5.28 / 5.71 / 6.45 / 8.80), and more so between other kernels: six layers of hidden size
// 1024 with Q4_K, Q6_K and Q8_0, four tokens, 309 us and 358.
static bool gt_fits(const WeightDev& w) {
    const int tp = w.fmt == B2_FMT_Q8_0 ? 8 : GT_TOKENS;
    return (w.fmt == B2_FMT_Q4_K || w.fmt == B2_FMT_MLX4 || (w.fmt == B2_FMT_Q8_0 && ((uintptr_t)w.p1 & 15) == 0)) && ((uintptr_t)w.p0 & 15) == 0 && w.n_in % 256 == 0 &&
           w.n_in > 0 && gt_fixed(w.fmt, w.n_in, tp) + 2 * gt_raw(w.fmt) <= gt_smem(tp);
}

bool gemv_tc_supports(const WeightDev& w) { return w.n_in > 1024 && gt_fits(w); }
// Several matrices in one launch: shorter rows too where their sums have one order here and there, a block a part (one, two or four blocks; q / k / v of
// one token from host to host, K = 1024: 27.5 us, in a launch each 32).
bool gemv_tc_jobs_supports(const WeightDev& w) {
    return w.fmt != B2_FMT_Q8_0 && gt_fits(w) && (w.n_in > 1024 || w.n_in == 256 || w.n_in == 512 || w.n_in == 1024);
}

cudaError_t launch_gemv_tc(const WeightDev& w, const WeightDev* up, const GemvIn& in, int T, float* y, size_t y_stride, int mode, const float* gate,
                           size_t gate_stride, int sm_count, cudaStream_t st, bool pdl) {
    if (!gemv_tc_supports(w) || !in.status || T < 1) return cudaErrorInvalidValue;
    const bool pair = mode == B2_MODE_SILU_PAIR || mode == B2_MODE_GELU_PAIR;
    for (int t = 0; t < T; t += 2 * GT_TOKENS) {
        GemvIn at = in;
        if (in.x) at.x = in.x + (size_t)t * in.x_stride;
        if (in.rec) at.rec = in.rec + (size_t)t * in.rec_stride;
        GtArgs a = gt_args(w, at, std::min(T - t, 2 * GT_TOKENS));
        a.y = y + (size_t)t * y_stride;
        a.y_stride = y_stride;
        a.gate = gate ? gate + (size_t)t * gate_stride : nullptr;
        a.gate_stride = gate_stride;
        a.mode = mode;
        a.n_out = w.n_out;
        cudaError_t e;
        switch (w.fmt) {
            case B2_FMT_MLX4: e = pair ? gt_tokens<B2_FMT_MLX4, true>(w, up, a, sm_count, st, pdl) : gt_tokens<B2_FMT_MLX4, false>(w, up, a, sm_count, st, pdl); break;
            case B2_FMT_Q4_K: e = pair ? gt_tokens<B2_FMT_Q4_K, true>(w, up, a, sm_count, st, pdl) : gt_tokens<B2_FMT_Q4_K, false>(w, up, a, sm_count, st, pdl); break;
            default: e = pair ? gt_tokens<B2_FMT_Q8_0, true>(w, up, a, sm_count, st, pdl) : gt_tokens<B2_FMT_Q8_0, false>(w, up, a, sm_count, st, pdl); break;
        }
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_gemv_tc_jobs(const GemvTcJob* jobs, int n_jobs, const GemvIn& in, int T, int sm_count, cudaStream_t st, bool pdl) {
    if (n_jobs < 1 || n_jobs > GEMV_TC_JOBS || !in.status || T < 1 || T > 2 * GT_TOKENS) return cudaErrorInvalidValue;
    const WeightDev& w = *jobs[0].w;
    for (int j = 0; j < n_jobs; j++)
        if (!gemv_tc_jobs_supports(*jobs[j].w) || jobs[j].w->fmt != w.fmt || jobs[j].w->n_in != w.n_in) return cudaErrorInvalidValue;
    const GtArgs a = gt_args(w, in, T);
    return w.fmt == B2_FMT_MLX4 ? gt_tokens<B2_FMT_MLX4, false, true>(w, nullptr, a, sm_count, st, pdl, jobs, n_jobs)
                                : gt_tokens<B2_FMT_Q4_K, false, true>(w, nullptr, a, sm_count, st, pdl, jobs, n_jobs);
}

}  // namespace b2
