// Dequant-GEMM with the weights in tensor memory, CTA-pair form: more than 128 tokens, and routed experts with long segments.
//
//   y[t][n_out] = x[t][K] * W^T      (one-term f16 operands, two-term ones for Q4_K experts; f32 sums; the order of the sums of gemm_wt.cu)
//
// A pair of CTAs (tcgen05 cta_group::2, M = 256) multiplies 256 weight rows by a segment of up to 256 tokens over the whole K: each CTA
// expands 128 of the rows into its own tensor memory (the A operand, a ring of slots of 128 k) and copies half of the segment's
// tokens into its shared memory (half of the B operand). The pairs are persistent; Segments says what each of them takes.
//   warps 0..15  : dequantizers, four sets of four warps, a thread per weight row; set s takes every fourth group of 64 k.
//   warps 16..19 : epilogue, through staging tiles and the copy engine.
//   warp 20      : copies the activations; warp 21 of the even CTA issues the instructions; warp 22 copies the packed weights.
// What bounds it: a stage of 128 k takes the tensor cores 4 cycles a token and the dequantizers about 780 cycles whatever the tokens, and the
// sums of a segment leave at the rate of the L2 (8000 cycles for 256 tokens when all CTAs store at once). Two layouts of tensor memory: two
// accumulators of 160 tokens, whose sums leave while the next segment is multiplied (grouped launches: many short segments), or one of 256
// (in halves, for short segments in turn), bound by the tensor cores until its sums leave (dense launches).
// (The form with tokens on M, gemm_tc.cu, needs 1250 cycles of shared memory for 830 of tensor cores.)
//
// A CTA takes all 512 columns of tensor memory and more than half of the shared memory, so it has its SM to itself.
#include <cuda.h>

#include <algorithm>

#include "expand.cuh"
#include "gemm_wt.h"
#include "tcgen05.cuh"

namespace b2 {

namespace {

constexpr int WP_THREADS = 736, WP_ROWS = 128, WP_SEG = WP_MOST_ROWS, WP_UNIT = 32, WP_PANEL = 8;
constexpr uint32_t WP_SLOT_COLS = 64;                           // an A slot of 128 k; the slots are tensor memory's last columns
constexpr int WP_TWO = WP_TILE_ROWS;                            // longest segment of the layout with two accumulators
// The two layouts: A slots, activation stages of 128 k, and what the epilogue stages its results in (two tiles of 32 tokens x 32 rows a warp).
__host__ __device__ constexpr int wp_n_a(bool two) { return two ? 3 : 4; }
__host__ __device__ constexpr int wp_n_b(bool two) { return two ? 4 : 3; }
__host__ __device__ constexpr uint32_t wp_b_stage(bool two) { return (two ? WP_TWO : WP_SEG) / 2 * 256; }
__host__ __device__ constexpr uint32_t wp_staging(bool two) { return two ? 0 : 4 * 2 * 4096; }
__host__ __device__ constexpr int wp_raw_slot(int fmt) { return WP_ROWS * (fmt == B2_FMT_F8E4M3 || fmt == B2_FMT_Q8_0 ? 64 : fmt == B2_FMT_Q6_K ? 192 : 144); }
__host__ __device__ constexpr int wp_n_raw(int fmt, bool two) { return two ? 8 : fmt == B2_FMT_F8E4M3 || fmt == B2_FMT_Q8_0 ? 12 : fmt == B2_FMT_Q6_K ? 4 : 5; }

struct __align__(8) WpShared {
    uint64_t a_full[4];            // even CTA: both CTAs' dequantizers
    uint64_t b_full[4];            // even CTA: both CTAs' copies
    uint64_t done[4];              // each CTA: the instructions of stage i (mod 4) have completed
    uint64_t raw_full[16], raw_empty[16];
    uint64_t acc_full[2];          // each CTA, [half]: the sums of the segment that starts there
    uint64_t acc_empty[2];         // even CTA, [half]: both CTAs' epilogues have read it
    uint32_t tmem_base;
    volatile uint32_t abort_flag;
};
constexpr size_t wp_smem(int fmt, bool two) {
    return 1024 + (size_t)wp_n_b(two) * wp_b_stage(two) + (size_t)wp_n_raw(fmt, two) * wp_raw_slot(fmt) + wp_staging(two);
}
static_assert(wp_smem(B2_FMT_Q4_K, false) + sizeof(WpShared) <= 227 * 1024 && wp_smem(B2_FMT_Q6_K, false) + sizeof(WpShared) <= 227 * 1024 &&
              wp_smem(B2_FMT_Q8_0, false) + sizeof(WpShared) <= 227 * 1024 && wp_smem(B2_FMT_MLX4, true) + sizeof(WpShared) <= 227 * 1024, "shared memory budget");
static_assert(wp_smem(B2_FMT_Q4_K, false) >= TMEM_512_SMEM && wp_smem(B2_FMT_Q4_K, true) >= TMEM_512_SMEM && wp_smem(B2_FMT_MLX4, false) >= TMEM_512_SMEM &&
              wp_smem(B2_FMT_MLX4, true) >= TMEM_512_SMEM && wp_smem(B2_FMT_Q6_K, false) >= TMEM_512_SMEM && wp_smem(B2_FMT_Q8_0, false) >= TMEM_512_SMEM &&
              wp_smem(B2_FMT_F8E4M3, false) >= TMEM_512_SMEM);

struct WpArgs {
    int K, n_out, t;
    WpShare share;        // dense: how the work is shared out (Segments)
    int y_bf16, zero, staged;  // staged: results leave through tmap_y
    size_t y_ld;
    void* y;
    GemmStatus* status;
    const WtTile* tiles;  // grouped launches; null: dense
    int n_tiles;
    int lo_row0;          // two-term operands: the activations' second terms lie this many rows below the first
    const float* row_unscale;
    const float* s;       // scales beside the packed rows, as in gemm_tc.cu
    const void* s2;
    int f8_rows, f8_ncb, f8_row0;
};

// The segments of a pair, the same for every role of both CTAs. Grouped launches: every tile with every row block, dealt out in turn. Dense, one of
// - pieces > 0: every row block of 256 in `pieces` equal segments, dealt out in turn, of `split` parts each from number `whole` on (the last wave).
//   They go in panels of WP_PANEL token ranges, a panel's row blocks before the next panel, its token ranges fastest: pairs that run together share
//   8 token ranges and about 9 row blocks, which fit L2 over a long stretch of K.
// - pieces 0: one list of units of 32 tokens, row block by row block, of which every pair takes an equal run, cut at the ends of row blocks; a
//   run's end within `snap` units of a row block's end is moved there. Pairs stand at unrelated tokens: for launches whose operands fit L2.
template <bool GROUPED>
struct Segments {
    int pos, end;
    int row, w_row, x_row0, n, count;  // first of the 256 rows in its matrix / in the stack; tokens: first, padded to 32, real
    __host__ __device__ __forceinline__ Segments(int n_out, int t, int n_tiles, const WpShare& share, int c, int pairs) {
        const int blocks = (n_out + 2 * WP_ROWS - 1) / (2 * WP_ROWS);
        pos = c;
        end = GROUPED ? n_tiles * blocks : share.whole + (share.pieces * blocks - share.whole) * share.split;
        if (!GROUPED && !share.pieces) {
            pos = bound(blocks, (t + WP_UNIT - 1) / WP_UNIT, c, pairs, share.snap);
            end = bound(blocks, (t + WP_UNIT - 1) / WP_UNIT, c + 1, pairs, share.snap);
        }
    }
    __host__ __device__ __forceinline__ static int bound(int blocks, int per_block, int i, int pairs, int snap) {
        const int p = (int)((long long)blocks * per_block * i / pairs), u = p % per_block;
        return u <= snap ? p - u : per_block - u <= snap ? p - u + per_block : p;
    }
    __host__ __device__ __forceinline__ bool next(const WtTile* tiles, int n_out, int t, const WpShare& share, int pairs) {
        if (pos >= end) return false;
        const int blocks = (n_out + 2 * WP_ROWS - 1) / (2 * WP_ROWS);
        if constexpr (GROUPED) {
            const WtTile tile = tiles[pos / blocks];
            row = pos % blocks * (2 * WP_ROWS);
            w_row = tile.expert * n_out + row;
            x_row0 = tile.row0;
            count = tile.count;
            n = (count + WP_UNIT - 1) / WP_UNIT * WP_UNIT;
            pos += pairs;
            return true;
        }
        int u, take;
        if (share.pieces) {
            // (no 64-bit division: the first segment's place is on the way to a launch's first weights. With two of them 2816 x 1024, 300 tokens,
            // took 8.9 us instead of 8.4.)
            const int over = pos - share.whole;
            int tile = pos, part = 0, panel = 0, wide = share.pieces;
            if (over >= 0 && share.split > 1) {
                tile = share.whole + over / share.split;
                part = over % share.split;
            }
            int in = tile;
            if (share.pieces > WP_PANEL) {
                panel = tile / (WP_PANEL * blocks);
                in -= panel * (WP_PANEL * blocks);
                const int left = share.pieces - panel * WP_PANEL;
                wide = left < WP_PANEL ? left : WP_PANEL;
            }
            const int block = in / wide, p = panel * WP_PANEL + in - block * wide;
            row = block * (2 * WP_ROWS);
            u = share.units * p + (p < share.longer ? p : share.longer);
            take = share.units + (p < share.longer ? 1 : 0);
            if (over >= 0 && share.split > 1) {
                const int from = take * part / share.split;
                take = take * (part + 1) / share.split - from;
                u += from;
            }
            pos += pairs;
        } else {
            constexpr int most = WP_SEG / WP_UNIT;
            const int per_block = (t + WP_UNIT - 1) / WP_UNIT;
            u = pos % per_block;
            const int left = per_block - u < end - pos ? per_block - u : end - pos, parts = (left + most - 1) / most;
            take = (left + parts - 1) / parts;
            row = pos / per_block * (2 * WP_ROWS);
            pos += take;
        }
        w_row = row;
        x_row0 = u * WP_UNIT;
        n = take * WP_UNIT;
        count = n < t - x_row0 ? n : t - x_row0;
        return true;
    }
};

// The accumulators of a pair's segments, the same for the issuing warp and the epilogues. Two: in turn. One: segments of up to 128 tokens take
// its halves in turn, longer ones both (`both`).
template <int SECOND>  // first column of the second accumulator; 0: one
struct Halves {
    int turn = 0, uses[2] = {0, 0}, sums[2] = {0, 0};
    int half;
    uint32_t col;  // first column
    bool both;
    uint32_t empty_parity[2], full_parity;
    __device__ __forceinline__ void next(int n) {
        both = !SECOND && n > 128;
        half = both ? 0 : turn;
        turn = both ? 0 : turn ^ 1;
        col = half ? (SECOND ? (uint32_t)SECOND : 128u) : 0u;
        empty_parity[0] = (uint32_t)(uses[0] & 1) ^ 1u;
        empty_parity[1] = (uint32_t)(uses[1] & 1) ^ 1u;
        full_parity = (uint32_t)((half ? sums[1] : sums[0]) & 1);
        if (both || half == 0) uses[0]++;
        if (both || half == 1) uses[1]++;
        if (half)
            sums[1]++;
        else
            sums[0]++;
    }
};

__device__ __forceinline__ void mma_f16_ts_pair(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
        "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// An arrival on the even CTA's barrier. What it announces lies in tensor memory and is ordered by the tcgen05 fence in front of it; with
// release semantics at cluster scope (tcgen05.cuh's form, for data in shared memory) the arrival took 1500 cycles.
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}

// TWO: the layout with two accumulators, for grouped launches; the other for dense ones. W2 (grouped, Q4_K): weights and activations as two f16
// terms; a stage is then 64 k, its slots hold both terms, the accumulators are 128 columns and the A slots four.
template <int FMT, bool TWO, bool W2 = false>
__global__ void __launch_bounds__(WP_THREADS, 1)
gemm_wp_kernel(const __grid_constant__ XMaps maps, const __grid_constant__ CUtensorMap tmap_w,
               const __grid_constant__ CUtensorMap tmap_w2, const __grid_constant__ CUtensorMap tmap_y, const __grid_constant__ WpArgs a) {
    // A dependent launch: see gemm_wt.cu.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    constexpr bool BYTE_ROWS = FMT == B2_FMT_F8E4M3 || FMT == B2_FMT_Q8_0;
    constexpr bool PRE_SCALED = BYTE_ROWS || FMT == B2_FMT_Q6_K;
    constexpr int NRAW = wp_n_raw(FMT, TWO), RAW_SLOT = wp_raw_slot(FMT), NA = W2 ? 4 : wp_n_a(TWO), NB = wp_n_b(TWO);
    constexpr int GROUPS = W2 ? 1 : 2;                  // groups of 64 k in a stage
    constexpr int SECOND = !TWO ? 0 : W2 ? 128 : WP_TWO;
    constexpr uint32_t B_STAGE = wp_b_stage(TWO);
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* b_tiles = smem;
    uint8_t* raw = smem + NB * B_STAGE;
    __shared__ WpShared shared;
    WpShared* sh = &shared;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int groups = a.K / 64, stages = groups / GROUPS;  // of a segment

    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; s++) {
            mbar_init(&sh->acc_full[s], 1);
            mbar_init(&sh->acc_empty[s], 8);
        }
        for (int s = 0; s < 4; s++) mbar_init(&sh->a_full[s], 8 * GROUPS);
        for (int s = 0; s < 4; s++) {
            mbar_init(&sh->b_full[s], 1);
            mbar_init(&sh->done[s], 1);
        }
        for (int s = 0; s < NRAW; s++) {
            mbar_init(&sh->raw_full[s], 1);
            mbar_init(&sh->raw_empty[s], BYTE_ROWS ? 4 : 16);
        }
        sh->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 21) {  // the same warp of both CTAs
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh->tmem_base)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // both CTAs' barriers exist before either signals the other's
    tc_fence_after();
    const uint32_t tmem = sh->tmem_base, a_cols = tmem + 512u - NA * WP_SLOT_COLS;
    Segments<TWO> seg(a.n_out, a.t, a.n_tiles, a.share, blockIdx.x >> 1, gridDim.x >> 1);

    if (warp == 20) {
        // ---------------- activations: this CTA's half of the segment's tokens ----------------
        {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            int it = 0, s = 0;
            bool ok = true;
            while (ok && seg.next(a.tiles, a.n_out, a.t, a.share, gridDim.x >> 1)) {
                const int half = seg.n / 2, y0 = seg.x_row0 + (int)rank * half;
                const CUtensorMap* tmap_x = &maps.m[half / 16 - 1];
                for (int ks = 0; ks < stages; ks++, it++, s = s + 1 == NB ? 0 : s + 1) {
                    const int old = it - NB;
                    if (old >= 0) ok = __all_sync(0xffffffffu, mbar_wait(&sh->done[old & 3], (uint32_t)((old >> 2) & 1), sh, a.status, 41, (uint32_t)it));
                    if (!ok) break;
                    if (!elect_one()) continue;
                    if (rank == 0) mbar_arrive_expect_tx(&sh->b_full[s], (uint32_t)(seg.n * 256));
                    tma_load_3d_pair(b_tiles + (size_t)s * B_STAGE, tmap_x, cluster_addr(&sh->b_full[s], 0), 0, y0, GROUPS * ks);  // [group or term][tokens][64]
                    if (W2) tma_load_3d_pair(b_tiles + (size_t)s * B_STAGE + (size_t)half * 128, tmap_x, cluster_addr(&sh->b_full[s], 0), 0, a.lo_row0 + y0, ks);
                }
            }
            __syncwarp();
            if (sh->abort_flag && rank == 0)  // (the odd CTA's copies are counted here too; the CTAs meet before the shared memory goes away)
                for (int i = max(0, it - NB); i < it; i++) mbar_wait(&sh->b_full[i % NB], (uint32_t)((i / NB) & 1), sh, a.status, 42, (uint32_t)i, false);
        }
    } else if (warp == 22) {
        // ---------------- packed weights: this CTA's 128 rows ----------------
        {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_w) : "memory");
            const int copies = BYTE_ROWS ? groups : groups / 4;
            int issued = 0, s = 0, ph = 0;
            bool ok = true;
            while (ok && seg.next(a.tiles, a.n_out, a.t, a.share, gridDim.x >> 1)) {
                const int w_row = seg.w_row + (int)rank * WP_ROWS;
                for (int c = 0; c < copies; c++, issued++) {
                    ok = __all_sync(0xffffffffu, mbar_wait(&sh->raw_empty[s], (uint32_t)(ph ^ 1), sh, a.status, 43, (uint32_t)issued));
                    if (!ok) break;
                    if (elect_one()) {
                        mbar_arrive_expect_tx(&sh->raw_full[s], (uint32_t)RAW_SLOT);
                        uint8_t* dst = raw + (size_t)s * RAW_SLOT;
                        if constexpr (FMT == B2_FMT_Q6_K) {
                            tma_load_2d(dst, &tmap_w, &sh->raw_full[s], c * 128, w_row);
                            tma_load_2d(dst + WP_ROWS * 128, &tmap_w2, &sh->raw_full[s], c * 64, w_row);
                        } else {
                            tma_load_2d(dst, &tmap_w, &sh->raw_full[s], c * (BYTE_ROWS ? 64 : 144), w_row);
                        }
                    }
                    __syncwarp();
                    if (++s == NRAW) s = 0, ph ^= 1;
                }
            }
            if (sh->abort_flag)
                for (int c = max(0, issued - NRAW); c < issued; c++)
                    mbar_wait(&sh->raw_full[c % NRAW], (uint32_t)((c / NRAW) & 1), sh, a.status, 44, (uint32_t)c, false);
        }
    } else if (warp == 21) {
        // ---------------- instructions (even CTA) ----------------
        if (rank == 0) {
            const uint64_t bdesc0 = smem_desc_sw128(smem_u32(b_tiles));
            const uint32_t done_of[2] = {cluster_addr(&sh->done[0], 0), cluster_addr(&sh->done[0], 1)};
            bool ok = true;
            int it = 0, sa = 0, pa = 0, s = 0, ph = 0;
            Halves<SECOND> acc_of;
            while (ok && seg.next(a.tiles, a.n_out, a.t, a.share, gridDim.x >> 1)) {
                acc_of.next(seg.n);
                const uint32_t acc = tmem + acc_of.col;
                const uint32_t idesc = (1u << 4) | ((uint32_t)(seg.n >> 3) << 17) | ((256u >> 4) << 24);
                const uint32_t group_b = (uint32_t)(seg.n / 2 * 128) >> 4;
                ok = __all_sync(0xffffffffu, (!(acc_of.both || acc_of.half == 0) || mbar_wait(&sh->acc_empty[0], acc_of.empty_parity[0], sh, a.status, 45, (uint32_t)it)) &&
                                                 (!(acc_of.both || acc_of.half == 1) || mbar_wait(&sh->acc_empty[1], acc_of.empty_parity[1], sh, a.status, 45, (uint32_t)it)));
                if (!ok) break;
                tc_fence_after();
                for (int ks = 0; ks < stages; ks++, it++) {
                    ok = __all_sync(0xffffffffu, mbar_wait_both(&sh->b_full[s], (uint32_t)ph, &sh->a_full[sa], (uint32_t)pa, sh,
                                                                    a.status, 46, (uint32_t)it));
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const uint64_t bd = bdesc0 + (uint64_t)(((uint32_t)s * B_STAGE) >> 4);
                        const uint32_t at = a_cols + (uint32_t)sa * WP_SLOT_COLS;
#pragma unroll
                        for (int g = 0; g < GROUPS; g++)
#pragma unroll
                            for (int kk = 0; kk < 4; kk++) {
                                mma_f16_ts_pair(acc, at + 32 * g + 8 * kk, bd + g * group_b + 2 * kk, idesc, ks > 0 || g > 0 || kk > 0 ? 1u : 0u);
                                if (W2) {  // (second terms of both: below f32's rounding)
                                    mma_f16_ts_pair(acc, at + 8 * kk, bd + group_b + 2 * kk, idesc, 1u);
                                    mma_f16_ts_pair(acc, at + 32 + 8 * kk, bd + 2 * kk, idesc, 1u);
                                }
                            }
                        mma_commit_pair(done_of[0] + (uint32_t)(it & 3) * 8u);
                        mma_commit_pair(done_of[1] + (uint32_t)(it & 3) * 8u);
                        if (ks == stages - 1) {
                            mma_commit_pair(cluster_addr(&sh->acc_full[acc_of.half], 0));
                            mma_commit_pair(cluster_addr(&sh->acc_full[acc_of.half], 1));
                        }
                    }
                    __syncwarp();
                    if (++sa == NA) sa = 0, pa ^= 1;
                    if (++s == NB) s = 0, ph ^= 1;
                }
            }
            if (!ok && it > 0) mbar_wait(&sh->done[(it - 1) & 3], (uint32_t)(((it - 1) >> 2) & 1), sh, a.status, 48, 0, false);  // what was issued completes
        }
    } else if (warp >= 16) {
        // ---------------- epilogue ----------------
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const uint32_t acc_lane = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        const uint32_t empty_even = cluster_addr(&sh->acc_empty[0], 0);
        uint8_t* staging = raw + (size_t)NRAW * RAW_SLOT + (size_t)(warp & 3) * 8192;
        Halves<SECOND> acc_of;
        int tile = 0;
        while (seg.next(a.tiles, a.n_out, a.t, a.share, gridDim.x >> 1)) {
            acc_of.next(seg.n);
            const int row0 = seg.row + (int)rank * WP_ROWS + (warp & 3) * 32, row = row0 + lane;
            auto factor = [&](int c) {  // of token c + lane
                return (PRE_SCALED ? 1.0f / WT_PRE : 1.0f) * (a.row_unscale && c + lane < seg.count ? __ldg(a.row_unscale + seg.x_row0 + c + lane) : 1.0f);
            };
            float next = factor(0);
            if (!__all_sync(0xffffffffu, mbar_wait(&sh->acc_full[acc_of.half], acc_of.full_parity, sh, a.status, 49, (uint32_t)tile) && !sh->abort_flag)) break;
            tc_fence_after();
            // (a loop of one chunk: unrolled over the segment it is 24 KB of code that runs once a segment, at the rate of its instruction
            // fetches, 15000 cycles)
#pragma unroll 1
            for (int c = 0; c < seg.n; c += 32) {
                const float f = next;
                next = factor(c + 32);
                uint32_t v[32];
                tmem_ld32(acc_lane + acc_of.col + (uint32_t)c, v);
                if (c == 96 && acc_of.both) {  // the first half is free
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_remote(empty_even);
                }
                const int live = seg.count - c;  // tokens to store
                if (!TWO && a.staged) {  // (the copy engine leaves out what lies past t and n_out)
                    uint8_t* buf = staging + (tile++ & 1) * 4096;
                    if (elect_one()) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");  // the store before the last has read this tile
                    __syncwarp();
                    if (a.y_bf16) {
#pragma unroll
                        for (int j = 0; j < 32; j++)
                            ((__nv_bfloat16*)buf)[j * 32 + lane] = __float2bfloat16_rn(__uint_as_float(v[j]) * __shfl_sync(0xffffffffu, f, j));
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; j++) ((float*)buf)[j * 32 + lane] = __uint_as_float(v[j]) * __shfl_sync(0xffffffffu, f, j);
                    }
                    fence_proxy_async();
                    __syncwarp();
                    if (elect_one()) {
                        asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(&tmap_y), "r"(smem_u32(buf)),
                                     "r"(row0), "r"(seg.x_row0 + c)
                                     : "memory");
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    }
                    __syncwarp();
                    continue;
                }
                const size_t at = (size_t)(seg.x_row0 + c) * a.y_ld + row;
                const int rows = row < a.n_out ? live : 0;
                if (TWO || !a.y_bf16) {
                    float* o = (float*)a.y + at;
#pragma unroll
                    for (int j = 0; j < 32; j++, o += a.y_ld) {
                        const float w = __uint_as_float(v[j]) * __shfl_sync(0xffffffffu, f, j);
                        if (j < rows) *o = w;
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 32; j++) {
                        const float w = __uint_as_float(v[j]) * __shfl_sync(0xffffffffu, f, j);
                        if (j < rows) ((__nv_bfloat16*)a.y)[at + (size_t)j * a.y_ld] = __float2bfloat16_rn(w);
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_remote(empty_even + (acc_of.both || acc_of.half == 1 ? 8u : 0u));
        }
        if (elect_one()) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");  // the staging tiles have been read and written out
        __syncwarp();
    } else {
        // ---------------- dequantizers ----------------
        const int set = warp >> 2, r = (warp & 3) * 32 + lane;
        const uint32_t swz = (uint32_t)(r & 7), swh = (uint32_t)((r >> 1) & 3);
        const uint32_t a_lane = a_cols + ((uint32_t)((warp & 3) * 32) << 16);
        const uint32_t full_even = cluster_addr(&sh->a_full[0], 0);
        bool ok = true;
        // 64 expanded weights, group g of the segment whose first stage is it0, to this lane of tensor memory. W2: `term` 0, then 1.
        int stage_a = 0, sa = 0;  // (a set's groups come in ascending order)
        auto put = [&](int it0, int g, const uint32_t(&o)[32], int term = 0) {
            const int it = it0 + g / GROUPS, old = it - NA;
            for (; stage_a < it; stage_a++) sa = sa + 1 == NA ? 0 : sa + 1;
            if (old >= 0 && term == 0) ok = __all_sync(0xffffffffu, mbar_wait(&sh->done[old & 3], (uint32_t)((old >> 2) & 1), sh, a.status, 50, (uint32_t)it));
            if (!ok) return;
            tc_fence_after();
            tmem_st32(a_lane + (uint32_t)sa * WP_SLOT_COLS + (uint32_t)(W2 ? term : g & 1) * 32u, o);
            if (W2 && term == 0) return;
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_remote(full_even + (uint32_t)sa * 8u);
        };
        auto raw_ready = [&](int slot, int ph, int c) {
            ok = __all_sync(0xffffffffu, mbar_wait(&sh->raw_full[slot], (uint32_t)ph, sh, a.status, 51, (uint32_t)c));
            return ok;
        };
        int it0 = 0, slot = 0, ph = 0, base = 0;
        for (; ok && seg.next(a.tiles, a.n_out, a.t, a.share, gridDim.x >> 1); it0 += stages) {
            const int row = seg.row + (int)rank * WP_ROWS + r;
            const bool live = row < a.n_out;
            const size_t wrow = live ? (size_t)row : 0;
            if constexpr (BYTE_ROWS) {
                const uint8_t* sc_row = (const uint8_t*)a.s;  // (Q8_0: two f16 a group; FP8: one f32 for two groups)
                if constexpr (FMT == B2_FMT_Q8_0)
                    sc_row += wrow * (size_t)a.f8_ncb * 2;
                else
                    sc_row = a.s ? sc_row + (wrow + a.f8_row0) / a.f8_rows * a.f8_ncb * 4 : nullptr;
                auto scales_of = [&](int g) {
                    return live && g < groups && sc_row ? __ldg((const uint32_t*)(sc_row + (size_t)(FMT == B2_FMT_Q8_0 ? g : g >> 1) * 4)) : 0u;
                };
                // The staging slots run on over the segments, and a slot stays with one set: its waits then come in the order of the slot's
                // phases also where a segment has no whole number of four groups (K a multiple of 128 and not of 256).
                static_assert(!BYTE_ROWS || NRAW % 4 == 0, "a slot has one owner");
                const int first = (set - base) & 3;
                uint32_t next = scales_of(first);
                for (int g = first; g < groups; g += 4) {
                    const uint32_t sc = next;
                    next = scales_of(g + 4);
                    const int c = base + g, s = c % NRAW;
                    if (!raw_ready(s, (c / NRAW) & 1, c)) break;
                    const uint4* my = (const uint4*)(raw + (size_t)s * RAW_SLOT + (size_t)r * 64);
                    uint4 q[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) q[i] = my[(uint32_t)i ^ swh];
                    release_raw(&sh->raw_empty[s], q[0].x | q[1].x | q[2].x | q[3].x, a.zero, lane);
                    uint32_t o[32];
                    if constexpr (FMT == B2_FMT_Q8_0)
                        expand_q8_0(q, sc, o);
                    else
                        expand_f8(q, a.s ? __uint_as_float(sc) : 1.0f, o);
                    put(it0, g, o);
                    if (!ok) break;
                }
                base += groups;
            } else if constexpr (FMT == B2_FMT_Q6_K) {
                // set s: half s / 2 of every super-block, its low (s even) or high nibbles
                const int half = set >> 1, odd = set & 1;
                const uint8_t* sc_row = (const uint8_t*)a.s + wrow * (size_t)(a.K / 16) + 4 * set;
                const unsigned short* d_row = (const unsigned short*)a.s2 + wrow * (size_t)(a.K / 256);
                uint32_t next_d = live ? __ldg(d_row) : 0u, next_sc = live ? __ldg((const uint32_t*)sc_row) : 0u;
                for (int sb = 0; sb < groups / 4; sb++) {
                    const float d = __half2float(__ushort_as_half((unsigned short)next_d));
                    const uint32_t sc4 = next_sc;
                    if (live && sb + 1 < groups / 4) {
                        next_d = __ldg(d_row + sb + 1);
                        next_sc = __ldg((const uint32_t*)(sc_row + (size_t)(sb + 1) * 16));
                    }
                    if (!raw_ready(slot, ph, sb)) break;
                    const uint4* my = (const uint4*)(raw + (size_t)slot * RAW_SLOT + (size_t)r * 128);
                    const uint4* my_qh = (const uint4*)(raw + (size_t)slot * RAW_SLOT + WP_ROWS * 128 + (size_t)r * 64);
                    uint4 ql4[4], qh4[2];
#pragma unroll
                    for (int c = 0; c < 4; c++) ql4[c] = my[((uint32_t)(4 * half + c)) ^ swz];
#pragma unroll
                    for (int c = 0; c < 2; c++) qh4[c] = my_qh[((uint32_t)(2 * half + c)) ^ swh];
                    release_raw(&sh->raw_empty[slot], ql4[0].x | ql4[1].x | ql4[2].x | ql4[3].x | qh4[0].x | qh4[1].x, a.zero, lane);
                    if (++slot == NRAW) slot = 0, ph ^= 1;
                    uint32_t o[32];
                    if (odd)
                        expand_q6k(ql4, qh4, d, sc4, true, o);
                    else
                        expand_q6k(ql4, qh4, d, sc4, false, o);
                    put(it0, sb * 4 + set, o);
                    if (!ok) break;
                }
            } else {
                for (int sb = 0; sb < groups / 4; sb++) {
                    if (!raw_ready(slot, ph, sb)) break;
                    const uint4* my = (const uint4*)(raw + (size_t)slot * RAW_SLOT + (size_t)r * 144);
                    const uint4 hdr = my[0], q0 = my[1 + 2 * set], q1 = my[2 + 2 * set];
                    release_raw(&sh->raw_empty[slot], hdr.x | q0.x | q1.x, a.zero, lane);
                    if (++slot == NRAW) slot = 0, ph ^= 1;
                    const uint32_t qw[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
                    uint32_t o[32];
                    expand_4bit<FMT>(hdr, qw, set, o);
                    put(it0, sb * 4 + set, o);
                    if (W2 && ok) {
                        expand_4bit_rest(hdr, qw, set, o);
                        put(it0, sb * 4 + set, o, 1);
                    }
                    if (!ok) break;
                }
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // neither CTA's shared or tensor memory goes away while the other may still signal or read it
    if (warp == 21) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

}  // namespace

// How a dense launch is shared out, and what its slowest pair takes in cycles: a stage of 128 k max(780, 4 tokens), the sums of a segment
// of more than 128 tokens 7500 (nothing is multiplied meanwhile). Runs of up to 16 units come as equal runs or as whole segments, whichever ends first;
// longer ones, whose launches' operands may not fit L2, in panels: FP8 28672 x 12288, 8192 tokens, read 24.9 GB from DRAM in equal runs (5.36 ms)
// and reads 6.8 in panels (4.27); Q4_K 4096 x 14336, 8192 tokens, 2.07 GB (732 us) and 0.72 (654).
double gemm_wp_share(GemmWp* g, size_t n_out_, size_t t_, size_t n_in, int sm_count) {
    const int n_out = (int)n_out_, t = (int)t_, stages = (int)(n_in / 128), units = (t + WP_UNIT - 1) / WP_UNIT, blocks = (n_out + 2 * WP_ROWS - 1) / (2 * WP_ROWS);
    const int pairs = (int)std::min<long long>(std::max(1, sm_count / 2), (long long)blocks * units), most = WP_SEG / WP_UNIT, least = (units + most - 1) / most;
    auto segment = [&](int n) { return stages * std::max(780.0, 4.0 * n) + (n > 128 ? 7500.0 : 500.0); };
    double best = 1e30;
    auto take = [&](double cost, int busy, const WpShare& share) {
        if (cost >= best) return;
        best = cost;
        g->busy = std::min(busy, pairs);
        g->share = share;
    };
    auto run = [&](int snap) {
        const WpShare share{0, snap, 0, 1, 0, 0};
        double cost = 0.0;
        int busy = 0;
        for (int c = 0; c < pairs && cost < best; c++) {
            double sum = 0.0;
            for (Segments<false> s(n_out, t, 0, share, c, pairs); s.next(nullptr, n_out, t, share, pairs);) sum += segment(s.n);
            cost = std::max(cost, sum);
            busy += sum > 0.0;
        }
        take(cost, busy, share);
    };
    auto deal = [&](int pieces, int most_parts) {  // whole waves of whole segments, and the rest in as many parts as cost least
        const int tiles = pieces * blocks, rest = tiles % pairs, longest = (units + pieces - 1) / pieces;
        for (int split = 1; split <= most_parts; split++)
            take(tiles / pairs * segment(longest * WP_UNIT) + (rest * split + pairs - 1) / pairs * segment((longest + split - 1) / split * WP_UNIT),
                 tiles - rest + rest * split, WpShare{pieces, 0, tiles - rest, split, units / pieces, units % pieces});
    };
    g->pairs = pairs;
    if ((long long)blocks * units / pairs <= 16) {
        run(std::min(3, (units - 1) / 2));
        run(0);
        deal(least, 1);
        if (least < units) deal(least + 1, 1);
    } else {
        deal(least, units / least);
    }
    return best;
}

bool gemm_wp_encode(GemmWp* g, const WeightDev& w, size_t experts, bool grouped, const void* x16, size_t x_rows, int sm_count, void* y, int y_dtype, size_t y_ld, size_t lo_row0) {
    GemmWt m;  // the weights' maps are gemm_wt.cu's (boxes of 128 rows)
    if (!gemm_wt_encode(&m, w, experts, x16, x_rows, 16, 1, 0, false)) return false;
    g->w = m.w;
    g->w2 = m.w2;
    g->y = m.w;
    const size_t esize = y_dtype == B2_BF16 ? 2 : 4;
    g->staged = !grouped && y_ld * esize % 16 == 0 && ((uintptr_t)y & 15) == 0;
    if (g->staged) {
        cuuint64_t dims[2] = {(cuuint64_t)w.n_out, (cuuint64_t)x_rows};
        cuuint64_t strides[1] = {(cuuint64_t)(y_ld * esize)};
        cuuint32_t box[2] = {32, 32}, estr[2] = {1, 1};
        if (tensor_map_encode()(&g->y, esize == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, y, dims, strides, box, estr,
                                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return false;
    }
    if (grouped) g->pairs = std::max(1, sm_count / 2);
    g->lo_row0 = (int)lo_row0;
    return gemm_x_maps(&g->x, 0, WP_SEG / 32 - 1, x16, lo_row0 + x_rows, w.n_in, lo_row0 ? 1 : 2);
}

cudaError_t launch_gemm_wp(const GemmWp& g, const WeightDev& w, size_t t, const WtTile* tiles, int n_tiles, void* y, int y_dtype, size_t y_ld,
                           GemmStatus* status, const float* row_unscale, cudaStream_t st) {
    using Kern = void (*)(XMaps, CUtensorMap, CUtensorMap, CUtensorMap, WpArgs);
    if (tiles && w.fmt != (g.lo_row0 ? B2_FMT_Q4_K : B2_FMT_MLX4)) return cudaErrorInvalidValue;
    Kern kern = tiles && g.lo_row0       ? gemm_wp_kernel<B2_FMT_Q4_K, true, true>
                : tiles                  ? gemm_wp_kernel<B2_FMT_MLX4, true>
                : w.fmt == B2_FMT_Q6_K   ? gemm_wp_kernel<B2_FMT_Q6_K, false>
                : w.fmt == B2_FMT_Q8_0   ? gemm_wp_kernel<B2_FMT_Q8_0, false>
                : w.fmt == B2_FMT_MLX4   ? gemm_wp_kernel<B2_FMT_MLX4, false>
                : w.fmt == B2_FMT_F8E4M3 ? gemm_wp_kernel<B2_FMT_F8E4M3, false>
                                         : gemm_wp_kernel<B2_FMT_Q4_K, false>;
    const size_t smem = wp_smem(w.fmt, tiles != nullptr);
    if (cudaError_t e = ensure_dynamic_smem((const void*)kern, smem, 0); e != cudaSuccess) return e;
    WpArgs a{};
    a.K = (int)w.n_in;
    a.n_out = (int)w.n_out;
    a.t = (int)t;
    a.share = g.share;
    a.staged = g.staged;
    a.y_bf16 = y_dtype == B2_BF16;
    a.y_ld = y_ld;
    a.y = y;
    a.status = status;
    a.tiles = tiles;
    a.n_tiles = n_tiles;
    a.lo_row0 = g.lo_row0;
    a.row_unscale = row_unscale;
    a.s = (const float*)(w.fmt == B2_FMT_Q6_K ? w.p2 : w.p1);
    a.s2 = w.p3;
    a.f8_rows = w.fmt == B2_FMT_F8E4M3 ? (int)w.bs_rows : 1;
    a.f8_ncb = w.fmt == B2_FMT_Q8_0 ? (int)(w.n_in / 32) : (int)w.bs_ncb;
    a.f8_row0 = (int)w.bs_row0;
    const size_t blocks = (w.n_out + 2 * WP_ROWS - 1) / (2 * WP_ROWS);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(2 * (tiles ? std::min<size_t>(blocks * (size_t)n_tiles, (size_t)g.pairs) : (size_t)g.pairs)));
    cfg.blockDim = dim3(WP_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2] = {};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 2;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kern, g.x, g.w, g.w2, g.y, a);
}

}  // namespace b2
