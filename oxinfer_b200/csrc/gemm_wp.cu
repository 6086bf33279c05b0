// Dequant-GEMM with the weights in tensor memory, CTA-pair form: more than 128 tokens, and routed experts with long segments.
//
//   y[t][n_out] = x[t][K] * W^T      (one-term f16 operands, f32 sums; the operands and the order of the sums of gemm_wt.cu)
//
// A pair of CTAs (tcgen05 cta_group::2, M = 256) multiplies 256 weight rows by a segment of up to 160 tokens over the whole K: each CTA
// expands 128 of the rows into its own tensor memory (the A operand) and copies half of the segment's tokens into its shared memory
// (half of the B operand). The pairs are persistent and share the work out evenly:
// the units (row block, 32 tokens) are one list of which every pair takes an equal run, cut into segments at the ends of row blocks.
//   warps 0..15  : dequantizers, four sets of four warps, a thread per weight row; set s takes every fourth group of 64 k.
//   warps 16..19 : epilogue. The accumulator is double (2 x 160 columns), so a segment's sums leave while the next one is multiplied.
//   warp 20      : copies the activations; warp 21 of the even CTA issues the instructions; warp 22 copies the packed weights.
// What bounds it: the form it replaces (tokens on M, expanded weights through shared memory) used 1250 cycles of shared memory a stage of
// 64 k for 830 cycles of tensor cores, in tiles that leave half of a last wave idle (14336 x 512 tokens: 138 CTAs of 148). Here
// shared memory works two thirds as long as the tensor cores.
//
// A CTA takes all 512 columns of tensor memory and more than half of the shared memory, so it has its SM to itself.
#include <cuda.h>

#include <algorithm>

#include "expand.cuh"
#include "gemm_wt.h"
#include "tcgen05.cuh"

namespace b2 {

namespace {

constexpr int WP_THREADS = 736, WP_ROWS = 128, WP_SEG = WP_MOST_ROWS, WP_UNIT = 32;
constexpr int WP_NB = 4;                                        // activation stages of 128 k x 80 tokens
constexpr uint32_t WP_B_STAGE = WP_SEG / 2 * 256;
constexpr uint32_t WP_A_COL = 2 * WP_SEG, WP_SLOT_COLS = 64;    // two accumulators, then the A slots of 128 k
constexpr int WP_NA = (512 - 2 * WP_SEG) / 64;
__host__ __device__ constexpr int wp_raw_slot(int fmt) { return WP_ROWS * (fmt == B2_FMT_F8E4M3 || fmt == B2_FMT_Q8_0 ? 64 : fmt == B2_FMT_Q6_K ? 192 : 144); }
__host__ __device__ constexpr int wp_n_raw(int fmt) { return fmt == B2_FMT_F8E4M3 || fmt == B2_FMT_Q8_0 ? 16 : 6; }

struct __align__(8) WpShared {
    uint64_t a_full[WP_NA];        // even CTA: both CTAs' dequantizers
    uint64_t b_full[WP_NB];        // even CTA: both CTAs' copies
    uint64_t done[4];              // each CTA: the instructions of stage i (mod 4) have completed
    uint64_t raw_full[16], raw_empty[16];
    uint64_t acc_full[2];          // each CTA
    uint64_t acc_empty[2];         // even CTA: both CTAs' epilogues
    uint32_t tmem_base;
    volatile uint32_t abort_flag;
};
constexpr size_t wp_smem(int fmt) { return 1024 + (size_t)WP_NB * WP_B_STAGE + (size_t)wp_n_raw(fmt) * wp_raw_slot(fmt); }
static_assert(wp_smem(B2_FMT_Q4_K) + sizeof(WpShared) <= 227 * 1024 && wp_smem(B2_FMT_Q6_K) + sizeof(WpShared) <= 227 * 1024 &&
              wp_smem(B2_FMT_Q8_0) + sizeof(WpShared) <= 227 * 1024, "shared memory budget");

struct WpArgs {
    int K, n_out, t;
    int y_bf16, zero;
    size_t y_ld;
    void* y;
    GemmStatus* status;
    const WtTile* tiles;  // grouped launches; null: dense
    int n_tiles;
    const float* row_unscale;
    const float* s;       // scales beside the packed rows, as in gemm_tc.cu
    const void* s2;
    int f8_rows, f8_ncb, f8_row0;
    int n_more;           // other ranks' copies of y
    float* more[7];
};

// The segments of a pair, the same for every role of both CTAs.
struct Segments {
    int pos, end, per_block, blocks;
    int row, w_row, x_row0, n, count;  // first of the 256 rows in its matrix / in the stack; tokens: first, padded to 32, real
    __device__ __forceinline__ Segments(const WpArgs& a) {
        const int c = blockIdx.x >> 1, pairs = gridDim.x >> 1;
        blocks = (a.n_out + 2 * WP_ROWS - 1) / (2 * WP_ROWS);
        per_block = (a.t + WP_UNIT - 1) / WP_UNIT;
        if (a.tiles) {
            pos = c;
            end = a.n_tiles * blocks;
        } else {
            // (a run that would end or start within a unit or two of a row block's end is moved there: a segment of 32 tokens takes as
            // long as one of 128)
            const long long units = (long long)blocks * per_block;
            auto bound = [&](int i) {
                const int p = (int)(units * i / pairs), u = p % per_block;
                return per_block < 8 ? p : u <= 2 ? p - u : per_block - u <= 2 ? p - u + per_block : p;
            };
            pos = bound(c);
            end = bound(c + 1);
        }
    }
    __device__ __forceinline__ bool next(const WpArgs& a) {
        if (pos >= end) return false;
        if (a.tiles) {
            const WtTile tile = a.tiles[pos / blocks];
            row = pos % blocks * (2 * WP_ROWS);
            w_row = tile.expert * a.n_out + row;
            x_row0 = tile.row0;
            count = tile.count;
            n = (count + WP_UNIT - 1) / WP_UNIT * WP_UNIT;
            pos += gridDim.x >> 1;
        } else {
            const int u = pos % per_block, left = min(per_block - u, end - pos);
            const int pieces = (left + WP_SEG / WP_UNIT - 1) / (WP_SEG / WP_UNIT), take = (left + pieces - 1) / pieces;
            row = w_row = pos / per_block * (2 * WP_ROWS);
            x_row0 = u * WP_UNIT;
            n = take * WP_UNIT;
            count = min(n, a.t - x_row0);
            pos += take;
        }
        return true;
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

template <int FMT>
__global__ void __launch_bounds__(WP_THREADS, 1)
gemm_wp_kernel(const __grid_constant__ XMaps maps, const __grid_constant__ CUtensorMap tmap_w,
               const __grid_constant__ CUtensorMap tmap_w2, const __grid_constant__ WpArgs a) {
    // A dependent launch: see gemm_wt.cu.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    constexpr bool BYTE_ROWS = FMT == B2_FMT_F8E4M3 || FMT == B2_FMT_Q8_0;
    constexpr bool PRE_SCALED = BYTE_ROWS || FMT == B2_FMT_Q6_K;
    constexpr int NRAW = wp_n_raw(FMT), RAW_SLOT = wp_raw_slot(FMT);
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* b_tiles = smem;
    uint8_t* raw = smem + (size_t)WP_NB * WP_B_STAGE;
    __shared__ WpShared shared;
    WpShared* sh = &shared;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int groups = a.K / 64, stages = groups / 2;  // of a segment

    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; s++) {
            mbar_init(&sh->acc_full[s], 1);
            mbar_init(&sh->acc_empty[s], 8);
        }
        for (int s = 0; s < WP_NA; s++) mbar_init(&sh->a_full[s], 16);
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
    const uint32_t tmem = sh->tmem_base;
    Segments seg(a);

    if (warp == 20) {
        // ---------------- activations: this CTA's half of the segment's tokens ----------------
        {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            int it = 0;
            bool ok = true;
            while (ok && seg.next(a)) {
                const int half = seg.n / 2, y0 = seg.x_row0 + (int)rank * half;
                const CUtensorMap* tmap_x = &maps.m[half / 16 - 1];
                for (int ks = 0; ks < stages; ks++, it++) {
                    const int old = it - WP_NB, s = it & (WP_NB - 1);
                    if (old >= 0) ok = __all_sync(0xffffffffu, mbar_wait(&sh->done[old & 3], (uint32_t)((old >> 2) & 1), sh, a.status, 41, (uint32_t)it));
                    if (!ok) break;
                    if (!elect_one()) continue;
                    if (rank == 0) mbar_arrive_expect_tx(&sh->b_full[s], (uint32_t)(seg.n * 256));
                    tma_load_3d_pair(b_tiles + (size_t)s * WP_B_STAGE, tmap_x, cluster_addr(&sh->b_full[s], 0), 0, y0, 2 * ks);  // [group][tokens][64]
                }
            }
            __syncwarp();
            if (sh->abort_flag && rank == 0)  // (the odd CTA's copies are counted here too; the CTAs meet before the shared memory goes away)
                for (int i = max(0, it - WP_NB); i < it; i++) mbar_wait(&sh->b_full[i & (WP_NB - 1)], (uint32_t)((i / WP_NB) & 1), sh, a.status, 42, (uint32_t)i, false);
        }
    } else if (warp == 22) {
        // ---------------- packed weights: this CTA's 128 rows ----------------
        {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_w) : "memory");
            const int copies = BYTE_ROWS ? groups : groups / 4;
            int issued = 0, s = 0, ph = 0;
            bool ok = true;
            while (ok && seg.next(a)) {
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
            int it = 0, si = 0;
            for (; ok && seg.next(a); si++) {
                const int buf = si & 1;
                const uint32_t acc = tmem + (uint32_t)(buf * WP_SEG);
                const uint32_t idesc = (1u << 4) | ((uint32_t)(seg.n >> 3) << 17) | ((256u >> 4) << 24);
                const uint32_t group_b = (uint32_t)(seg.n / 2 * 128) >> 4;
                ok = __all_sync(0xffffffffu, mbar_wait(&sh->acc_empty[buf], (uint32_t)(((si >> 1) & 1) ^ 1), sh, a.status, 45, (uint32_t)si));
                if (!ok) break;
                tc_fence_after();
                for (int ks = 0; ks < stages; ks++, it++) {
                    const int s = it & (WP_NB - 1), sa = it % WP_NA;
                    ok = __all_sync(0xffffffffu, mbar_wait_both(&sh->b_full[s], (uint32_t)((it / WP_NB) & 1), &sh->a_full[sa], (uint32_t)((it / WP_NA) & 1), sh,
                                                                    a.status, 46, (uint32_t)it));
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const uint64_t bd = bdesc0 + (uint64_t)(((uint32_t)s * WP_B_STAGE) >> 4);
                        const uint32_t at = tmem + WP_A_COL + (uint32_t)sa * WP_SLOT_COLS;
#pragma unroll
                        for (int g = 0; g < 2; g++)
#pragma unroll
                            for (int kk = 0; kk < 4; kk++)
                                mma_f16_ts_pair(acc, at + 32 * g + 8 * kk, bd + g * group_b + 2 * kk, idesc, ks > 0 || g > 0 || kk > 0 ? 1u : 0u);
                        mma_commit_pair(done_of[0] + (uint32_t)(it & 3) * 8u);
                        mma_commit_pair(done_of[1] + (uint32_t)(it & 3) * 8u);
                        if (ks == stages - 1) {
                            mma_commit_pair(cluster_addr(&sh->acc_full[buf], 0));
                            mma_commit_pair(cluster_addr(&sh->acc_full[buf], 1));
                        }
                    }
                    __syncwarp();
                }
            }
            if (!ok && it > 0) mbar_wait(&sh->done[(it - 1) & 3], (uint32_t)(((it - 1) >> 2) & 1), sh, a.status, 48, 0, false);  // what was issued completes
        }
    } else if (warp >= 16) {
        // ---------------- epilogue ----------------
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const uint32_t acc_lane = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        const uint32_t empty_even = cluster_addr(&sh->acc_empty[0], 0);
        const bool plain = !a.y_bf16 && a.n_more == 0;
        for (int si = 0; seg.next(a); si++) {
            const int buf = si & 1, row = seg.row + (int)rank * WP_ROWS + (warp & 3) * 32 + lane;
            auto factor = [&](int c) {  // of token c + lane
                return (PRE_SCALED ? 1.0f / WT_PRE : 1.0f) * (a.row_unscale && c + lane < seg.count ? __ldg(a.row_unscale + seg.x_row0 + c + lane) : 1.0f);
            };
            float next = factor(0);
            if (!__all_sync(0xffffffffu, mbar_wait(&sh->acc_full[buf], (uint32_t)((si >> 1) & 1), sh, a.status, 49, (uint32_t)si) && !sh->abort_flag)) break;
            tc_fence_after();
            // (a loop of one chunk: unrolled over the segment it is 24 KB of code that runs once a segment, at the rate of its instruction
            // fetches, 15000 cycles)
#pragma unroll 1
            for (int c = 0; c < seg.n; c += 32) {
                const float f = next;
                next = factor(c + 32);
                uint32_t v[32];
                tmem_ld32(acc_lane + (uint32_t)(buf * WP_SEG + c), v);
                const size_t at = (size_t)(seg.x_row0 + c) * a.y_ld + row;
                const int live = row < a.n_out ? seg.count - c : 0;  // tokens to store
                if (plain) {
                    float* o = (float*)a.y + at;
#pragma unroll
                    for (int j = 0; j < 32; j++, o += a.y_ld) {
                        const float w = __uint_as_float(v[j]) * __shfl_sync(0xffffffffu, f, j);
                        if (j < live) *o = w;
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 32; j++) {
                        const float w = __uint_as_float(v[j]) * __shfl_sync(0xffffffffu, f, j);
                        const size_t o = at + (size_t)j * a.y_ld;
                        if (j < live) {
                            if (a.y_bf16)
                                ((__nv_bfloat16*)a.y)[o] = __float2bfloat16_rn(w);
                            else
                                ((float*)a.y)[o] = w;
                            for (int d = 0; d < a.n_more; d++) a.more[d][o] = w;
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_remote(empty_even + (uint32_t)buf * 8u);
        }
    } else {
        // ---------------- dequantizers ----------------
        const int set = warp >> 2, r = (warp & 3) * 32 + lane;
        const uint32_t swz = (uint32_t)(r & 7), swh = (uint32_t)((r >> 1) & 3);
        const uint32_t a_lane = tmem + WP_A_COL + ((uint32_t)((warp & 3) * 32) << 16);
        const uint32_t full_even = cluster_addr(&sh->a_full[0], 0);
        bool ok = true;
        // 64 expanded weights, group g of the segment whose first stage is it0, to this lane of tensor memory
        auto put = [&](int it0, int g, const uint32_t(&o)[32]) {
            const int it = it0 + (g >> 1), old = it - WP_NA, sa = it % WP_NA;
            if (old >= 0) ok = __all_sync(0xffffffffu, mbar_wait(&sh->done[old & 3], (uint32_t)((old >> 2) & 1), sh, a.status, 50, (uint32_t)it));
            if (!ok) return;
            tc_fence_after();
            tmem_st32(a_lane + (uint32_t)sa * WP_SLOT_COLS + (uint32_t)(g & 1) * 32u, o);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_remote(full_even + (uint32_t)sa * 8u);
        };
        auto raw_ready = [&](int slot, int ph, int c) {
            ok = __all_sync(0xffffffffu, mbar_wait(&sh->raw_full[slot], (uint32_t)ph, sh, a.status, 51, (uint32_t)c));
            return ok;
        };
        int it0 = 0, slot = 0, ph = 0, base = 0;
        for (; ok && seg.next(a); it0 += stages) {
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
                uint32_t next = scales_of(set);
                for (int g = set; g < groups; g += 4) {
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
                    expand_4bit<FMT, false>(hdr, qw, set, o);
                    put(it0, sb * 4 + set, o);
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

bool gemm_wp_encode(GemmWp* g, const WeightDev& w, size_t experts, const void* x16, size_t x_rows) {
    GemmWt m;  // the weights' maps are gemm_wt.cu's (boxes of 128 rows)
    if (!gemm_wt_encode(&m, w, experts, x16, x_rows, 16, 1, 0, false, false)) return false;
    g->w = m.w;
    g->w2 = m.w2;
    return gemm_x_maps(&g->x, 0, WP_SEG / 32 - 1, x16, x_rows, w.n_in, 2);
}

cudaError_t launch_gemm_wp(const GemmWp& g, const WeightDev& w, size_t t, const WtTile* tiles, int n_tiles, void* y, int y_dtype, size_t y_ld, float* const* more, int n_more,
                           GemmStatus* status, int sm_count, const float* row_unscale, cudaStream_t st) {
    using Kern = void (*)(XMaps, CUtensorMap, CUtensorMap, WpArgs);
    Kern kern = w.fmt == B2_FMT_Q6_K     ? gemm_wp_kernel<B2_FMT_Q6_K>
                : w.fmt == B2_FMT_Q8_0   ? gemm_wp_kernel<B2_FMT_Q8_0>
                : w.fmt == B2_FMT_MLX4   ? gemm_wp_kernel<B2_FMT_MLX4>
                : w.fmt == B2_FMT_F8E4M3 ? gemm_wp_kernel<B2_FMT_F8E4M3>
                                         : gemm_wp_kernel<B2_FMT_Q4_K>;
    const size_t smem = wp_smem(w.fmt);
    if (cudaError_t e = ensure_dynamic_smem((const void*)kern, smem, 0); e != cudaSuccess) return e;
    WpArgs a{};
    a.K = (int)w.n_in;
    a.n_out = (int)w.n_out;
    a.t = (int)t;
    a.y_bf16 = y_dtype == B2_BF16;
    a.y_ld = y_ld;
    a.y = y;
    a.status = status;
    a.tiles = tiles;
    a.n_tiles = n_tiles;
    a.row_unscale = row_unscale;
    a.s = (const float*)(w.fmt == B2_FMT_Q6_K ? w.p2 : w.p1);
    a.s2 = w.p3;
    a.f8_rows = w.fmt == B2_FMT_F8E4M3 ? (int)w.bs_rows : 1;
    a.f8_ncb = w.fmt == B2_FMT_Q8_0 ? (int)(w.n_in / 32) : (int)w.bs_ncb;
    a.f8_row0 = (int)w.bs_row0;
    a.n_more = n_more;
    for (int i = 0; i < n_more; i++) a.more[i] = more[i];
    const size_t blocks = (w.n_out + 2 * WP_ROWS - 1) / (2 * WP_ROWS);
    const size_t units = tiles ? blocks * (size_t)n_tiles : blocks * ((t + WP_UNIT - 1) / WP_UNIT);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(2 * std::min<size_t>(units, (size_t)std::max(1, sm_count / 2))));
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
    return cudaLaunchKernelEx(&cfg, kern, g.x, g.w, g.w2, a);
}

}  // namespace b2
