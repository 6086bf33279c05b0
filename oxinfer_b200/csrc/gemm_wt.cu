// Dequant-GEMM with the weights in tensor memory and the tokens on the instruction's N side (tcgen05): dense batches of up to 128 tokens, and
// MLX-4 experts under the exact switch (two-term activations; all other experts' segments run on gemm_wp.cu).
//
//   y[t][n_out] = x[t][K] * W^T
//
// One CTA multiplies 128 weight rows by n <= 128 tokens (n a multiple of 16, chosen per tile at run time) over one of `splits` parts of K:
//   warps 0..7 : dequantizers, a thread per weight row in each of two sets of four warps. A thread copies its row's packed bytes from the
//                staging ring to registers, expands 64 weights to f16 (the arithmetic of gemm_tc.cu) and writes them to its lane of tensor
//                memory (tcgen05.st): the A operand, a ring of two or three slots of 128 k. Then the epilogue.
//   warp 8     : copies the activations (f16, tiles of 64 k x n tokens, one or two terms) into a ring: the B operand.
//   warp 9     : allocates tensor memory and issues tcgen05.mma with A from tensor memory, M = 128 rows, N = n.
//   warp 10    : copies the packed weights into the staging ring.
// What bounds it: with tokens on M (gemm_tc.cu) a batch of 37 pays for 128, and every expanded weight is written to shared memory once and
// read by the tensor cores twice; shared memory then limits both. Here the tensor cores' work follows the token count in steps of
// 16, an expanded weight never touches shared memory, and two CTAs fit an SM, so that one's start and epilogue run under the other's loop.
//
// K is divided into parts by K alone (wt_splits), so that a row's bits depend neither on the other rows of its matrix nor on the batch
// beside it: row shards equal the unsharded rows. The parts of a tile are the CTAs of a cluster; each leaves its sums in its own
// shared memory, and the cluster adds them in the order of the parts, each CTA a share of the tokens.
//
// Tensor memory: a CTA takes 256 of the 512 columns and at least 77 KB of shared memory, so that no more than two CTAs of these kernels fit
// an SM and an allocation never waits for a CTA that itself waits for another CTA of its cluster.
#include <cuda.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>

#include "expand.cuh"
#include "gemm_wt.h"
#include "tcgen05.cuh"

namespace b2 {

namespace {

constexpr int WT_THREADS = 352;
constexpr int WT_ROWS = 128;
constexpr uint32_t WT_TMEM_COLS = 256, WT_SLOT_COLS = 64;  // the accumulator, 64 or 128 columns, and the A ring behind it
constexpr int WT_MAX_RING = 8;
constexpr size_t WT_SMEM_MAX = 113 * 1024, WT_SMEM_MIN = TMEM_256_SMEM;

struct __align__(8) WtShared {
    uint64_t a_full[4], b_full[4];
    uint64_t done[4];  // [stage % 4]: its instructions have completed, which frees its A slot and its B slot
    uint64_t raw_full[WT_MAX_RING], raw_empty[WT_MAX_RING];
    uint64_t acc_full;
    uint32_t tmem_base;
    volatile uint32_t abort_flag;
};

struct WtArgs {
    int K, n_out, t;
    int n_raw, n_b, n_a;  // slots of the two rings in shared memory and of the one in tensor memory
    int groups;           // 64-k groups of a stage: 1 or 2
    int splits;           // parts of K = CTAs of a cluster
    int n_max;            // the B ring's stage holds this many tokens
    int x_terms, lo_row0; // 2: activations as two f16 terms, the second lo_row0 rows below the first
    int y_bf16, zero;
    size_t y_ld;
    void* y;
    GemmStatus* status;
    const WtTile* tiles;  // grouped launches: one per blockIdx.y; null: token tiles of n_max
    const float* row_unscale;
    const float* s;       // scales beside the packed rows, as in gemm_tc.cu
    const void* s2;
    int f8_rows, f8_ncb, f8_row0;
    int n_more;           // other ranks' copies of y
    float* more[7];
};

__device__ __forceinline__ void mma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
        "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ void store_y(const WtArgs& a, size_t at, float v) {
    if (a.y_bf16) {
        ((__nv_bfloat16*)a.y)[at] = __float2bfloat16_rn(v);
        return;
    }
    ((float*)a.y)[at] = v;
    for (int d = 0; d < a.n_more; d++) a.more[d][at] = v;
}

template <int FMT>
__global__ void __launch_bounds__(WT_THREADS, 2)
gemm_wt_kernel(const __grid_constant__ XMaps maps, const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_w2,
               const __grid_constant__ WtArgs a) {
    // A dependent launch: the weights, their expansion and the set-up run under the kernel ahead; the activations, the row factors and y
    // wait for it.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    constexpr bool BYTE_ROWS = FMT == B2_FMT_F8E4M3 || FMT == B2_FMT_Q8_0;
    constexpr bool PRE_SCALED = BYTE_ROWS || FMT == B2_FMT_Q6_K;
    constexpr int SB_K = BYTE_ROWS ? 128 : 256;         // a super-block, what a part of K is a whole number of
    constexpr int SB_G = SB_K / 64;                     // groups of 64 k in a super-block
    constexpr int RAW_SLOT = BYTE_ROWS ? WT_ROWS * 64 : WT_ROWS * (FMT == B2_FMT_Q6_K ? 192 : 144);
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t b_stage = (uint32_t)(a.n_max * 128 * a.x_terms * a.groups);
    uint8_t* b_tiles = smem;
    uint8_t* raw = smem + (size_t)a.n_b * b_stage;
    __shared__ WtShared shared;
    WtShared* sh = &shared;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int part = a.splits > 1 ? (int)cluster_rank() : 0;
    const int n0 = (int)(blockIdx.x / (unsigned)a.splits) * WT_ROWS;
    const int nsb_all = a.K / SB_K;
    const int sb0 = part * nsb_all / a.splits, nsb = (part + 1) * nsb_all / a.splits - sb0;
    const int nks = nsb * SB_G / a.groups;              // stages
    int w_row0 = 0, x_row0, count;
    if (a.tiles) {
        const WtTile tile = a.tiles[blockIdx.y];
        w_row0 = tile.expert * a.n_out;
        x_row0 = tile.row0;
        count = tile.count;
    } else {
        x_row0 = (int)blockIdx.y * a.n_max;
        count = min(a.n_max, a.t - x_row0);
    }
    const int n = a.tiles ? (count + 15) & ~15 : a.n_max;  // (a dense tile is one copy of n_max rows, past the last token too)

    if (threadIdx.x == 0) {
        for (int s = 0; s < 4; s++) {
            mbar_init(&sh->a_full[s], 4 * a.groups);
            mbar_init(&sh->b_full[s], 1);
            mbar_init(&sh->done[s], 1);
        }
        for (int s = 0; s < WT_MAX_RING; s++) {
            mbar_init(&sh->raw_full[s], 1);
            mbar_init(&sh->raw_empty[s], BYTE_ROWS ? 4 : 8);
        }
        mbar_init(&sh->acc_full, 1);
        sh->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh->tmem_base)), "r"(WT_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh->tmem_base, a_cols = tmem + WT_TMEM_COLS - (uint32_t)a.n_a * WT_SLOT_COLS;

    if (warp == 8) {
        // ---------------- activations ----------------
        {
            const CUtensorMap* tmap_x = &maps.m[n / 16 - 1];
            asm volatile("prefetch.tensormap [%0];" ::"l"(tmap_x) : "memory");
            const uint32_t bytes = (uint32_t)(n * 128 * a.x_terms * a.groups);
            asm volatile("griddepcontrol.wait;" ::: "memory");
            int issued = 0;
            for (int ks = 0, s = 0; ks < nks; ks++) {
                const int old = ks - a.n_b;  // the stage whose slot this one takes
                if (old >= 0 && !__all_sync(0xffffffffu, mbar_wait(&sh->done[old & 3], (uint32_t)((old >> 2) & 1), sh, a.status, 21, (uint32_t)ks))) break;
                issued = ks + 1;
                if (elect_one()) {
                    mbar_arrive_expect_tx(&sh->b_full[s], bytes);
                    uint8_t* dst = b_tiles + (size_t)s * b_stage;  // [term][group][n][64]
                    for (int term = 0; term < a.x_terms; term++, dst += (size_t)n * 128 * a.groups)
                        tma_load_3d(dst, tmap_x, &sh->b_full[s], 0, x_row0 + term * a.lo_row0, sb0 * SB_G + ks * a.groups);
                }
                __syncwarp();
                if (++s == a.n_b) s = 0;
            }
            if (sh->abort_flag)  // copies in flight land before the shared memory goes away
                for (int ks = max(0, issued - a.n_b); ks < issued; ks++)
                    mbar_wait(&sh->b_full[ks % a.n_b], (uint32_t)((ks / a.n_b) & 1), sh, a.status, 22, (uint32_t)ks, false);
        }
    } else if (warp == 10) {
        // ---------------- packed weights ----------------
        {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_w) : "memory");
            const int copies = BYTE_ROWS ? 2 * nsb : nsb;
            int issued = 0;
            for (int c = 0, s = 0, ph = 0; c < copies; c++) {
                if (!__all_sync(0xffffffffu, mbar_wait(&sh->raw_empty[s], (uint32_t)(ph ^ 1), sh, a.status, 23, (uint32_t)c))) break;
                issued = c + 1;
                if (elect_one()) {
                    mbar_arrive_expect_tx(&sh->raw_full[s], (uint32_t)RAW_SLOT);
                    uint8_t* dst = raw + (size_t)s * RAW_SLOT;
                    if constexpr (FMT == B2_FMT_Q6_K) {  // [128][128] low nibbles, then [128][64] high bit pairs
                        tma_load_2d(dst, &tmap_w, &sh->raw_full[s], (sb0 + c) * 128, w_row0 + n0);
                        tma_load_2d(dst + WT_ROWS * 128, &tmap_w2, &sh->raw_full[s], (sb0 + c) * 64, w_row0 + n0);
                    } else if constexpr (BYTE_ROWS) {
                        tma_load_2d(dst, &tmap_w, &sh->raw_full[s], (sb0 * 2 + c) * 64, w_row0 + n0);
                    } else {
                        tma_load_2d(dst, &tmap_w, &sh->raw_full[s], (sb0 + c) * 144, w_row0 + n0);
                    }
                }
                __syncwarp();
                if (++s == a.n_raw) s = 0, ph ^= 1;
            }
            if (sh->abort_flag)
                for (int c = max(0, issued - a.n_raw); c < issued; c++)
                    mbar_wait(&sh->raw_full[c % a.n_raw], (uint32_t)((c / a.n_raw) & 1), sh, a.status, 24, (uint32_t)c, false);
        }
    } else if (warp == 9) {
        // ---------------- instructions ----------------
        const uint32_t idesc = (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((128u >> 4) << 24);
        const uint64_t bdesc0 = smem_desc_sw128(smem_u32(b_tiles));
        const uint32_t tile = (uint32_t)(n * 128) >> 4, lo = tile * (uint32_t)a.groups;  // a group's tile, the second terms: in descriptor units
        bool ok = true;
        for (int ks = 0, sa = 0, pa = 0, s = 0, ph = 0; ks < nks; ks++) {
            ok = __all_sync(0xffffffffu, mbar_wait_both(&sh->b_full[s], (uint32_t)ph, &sh->a_full[sa], (uint32_t)pa, sh, a.status, 25, (uint32_t)ks));
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
                const uint64_t bdesc = bdesc0 + (uint64_t)(((uint32_t)s * b_stage) >> 4);
                const uint32_t at = a_cols + (uint32_t)sa * WT_SLOT_COLS;
                auto group = [&](uint32_t ag, uint64_t bg, bool first) {
#pragma unroll
                    for (int kk = 0; kk < 4; kk++) {
                        mma_f16_ts(tmem, ag + 8 * kk, bg + 2 * kk, idesc, first && kk == 0 ? 0u : 1u);
                        if (a.x_terms == 2) mma_f16_ts(tmem, ag + 8 * kk, bg + lo + 2 * kk, idesc, 1u);
                    }
                };
                group(at, bdesc, ks == 0);
                if (a.groups == 2) group(at + 32, bdesc + tile, false);
                mma_commit(&sh->done[ks & 3]);
            }
            __syncwarp();
            if (++sa == a.n_a) sa = 0, pa ^= 1;
            if (++s == a.n_b) s = 0, ph ^= 1;
        }
        if (elect_one()) mma_commit(&sh->acc_full);
        __syncwarp();
        if (!ok) mbar_wait(&sh->acc_full, 0, sh, a.status, 27, 0, false);
    } else {
        // ---------------- dequantizers ----------------
        const int set = warp >> 2, r = (warp & 3) * 32 + lane;
        const uint32_t swz = (uint32_t)(r & 7), swh = (uint32_t)((r >> 1) & 3);
        const uint32_t a_lane = a_cols + ((uint32_t)((warp & 3) * 32) << 16);
        bool ok = true;
        // 64 expanded weights, group g of this part of K, to this lane of tensor memory (a set's groups come in ascending order)
        int slot_a = 0, stage_a = 0;
        auto put = [&](int g, const uint32_t(&o)[32]) {
            const int ks = a.groups == 2 ? g >> 1 : g, old = ks - a.n_a;
            while (stage_a < ks) {
                stage_a++;
                if (++slot_a == a.n_a) slot_a = 0;
            }
            if (old >= 0) ok = __all_sync(0xffffffffu, mbar_wait(&sh->done[old & 3], (uint32_t)((old >> 2) & 1), sh, a.status, 28, (uint32_t)ks));
            if (!ok) return;
            tc_fence_after();
            tmem_st32(a_lane + (uint32_t)slot_a * WT_SLOT_COLS + (g - ks * a.groups ? 32u : 0u), o);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh->a_full[slot_a]);
        };
        auto raw_ready = [&](int slot, int ph, int c) {
            ok = __all_sync(0xffffffffu, mbar_wait(&sh->raw_full[slot], (uint32_t)ph, sh, a.status, 29, (uint32_t)c));
            return ok;
        };
        const bool live = n0 + r < a.n_out;
        const size_t wrow = live ? (size_t)(n0 + r) : 0;
        if constexpr (BYTE_ROWS) {
            // group g belongs to set g % 2; the scales (Q8_0: two f16, FP8: one f32) a super-block ahead
            const uint8_t* sc_row = (const uint8_t*)a.s;
            if constexpr (FMT == B2_FMT_Q8_0)
                sc_row += (wrow * (size_t)a.f8_ncb + (size_t)sb0 * 4 + set * 2) * 2;
            else
                sc_row = a.s ? sc_row + ((wrow + a.f8_row0) / a.f8_rows * a.f8_ncb + sb0) * 4 : nullptr;
            auto scales_of = [&](int sb) {
                return live && sb < nsb && sc_row ? __ldg((const uint32_t*)(sc_row + (size_t)sb * (FMT == B2_FMT_Q8_0 ? 8 : 4))) : 0u;
            };
            uint32_t next = scales_of(0);
            int slot = set, ph = 0;  // (n_raw is even and at least 2)
            for (int sb = 0; sb < nsb; sb++) {
                const uint32_t sc = next;
                next = scales_of(sb + 1);
                const int g = 2 * sb + set;
                if (!raw_ready(slot, ph, g)) break;
                const uint4* my = (const uint4*)(raw + (size_t)slot * RAW_SLOT + (size_t)r * 64);
                uint4 q[4];
#pragma unroll
                for (int c = 0; c < 4; c++) q[c] = my[(uint32_t)c ^ swh];
                release_raw(&sh->raw_empty[slot], q[0].x | q[1].x | q[2].x | q[3].x, a.zero, lane);
                slot += 2;
                if (slot >= a.n_raw) slot -= a.n_raw, ph ^= 1;
                uint32_t o[32];
                if constexpr (FMT == B2_FMT_Q8_0)
                    expand_q8_0(q, sc, o);
                else
                    expand_f8(q, a.s ? __uint_as_float(sc) : 1.0f, o);
                put(g, o);
                if (!ok) break;
            }
        } else if constexpr (FMT == B2_FMT_Q6_K) {
            // set s expands half s of every super-block: groups 2 s (low nibbles) and 2 s + 1 (high nibbles) of its 64 ql and 32 qh bytes
            const uint8_t* sc_row = (const uint8_t*)a.s + wrow * (size_t)(a.K / 16) + (size_t)sb0 * 16 + 8 * set;
            const unsigned short* d_row = (const unsigned short*)a.s2 + wrow * (size_t)(a.K / 256) + sb0;
            uint32_t next_d = 0;
            uint2 next_sc = make_uint2(0u, 0u);
            auto load_scales = [&](int sb) {
                if (!live || sb >= nsb) return;
                next_d = __ldg(d_row + sb);
                next_sc = __ldg((const uint2*)(sc_row + (size_t)sb * 16));
            };
            load_scales(0);
            int slot = 0, ph = 0;
            for (int sb = 0; sb < nsb && ok; sb++) {
                const float d = __half2float(__ushort_as_half((unsigned short)next_d));
                const uint32_t sc8[2] = {next_sc.x, next_sc.y};
                load_scales(sb + 1);
                if (!raw_ready(slot, ph, sb)) break;
                const uint4* my = (const uint4*)(raw + (size_t)slot * RAW_SLOT + (size_t)r * 128);
                const uint4* my_qh = (const uint4*)(raw + (size_t)slot * RAW_SLOT + WT_ROWS * 128 + (size_t)r * 64);
                uint4 ql4[4], qh4[2];
#pragma unroll
                for (int c = 0; c < 4; c++) ql4[c] = my[((uint32_t)(4 * set + c)) ^ swz];
#pragma unroll
                for (int c = 0; c < 2; c++) qh4[c] = my_qh[((uint32_t)(2 * set + c)) ^ swh];
                release_raw(&sh->raw_empty[slot], ql4[0].x | ql4[1].x | ql4[2].x | ql4[3].x | qh4[0].x | qh4[1].x, a.zero, lane);
                if (++slot == a.n_raw) slot = 0, ph ^= 1;
#pragma unroll
                for (int odd = 0; odd < 2; odd++) {
                    uint32_t o[32];
                    expand_q6k(ql4, qh4, d, sc8[odd], odd, o);
                    put(sb * 4 + 2 * set + odd, o);
                    if (!ok) break;
                }
            }
        } else {
            // set s expands groups s and s + 2 of every super-block
            constexpr int GROUPS = 2;
            int slot = 0, ph = 0;
            for (int sb = 0; sb < nsb && ok; sb++) {
                if (!raw_ready(slot, ph, sb)) break;
                const uint4* my = (const uint4*)(raw + (size_t)slot * RAW_SLOT + (size_t)r * 144);
                const uint4 hdr = my[0];
                uint4 q[2 * GROUPS];
                uint32_t words = hdr.x;
#pragma unroll
                for (int i = 0; i < 2 * GROUPS; i++) {
                    q[i] = my[1 + 2 * set + 4 * (i >> 1) + (i & 1)];
                    words |= q[i].x;
                }
                release_raw(&sh->raw_empty[slot], words, a.zero, lane);
                if (++slot == a.n_raw) slot = 0, ph ^= 1;
#pragma unroll
                for (int jj = 0; jj < GROUPS; jj++) {
                    const uint32_t qw[8] = {q[2 * jj].x,     q[2 * jj].y,     q[2 * jj].z,     q[2 * jj].w,
                                            q[2 * jj + 1].x, q[2 * jj + 1].y, q[2 * jj + 1].z, q[2 * jj + 1].w};
                    uint32_t o[32];
                    expand_4bit<FMT>(hdr, qw, 2 * jj + set, o);
                    put(sb * 4 + 2 * jj + set, o);
                    if (!ok) break;
                }
            }
        }
        // ---------------- sums out of tensor memory ----------------
        asm volatile("griddepcontrol.wait;" ::: "memory");
        // The row factors of this set's tokens, 16 of every 32, two lanes a token, are asked for ahead of the sums. (Chunk by chunk behind them, bf16
        // rows: Q6_K 4096 x 1024, 128 tokens 16.1 us, this way 13.5; 64 tokens 11.0 and 9.5.)
        float fac[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int tok = 32 * i + set * 16 + (lane & 15);
            fac[i] = (PRE_SCALED ? 1.0f / WT_PRE : 1.0f) * (a.splits == 1 && a.row_unscale && tok < count ? __ldg(a.row_unscale + x_row0 + tok) : 1.0f);
        }
        const bool acc_ok = __all_sync(0xffffffffu, mbar_wait(&sh->acc_full, 0, sh, a.status, 30, 0) && !sh->abort_flag);
        if (acc_ok) {
            tc_fence_after();
            const uint32_t acc = tmem + ((uint32_t)((warp & 3) * 32) << 16);
            float* sums = (float*)smem;  // parts of K: [token][128 rows], over the rings, which are idle now
            const bool plain = !a.y_bf16 && a.n_more == 0;
#pragma unroll
            for (int chunk = 0; chunk < 4; chunk++) {
                const int c = 32 * chunk + set * 16;
                if (c >= n) break;
                uint32_t v[16];
                tmem_ld16(acc + (uint32_t)c, v);
                if (a.splits > 1) {
#pragma unroll
                    for (int i = 0; i < 16; i++) sums[(c + i) * WT_ROWS + r] = __uint_as_float(v[i]);
                    continue;
                }
#pragma unroll
                for (int i = 0; i < 16; i++) v[i] = __float_as_uint(__uint_as_float(v[i]) * __shfl_sync(0xffffffffu, fac[chunk], i));
                if (live) {
                    const size_t at = (size_t)(x_row0 + c) * a.y_ld + n0 + r;
                    if (plain) {
                        float* o = (float*)a.y + at;
#pragma unroll
                        for (int i = 0; i < 16; i++)
                            if (c + i < count) o[(size_t)i * a.y_ld] = __uint_as_float(v[i]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 16; i++)
                            if (c + i < count) store_y(a, at + (size_t)i * a.y_ld, __uint_as_float(v[i]));
                    }
                }
                __syncwarp();
            }
        }
    }
    if (a.splits > 1) {
        // ---------------- the parts, added in order: this CTA's share of the tokens ----------------
        __syncwarp();
        cluster_sync_all();
        if (warp < 8 && !sh->abort_flag) {
            const uint32_t sums = smem_u32(smem);
            const int row = n0 + 4 * lane;
            const bool vec = !a.y_bf16 && (a.y_ld & 3) == 0 && ((uintptr_t)a.y & 15) == 0 && row + 4 <= a.n_out;  // (other ranks' copies are aligned as y)
            for (int tok = part * 8 + warp; tok < count; tok += 8 * a.splits) {
                const uint32_t at = sums + (uint32_t)(tok * WT_ROWS + 4 * lane) * 4u;
                const float f = (PRE_SCALED ? 1.0f / WT_PRE : 1.0f) * (a.row_unscale ? __ldg(a.row_unscale + x_row0 + tok) : 1.0f);
                float4 u[8];
#pragma unroll
                for (int p = 0; p < 8; p++) {
                    if (p >= a.splits) break;
                    uint32_t peer;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(at), "r"(p));
                    u[p] = ld_cluster_f4(peer);
                }
                float4 v = u[0];
#pragma unroll
                for (int p = 1; p < 8; p++) {
                    if (p >= a.splits) break;
                    v.x += u[p].x;
                    v.y += u[p].y;
                    v.z += u[p].z;
                    v.w += u[p].w;
                }
                const size_t o = (size_t)(x_row0 + tok) * a.y_ld + row;
                if (vec) {
                    const float4 w = make_float4(v.x * f, v.y * f, v.z * f, v.w * f);
                    *(float4*)((float*)a.y + o) = w;
                    for (int d = 0; d < a.n_more; d++) *(float4*)(a.more[d] + o) = w;
                } else {
                    const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        if (row + i < a.n_out) store_y(a, o + i, e[i] * f);
                }
            }
        }
        __syncwarp();
        cluster_sync_all();  // no CTA leaves while another reads its sums
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 9) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(WT_TMEM_COLS) : "memory");
    }
}

size_t raw_slot_bytes(int fmt) {
    return (size_t)WT_ROWS * (fmt == B2_FMT_F8E4M3 || fmt == B2_FMT_Q8_0 ? 64 : fmt == B2_FMT_Q6_K ? 192 : 144);
}

CUresult encode_2d(TensorMapEncodeFn enc, CUtensorMap* m, CUtensorMapDataType type, const void* base, size_t inner, size_t rows, size_t stride, uint32_t box_x,
                   uint32_t box_y, CUtensorMapSwizzle swizzle) {
    cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)stride};
    cuuint32_t box[2] = {box_x, box_y};
    cuuint32_t estr[2] = {1, 1};
    return enc(m, type, 2, (void*)base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
}

}  // namespace

// The parts have at least 1536 k: a CTA's start (about 4000 cycles until the first weights arrive) and the exchange of the sums (3000)
// cost as much as 1000 k of its loop. 14336 x 4096 with parts of 1024: Q6_K, 37 tokens, 34.9 us, of 2048: 25.6.
int wt_splits(size_t K) {
    int s = 1;
    while (s < 8 && K / (size_t)(2 * s) >= 1536) s *= 2;
    return s;
}

bool gemm_x_maps(XMaps* x, int first, int last, const void* x16, size_t rows, size_t n_in, int groups) {
    TensorMapEncodeFn enc = tensor_map_encode();
    cuuint64_t dims[3] = {64, (cuuint64_t)rows, (cuuint64_t)(n_in / 64)};
    cuuint64_t strides[2] = {(cuuint64_t)n_in * 2, 128};
    cuuint32_t estr[3] = {1, 1, 1};
    for (int i = first; enc && i <= last; i++) {
        cuuint32_t box[3] = {64, (cuuint32_t)(16 * (i + 1)), (cuuint32_t)groups};
        if (enc(&x->m[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, (void*)x16, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return false;
    }
    return enc != nullptr;
}

bool gemm_wt_encode(GemmWt* g, const WeightDev& w, size_t experts, const void* x16, size_t x_rows, size_t tokens, int x_terms, size_t lo_row0, bool grouped) {
    TensorMapEncodeFn enc = tensor_map_encode();
    if (!enc) return false;
    g->n_max = (int)std::min<size_t>(128, (tokens + 15) / 16 * 16);
    g->splits = grouped ? 1 : wt_splits(w.n_in);
    g->x_terms = x_terms;
    g->lo_row0 = (int)lo_row0;
    CUresult r;
    const size_t rows = w.n_out * experts;
    const CUtensorMapDataType u8 = CU_TENSOR_MAP_DATA_TYPE_UINT8;
    if (w.fmt == B2_FMT_Q6_K) {
        r = encode_2d(enc, &g->w, u8, w.p0, w.n_in / 2, rows, w.n_in / 2, 128, WT_ROWS, CU_TENSOR_MAP_SWIZZLE_128B);
        if (r == CUDA_SUCCESS) r = encode_2d(enc, &g->w2, u8, w.p1, w.n_in / 4, rows, w.n_in / 4, 64, WT_ROWS, CU_TENSOR_MAP_SWIZZLE_64B);
    } else if (w.fmt == B2_FMT_F8E4M3 || w.fmt == B2_FMT_Q8_0) {
        r = encode_2d(enc, &g->w, u8, w.p0, w.n_in, rows, w.n_in, 64, WT_ROWS, CU_TENSOR_MAP_SWIZZLE_64B);
        g->w2 = g->w;
    } else {
        const size_t row = w.n_in / 256 * 144;
        r = encode_2d(enc, &g->w, u8, w.p0, row, rows, row, 144, WT_ROWS, CU_TENSOR_MAP_SWIZZLE_NONE);
        g->w2 = g->w;
    }
    if (r != CUDA_SUCCESS) return false;
    // The rings in what two CTAs per SM leave: stages of 128 k (a stage costs the issuing warp about 400 cycles besides its instructions)
    // unless two of them do not fit, then packed weights from what is left, at least two slots (four of 64 k).
    const bool bytes = w.fmt == B2_FMT_F8E4M3 || w.fmt == B2_FMT_Q8_0;
    const size_t slot = raw_slot_bytes(w.fmt), tile = (size_t)g->n_max * 128 * x_terms, room = WT_SMEM_MAX - sizeof(WtShared) - 128 - 1024;
    const int least = bytes ? 4 : 2, most = bytes ? WT_MAX_RING : 5;
    g->groups = 4 * tile + (size_t)least * slot > room ? 1 : 2;
    if (!gemm_x_maps(&g->x, grouped ? 0 : g->n_max / 16 - 1, g->n_max / 16 - 1, x16, x_rows, w.n_in, g->groups)) return false;
    g->n_a = g->n_max <= 64 ? 3 : 2;
    g->n_b = (int)std::min<size_t>(4, (room - (size_t)least * slot) / (tile * g->groups));
    if (g->n_b < 2) return false;
    g->n_raw = (int)std::min<size_t>(most, (room - (size_t)g->n_b * tile * g->groups) / slot);
    if (bytes) g->n_raw &= ~1;
    g->smem = std::max({1024 + (size_t)g->n_b * tile * g->groups + (size_t)g->n_raw * slot, 1024 + (size_t)(g->splits > 1 ? g->n_max * WT_ROWS * 4 : 0), WT_SMEM_MIN});
    return true;
}

cudaError_t launch_gemm_wt(const GemmWt& g, const WeightDev& w, size_t t, const WtTile* tiles, int n_tiles, void* y, int y_dtype, size_t y_ld, float* const* more, int n_more,
                           GemmStatus* status, const float* row_unscale, cudaStream_t st) {
    using Kern = void (*)(XMaps, CUtensorMap, CUtensorMap, WtArgs);
    Kern kern = w.fmt == B2_FMT_Q6_K     ? gemm_wt_kernel<B2_FMT_Q6_K>
                : w.fmt == B2_FMT_Q8_0   ? gemm_wt_kernel<B2_FMT_Q8_0>
                : w.fmt == B2_FMT_MLX4   ? gemm_wt_kernel<B2_FMT_MLX4>
                : w.fmt == B2_FMT_F8E4M3 ? gemm_wt_kernel<B2_FMT_F8E4M3>
                                         : gemm_wt_kernel<B2_FMT_Q4_K>;
    if (cudaError_t e = ensure_dynamic_smem((const void*)kern, g.smem, 0); e != cudaSuccess) return e;
    WtArgs a{};
    a.K = (int)w.n_in;
    a.n_out = (int)w.n_out;
    a.t = (int)t;
    a.n_raw = g.n_raw;
    a.n_b = g.n_b;
    a.n_a = g.n_a;
    a.groups = g.groups;
    a.splits = g.splits;
    a.n_max = g.n_max;
    a.x_terms = g.x_terms;
    a.lo_row0 = g.lo_row0;
    a.y_bf16 = y_dtype == B2_BF16;
    a.y_ld = y_ld;
    a.y = y;
    a.status = status;
    a.tiles = tiles;
    a.row_unscale = row_unscale;
    a.s = (const float*)(w.fmt == B2_FMT_Q6_K ? w.p2 : w.p1);
    a.s2 = w.p3;
    a.f8_rows = w.fmt == B2_FMT_F8E4M3 ? (int)w.bs_rows : 1;
    a.f8_ncb = w.fmt == B2_FMT_Q8_0 ? (int)(w.n_in / 32) : (int)w.bs_ncb;
    a.f8_row0 = (int)w.bs_row0;
    a.n_more = n_more;
    for (int i = 0; i < n_more; i++) a.more[i] = more[i];
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)((w.n_out + WT_ROWS - 1) / WT_ROWS * (size_t)g.splits), (unsigned)(tiles ? (size_t)n_tiles : (t + g.n_max - 1) / g.n_max));
    cfg.blockDim = dim3(WT_THREADS);
    cfg.dynamicSmemBytes = g.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2] = {};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)g.splits;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g.splits > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kern, g.x, g.w, g.w2, a);
}

}  // namespace b2
