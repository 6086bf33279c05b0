// Dequant-GEMM with the weights in tensor memory and the tokens on the instruction's N side (tcgen05): dense batches of up to 128 tokens,
// and the routed experts' segments of any length.
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
#include <cuda_fp8.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>

#include "gemm_wt.h"
#include "tcgen05.cuh"

namespace b2 {

namespace {

constexpr int WT_THREADS = 352;
constexpr int WT_ROWS = 128;
constexpr uint32_t WT_TMEM_COLS = 256, WT_SLOT_COLS = 64;  // the accumulator, 64 or 128 columns, and the A ring behind it
constexpr int WT_MAX_RING = 8;
constexpr size_t WT_SMEM_MAX = 113 * 1024, WT_SMEM_MIN = 77 * 1024;

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
    int groups;           // 64-k groups of a stage: 1 or 2 (two-term weights: 1)
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
__device__ __forceinline__ bool elect_one() {  // true in one lane of a whole warp
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, "
        "%21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]),
        "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]),
        "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ __half2 as_h2(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }
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

// 64 weights of a 4-bit block: 32 bytes, low nibbles = elements 0..31, high nibbles = 32..63 (see gemm_tc.cu for the arithmetic).
// hdr: the block's 16 bytes in front; j: which of its four groups of 64. LO (Q4_K): the second term, the exact f32 weight minus the
// first term.
template <int FMT, bool LO>
__device__ __forceinline__ void expand_4bit(const uint4& hdr, const uint32_t (&qw)[8], int j, uint32_t (&o)[32]) {
    __half2 dmul, c1lo, c2lo, c1hi, c2hi, addlo, addhi;
    uint32_t sc0 = 0, mn0 = 0, sc1 = 0, mn1 = 0;
    if constexpr (FMT == B2_FMT_MLX4) {
        const uint32_t sw = (j & 2) ? hdr.y : hdr.x, bw = (j & 2) ? hdr.w : hdr.z;
        dmul = __half2half2(__ushort_as_half((unsigned short)((sw >> (16 * (j & 1))) & 0xffffu)));
        c1lo = __float2half2_rn(1.0f);
        c2lo = __float2half2_rn(-1032.0f);
        c1hi = __float2half2_rn(0.0625f);
        c2hi = __float2half2_rn(-72.0f);
        addlo = addhi = __float2half2_rn(bf16_bits_to_f32((bw >> (16 * (j & 1))) & 0xffffu));
    } else {
        q4k_scale_min(2 * j, hdr.y, hdr.z, hdr.w, sc0, mn0);
        q4k_scale_min(2 * j + 1, hdr.y, hdr.z, hdr.w, sc1, mn1);
        const float dmin = __half2float(__ushort_as_half((unsigned short)(hdr.x >> 16)));
        dmul = __half2half2(__ushort_as_half((unsigned short)(hdr.x & 0xffff)));
        c1lo = __float2half2_rn((float)sc0);
        c2lo = __float2half2_rn(-1024.0f * (float)sc0);
        c1hi = __float2half2_rn(0.0625f * (float)sc1);
        c2hi = __float2half2_rn(-64.0f * (float)sc1);
        addlo = __float2half2_rn(-(dmin * (float)mn0));
        addhi = __float2half2_rn(-(dmin * (float)mn1));
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t p0 = __byte_perm(qw[i], 0, 0x4140), p1 = __byte_perm(qw[i], 0, 0x4342);
        o[2 * i] = h2_bits(__hfma2(__hfma2(as_h2((p0 & 0x000F000Fu) | 0x64006400u), c1lo, c2lo), dmul, addlo));
        o[2 * i + 1] = h2_bits(__hfma2(__hfma2(as_h2((p1 & 0x000F000Fu) | 0x64006400u), c1lo, c2lo), dmul, addlo));
        o[16 + 2 * i] = h2_bits(__hfma2(__hfma2(as_h2((p0 & 0x00F000F0u) | 0x64006400u), c1hi, c2hi), dmul, addhi));
        o[16 + 2 * i + 1] = h2_bits(__hfma2(__hfma2(as_h2((p1 & 0x00F000F0u) | 0x64006400u), c1hi, c2hi), dmul, addhi));
    }
    if constexpr (LO) {
        const float d = __half2float(__ushort_as_half((unsigned short)(hdr.x & 0xffff)));
        const float dmin = __half2float(__ushort_as_half((unsigned short)(hdr.x >> 16)));
        const float d1l = __fmul_rn(d, (float)sc0), m1l = __fmul_rn(dmin, (float)mn0);
        const float d1h = __fmul_rn(d, (float)sc1), m1h = __fmul_rn(dmin, (float)mn1);
#pragma unroll
        for (int i = 0; i < 8; i++) {
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const uint32_t b0 = (qw[i] >> (16 * e)) & 0xffu, b1 = (qw[i] >> (16 * e + 8)) & 0xffu;
                const float2 hl = __half22float2(as_h2(o[2 * i + e])), hh = __half22float2(as_h2(o[16 + 2 * i + e]));
                const float vl0 = __fsub_rn(__fmul_rn(d1l, __uint_as_float(0x4B000000u | (b0 & 15u)) - 8388608.0f), m1l);
                const float vl1 = __fsub_rn(__fmul_rn(d1l, __uint_as_float(0x4B000000u | (b1 & 15u)) - 8388608.0f), m1l);
                const float vh0 = __fsub_rn(__fmul_rn(d1h, __uint_as_float(0x4B000000u | (b0 >> 4)) - 8388608.0f), m1h);
                const float vh1 = __fsub_rn(__fmul_rn(d1h, __uint_as_float(0x4B000000u | (b1 >> 4)) - 8388608.0f), m1h);
                o[2 * i + e] = h2_bits(__floats2half2_rn(vl0 - hl.x, vl1 - hl.y));
                o[16 + 2 * i + e] = h2_bits(__floats2half2_rn(vh0 - hh.x, vh1 - hh.y));
            }
        }
    }
}

// W2 (Q4_K): every weight as two f16 terms; set 0 expands the first terms of every stage, set 1 the second.
template <int FMT, bool W2>
__global__ void __launch_bounds__(WT_THREADS, 2)
gemm_wt_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_w2,
               const __grid_constant__ WtArgs a) {
    // A dependent launch: the weights, their expansion and the set-up run under the kernel ahead; the activations, the row factors and y
    // wait for it.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    constexpr bool BYTE_ROWS = FMT == B2_FMT_F8E4M3 || FMT == B2_FMT_Q8_0;
    constexpr bool PRE_SCALED = BYTE_ROWS || FMT == B2_FMT_Q6_K;
    constexpr float PRE = 256.0f;                       // power of two in the f16 weights of these formats
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
            mbar_init(&sh->a_full[s], W2 ? 8 : 4 * a.groups);
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
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_x) : "memory");
            const uint32_t bytes = (uint32_t)(n * 128 * a.x_terms * a.groups);
            asm volatile("griddepcontrol.wait;" ::: "memory");
            int issued = 0;
            for (int ks = 0, s = 0; ks < nks; ks++) {
                const int old = ks - a.n_b;  // the stage whose slot this one takes
                if (old >= 0 && !mbar_wait(&sh->done[old & 3], (uint32_t)((old >> 2) & 1), sh, a.status, 21, (uint32_t)ks)) break;
                mbar_arrive_expect_tx(&sh->b_full[s], bytes);
                uint8_t* dst = b_tiles + (size_t)s * b_stage;  // [group][term][n][64]
                for (int i = 0; i < a.groups * a.x_terms; i++, dst += (size_t)n * 128) {
                    const int term = a.x_terms == 2 ? i & 1 : 0, g = a.x_terms == 2 ? i >> 1 : i;
                    const int kx = (sb0 * SB_G + ks * a.groups + g) * 64, y = x_row0 + term * a.lo_row0;
                    if (!a.tiles) {
                        tma_load_2d(dst, &tmap_x, &sh->b_full[s], kx, y);
                        continue;
                    }
                    int r = 0;  // grouped: whole boxes of 64 tokens, then of 16
                    for (; r + 64 <= n; r += 64) tma_load_2d(dst + (size_t)r * 128, &tmap_w2, &sh->b_full[s], kx, y + r);
                    for (; r < n; r += 16) tma_load_2d(dst + (size_t)r * 128, &tmap_x, &sh->b_full[s], kx, y + r);
                }
                issued = ks + 1;
                if (++s == a.n_b) s = 0;
            }
            if (sh->abort_flag)  // copies in flight land before the shared memory goes away
                for (int ks = max(0, issued - a.n_b); ks < issued; ks++)
                    mbar_wait(&sh->b_full[ks % a.n_b], (uint32_t)((ks / a.n_b) & 1), sh, a.status, 22, (uint32_t)ks, false);
        }
    } else if (warp == 10) {
        // ---------------- packed weights ----------------
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_w) : "memory");
            const int copies = BYTE_ROWS ? 2 * nsb : nsb;
            int issued = 0;
            for (int c = 0, s = 0, ph = 0; c < copies; c++) {
                if (!mbar_wait(&sh->raw_empty[s], (uint32_t)(ph ^ 1), sh, a.status, 23, (uint32_t)c)) break;
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
                issued = c + 1;
                if (++s == a.n_raw) s = 0, ph ^= 1;
            }
            if (sh->abort_flag)
                for (int c = max(0, issued - a.n_raw); c < issued; c++)
                    mbar_wait(&sh->raw_full[c % a.n_raw], (uint32_t)((c / a.n_raw) & 1), sh, a.status, 24, (uint32_t)c, false);
        }
    } else if (warp == 9) {
        // ---------------- instructions ----------------
        // The warp stays together: every lane waits, one elected lane issues (in a branch of one lane the four instructions and the
        // commit of 64 k take 550 cycles, this way 250).
        const uint32_t idesc = (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((128u >> 4) << 24);
        const uint64_t bdesc0 = smem_desc_sw128(smem_u32(b_tiles));
        const uint32_t lo = (uint32_t)(n * 128) >> 4;  // the second term's tile, in descriptor units
        bool ok = true;
        for (int ks = 0, sa = 0, pa = 0, s = 0, ph = 0; ks < nks; ks++) {
            ok = __all_sync(0xffffffffu, mbar_wait(&sh->b_full[s], (uint32_t)ph, sh, a.status, 25, (uint32_t)ks) &&
                                             mbar_wait(&sh->a_full[sa], (uint32_t)pa, sh, a.status, 26, (uint32_t)ks));
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
                        if (W2) mma_f16_ts(tmem, ag + 32 + 8 * kk, bg + 2 * kk, idesc, 1u);  // (second terms of both: below f32's rounding)
                    }
                };
                group(at, bdesc, ks == 0);
                if (a.groups == 2) group(at + 32, bdesc + lo * (uint32_t)a.x_terms, false);
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
            tmem_st32(a_lane + (uint32_t)slot_a * WT_SLOT_COLS + ((W2 ? set : g - ks * a.groups) ? 32u : 0u), o);
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
                if constexpr (FMT == B2_FMT_Q8_0) {
                    const __half2 m0 = __float2half2_rn(__half2float(__ushort_as_half((unsigned short)(sc & 0xffffu))) * PRE);
                    const __half2 m1 = __float2half2_rn(__half2float(__ushort_as_half((unsigned short)(sc >> 16))) * PRE);
                    const __half2 bias = __float2half2_rn(1152.0f);  // 1024 under the exponent byte 0x64, and 128
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        const uint32_t wds[4] = {q[c].x, q[c].y, q[c].z, q[c].w};
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const uint32_t u = wds[i] ^ 0x80808080u;
                            o[8 * c + 2 * i] = h2_bits(__hmul2(__hsub2(as_h2(__byte_perm(u, 0x64646464u, 0x4140)), bias), c < 2 ? m0 : m1));
                            o[8 * c + 2 * i + 1] = h2_bits(__hmul2(__hsub2(as_h2(__byte_perm(u, 0x64646464u, 0x4342)), bias), c < 2 ? m0 : m1));
                        }
                    }
                } else {
                    const __half2 sc2 = __float2half2_rn((a.s ? __uint_as_float(sc) : 1.0f) * PRE);
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        const uint32_t wds[4] = {q[c].x, q[c].y, q[c].z, q[c].w};
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            __half2_raw h01 = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(wds[i] & 0xffff), __NV_E4M3);
                            __half2_raw h23 = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(wds[i] >> 16), __NV_E4M3);
                            o[8 * c + 2 * i] = h2_bits(__hmul2(*reinterpret_cast<__half2*>(&h01), sc2));
                            o[8 * c + 2 * i + 1] = h2_bits(__hmul2(*reinterpret_cast<__half2*>(&h23), sc2));
                        }
                    }
                }
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
                const uint32_t qlw[16] = {ql4[0].x, ql4[0].y, ql4[0].z, ql4[0].w, ql4[1].x, ql4[1].y, ql4[1].z, ql4[1].w,
                                          ql4[2].x, ql4[2].y, ql4[2].z, ql4[2].w, ql4[3].x, ql4[3].y, ql4[3].z, ql4[3].w};
                const uint32_t qhw[8] = {qh4[0].x, qh4[0].y, qh4[0].z, qh4[0].w, qh4[1].x, qh4[1].y, qh4[1].z, qh4[1].w};
                const __half2 bias = __float2half2_rn(1056.0f);  // 1024 under the exponent byte 0x64, and 32
#pragma unroll
                for (int odd = 0; odd < 2; odd++) {
                    __half2 mul[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) mul[i] = __float2half2_rn(d * (float)(int8_t)(sc8[odd] >> (8 * i)) * PRE);
                    uint32_t o[32];
#pragma unroll
                    for (int i = 0; i < 16; i++) {  // word i: elements 4 i .. 4 i + 3 of the group
                        const uint32_t nib = odd ? (qlw[i] >> 4) & 0x0F0F0F0Fu : qlw[i] & 0x0F0F0F0Fu;
                        const int at = 4 * odd + 2 * (i >> 3);  // the bit pair's place in its byte; it goes to bits 4 and 5
                        const uint32_t hb = (at < 4 ? qhw[i & 7] << (4 - at) : qhw[i & 7] >> (at - 4)) & 0x30303030u;
                        const uint32_t q4 = nib | hb;
                        o[2 * i] = h2_bits(__hmul2(__hsub2(as_h2(__byte_perm(q4, 0x64646464u, 0x4140)), bias), mul[i >> 2]));
                        o[2 * i + 1] = h2_bits(__hmul2(__hsub2(as_h2(__byte_perm(q4, 0x64646464u, 0x4342)), bias), mul[i >> 2]));
                    }
                    put(sb * 4 + 2 * set + odd, o);
                    if (!ok) break;
                }
            }
        } else {
            // one-term: set s expands groups s and s + 2 of every super-block; two-term: both sets all four groups
            constexpr int GROUPS = W2 ? 4 : 2;
            int slot = 0, ph = 0;
            for (int sb = 0; sb < nsb && ok; sb++) {
                if (!raw_ready(slot, ph, sb)) break;
                const uint4* my = (const uint4*)(raw + (size_t)slot * RAW_SLOT + (size_t)r * 144);
                const uint4 hdr = my[0];
                uint4 q[2 * GROUPS];
                uint32_t words = hdr.x;
#pragma unroll
                for (int i = 0; i < 2 * GROUPS; i++) {
                    q[i] = my[1 + (W2 ? i : 2 * set + 4 * (i >> 1) + (i & 1))];
                    words |= q[i].x;
                }
                release_raw(&sh->raw_empty[slot], words, a.zero, lane);
                if (++slot == a.n_raw) slot = 0, ph ^= 1;
#pragma unroll
                for (int jj = 0; jj < GROUPS; jj++) {
                    const uint32_t qw[8] = {q[2 * jj].x,     q[2 * jj].y,     q[2 * jj].z,     q[2 * jj].w,
                                            q[2 * jj + 1].x, q[2 * jj + 1].y, q[2 * jj + 1].z, q[2 * jj + 1].w};
                    uint32_t o[32];
                    if (W2 && set)
                        expand_4bit<FMT, W2>(hdr, qw, jj, o);
                    else
                        expand_4bit<FMT, false>(hdr, qw, W2 ? jj : 2 * jj + set, o);
                    put(sb * 4 + (W2 ? jj : 2 * jj + set), o);
                    if (!ok) break;
                }
            }
        }
        // ---------------- sums out of tensor memory ----------------
        const bool acc_ok = __all_sync(0xffffffffu, mbar_wait(&sh->acc_full, 0, sh, a.status, 30, 0) && !sh->abort_flag);
        if (acc_ok) {
            tc_fence_after();
            asm volatile("griddepcontrol.wait;" ::: "memory");
            const uint32_t acc = tmem + ((uint32_t)((warp & 3) * 32) << 16);
            float* sums = (float*)smem;  // parts of K: [token][128 rows], over the rings, which are idle now
            const bool plain = !a.y_bf16 && a.n_more == 0;
            for (int c = set * 16; c < n; c += 32) {
                uint32_t v[16];
                tmem_ld16(acc + (uint32_t)c, v);
                if (a.splits > 1) {
#pragma unroll
                    for (int i = 0; i < 16; i++) sums[(c + i) * WT_ROWS + r] = __uint_as_float(v[i]);
                    continue;
                }
                float f[16];
#pragma unroll
                for (int i = 0; i < 16; i++)
                    f[i] = (PRE_SCALED ? 1.0f / PRE : 1.0f) * (a.row_unscale && c + i < count ? __ldg(a.row_unscale + x_row0 + c + i) : 1.0f);
                if (live) {
                    const size_t at = (size_t)(x_row0 + c) * a.y_ld + n0 + r;
                    if (plain) {
                        float* o = (float*)a.y + at;
#pragma unroll
                        for (int i = 0; i < 16; i++)
                            if (c + i < count) o[(size_t)i * a.y_ld] = __uint_as_float(v[i]) * f[i];
                    } else {
#pragma unroll
                        for (int i = 0; i < 16; i++)
                            if (c + i < count) store_y(a, at + (size_t)i * a.y_ld, __uint_as_float(v[i]) * f[i]);
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
            const bool vec = !a.y_bf16 && a.n_more == 0 && (a.y_ld & 3) == 0 && ((uintptr_t)a.y & 15) == 0 && row + 4 <= a.n_out;
            for (int tok = part * 8 + warp; tok < count; tok += 8 * a.splits) {
                const uint32_t at = sums + (uint32_t)(tok * WT_ROWS + 4 * lane) * 4u;
                const float f = (PRE_SCALED ? 1.0f / PRE : 1.0f) * (a.row_unscale ? __ldg(a.row_unscale + x_row0 + tok) : 1.0f);
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
                    *(float4*)((float*)a.y + o) = make_float4(v.x * f, v.y * f, v.z * f, v.w * f);
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

bool gemm_wt_encode(GemmWt* g, const WeightDev& w, size_t experts, const void* x16, size_t x_rows, size_t tokens, int x_terms, size_t lo_row0, bool two_term_w, bool grouped) {
    TensorMapEncodeFn enc = tensor_map_encode();
    if (!enc) return false;
    if (grouped && w.fmt != B2_FMT_MLX4 && w.fmt != B2_FMT_Q4_K) return false;  // (w2 is then the longer box of x)
    g->n_max = (int)std::min<size_t>(128, (tokens + 15) / 16 * 16);
    g->splits = grouped ? 1 : wt_splits(w.n_in);
    g->x_terms = x_terms;
    g->lo_row0 = (int)lo_row0;
    g->two_term_w = two_term_w;
    auto x_map = [&](CUtensorMap* m, int box) {
        return encode_2d(enc, m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, x16, w.n_in, x_rows, w.n_in * 2, 64, (uint32_t)box, CU_TENSOR_MAP_SWIZZLE_128B);
    };
    CUresult r = x_map(&g->x, grouped ? 16 : g->n_max);
    const size_t rows = w.n_out * experts;
    const CUtensorMapDataType u8 = CU_TENSOR_MAP_DATA_TYPE_UINT8;
    if (r != CUDA_SUCCESS) return false;
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
        if (r == CUDA_SUCCESS && grouped) r = x_map(&g->w2, 64);
    }
    if (r != CUDA_SUCCESS) return false;
    // The rings in what two CTAs per SM leave: stages of 128 k (a stage costs the issuing warp about 400 cycles besides its instructions)
    // unless two of them do not fit, then packed weights from what is left, at least two slots (four of 64 k).
    const bool bytes = w.fmt == B2_FMT_F8E4M3 || w.fmt == B2_FMT_Q8_0;
    const size_t slot = raw_slot_bytes(w.fmt), tile = (size_t)g->n_max * 128 * x_terms, room = WT_SMEM_MAX - sizeof(WtShared) - 128 - 1024;
    const int least = bytes ? 4 : 2, most = bytes ? WT_MAX_RING : 5;
    g->groups = two_term_w || 4 * tile + (size_t)least * slot > room ? 1 : 2;
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
    using Kern = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, WtArgs);
    Kern kern = w.fmt == B2_FMT_Q6_K     ? gemm_wt_kernel<B2_FMT_Q6_K, false>
                : w.fmt == B2_FMT_Q8_0   ? gemm_wt_kernel<B2_FMT_Q8_0, false>
                : w.fmt == B2_FMT_MLX4   ? gemm_wt_kernel<B2_FMT_MLX4, false>
                : w.fmt == B2_FMT_F8E4M3 ? gemm_wt_kernel<B2_FMT_F8E4M3, false>
                : g.two_term_w           ? gemm_wt_kernel<B2_FMT_Q4_K, true>
                                         : gemm_wt_kernel<B2_FMT_Q4_K, false>;
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
