// Small-batch dequant products (1 .. 8 tokens) on the integer tensor path: device code of gemv_mma.cu.
//
// A warp multiplies 16 weight rows by blocks of k with mma.m16n8k32 (u8 or s8 x s8 -> s32): A = the packed integers of the weights under
// a mask, B = the digits of the activation split (split.cuh), four columns per token (three digits and one spare), two tokens to the
// eight columns of an instruction. The sums are exact; a format's integer scales multiply them in integers, its float scales once per
// block (per 32 / 64 values where they are floats). Up to two tokens cost what one costs, so a step of four reads and unpacks the
// weights once and pays two instructions where one token pays one. Columns that no token owns repeat another's and are never stored.
//
// The kernels are bound by instruction issue: at the HBM rate an SM has 3.1 warp instructions per 4-bit weight and lane. The dp4a form
// this replaced took 3.2; mma.m16n8k16 on f16 operands 2.6; this takes about 1.5 (Q4_K, one token).
#pragma once
#include <cuda_fp8.h>

#include "split.cuh"

namespace b2 {
namespace gmma {

#define B2_MMA_K32(NAME, TYPES)                                                                                                                     \
    __device__ __forceinline__ void NAME(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {               \
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32." TYPES ".s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"          \
                     : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])                                                                               \
                     : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));                                                                       \
    }                                                                                                                                               \
    __device__ __forceinline__ void NAME##_0(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {           \
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32." TYPES ".s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"      \
                     : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])                                                                               \
                     : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));                                                               \
    }
B2_MMA_K32(mma_us, "u8.s8")   // unsigned weights
B2_MMA_K32(mma_ss, "s8.s8")   // signed weights
#undef B2_MMA_K32
// sixteen k, from zero
__device__ __forceinline__ void mma_ss16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%7, %7, %7, %7};"
                 : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
                 : "r"(a0), "r"(a1), "r"(b0), "r"(0));
}
__device__ __forceinline__ void mma_us16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.u8.s8.s32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%7, %7, %7, %7};"
                 : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
                 : "r"(a0), "r"(a1), "r"(b0), "r"(0));
}
__device__ __forceinline__ float half_lo(uint32_t w) { return __half2float(__ushort_as_half((unsigned short)(w & 0xffffu))); }
__device__ __forceinline__ float half_hi(uint32_t w) { return __half2float(__ushort_as_half((unsigned short)(w >> 16))); }
// Shared memory by 32-bit address. Volatile: the loads of a slot stay ahead of the copies that refill it.
__device__ __forceinline__ uint32_t lds32(uint32_t p) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(p) : "memory");
    return v;
}
__device__ __forceinline__ float ldsf(uint32_t p) { return __uint_as_float(lds32(p)); }
__device__ __forceinline__ uint2 lds64(uint32_t p) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t p) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(p) : "memory");
    return v;
}

// 16 / 4 bytes global -> shared without passing through registers.
__device__ __forceinline__ void cp16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp4(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp16z(uint32_t dst, const void* src, bool live) {  // zeros where it is not live
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16u : 0u) : "memory");
}
__device__ __forceinline__ void cp4z(uint32_t dst, const void* src, bool live) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(live ? 4u : 0u) : "memory");
}
// from zero
__device__ __forceinline__ void mma_f16_0(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
                 : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// The activations of the CTA in shared memory for TP token places (1, 4 or 8), as this lane reads them.
// Digits: lane (g, t) feeds column g of an instruction (token g / 4 of its pair, digit g % 4) and holds the sums of columns 2 t and
// 2 t + 1: token t / 2 of the pair, digits 0 and 1 (t even) or 2 and (of four) 3 (t odd).
// Halves: column g is token g / 2 of its four, hi or lo; lane t holds both of token t.
template <int TP, bool HALVES, int DIGITS = 3>
struct XView {
    static constexpr int PER = HALVES ? 4 : 2;               // tokens of an instruction
    static constexpr int NT = (TP + PER - 1) / PER;          // instructions for all of them
    static constexpr uint32_t TOKEN = HALVES ? 128 : 64 * DIGITS;  // bytes of a token in a chunk of 32 k (halves) or a pair of chunks (digits)
    static constexpr uint32_t STEP = TOKEN * TP;             // from one such to the next
    static constexpr uint32_t NEXT = TOKEN * PER;            // from an instruction's tokens to the next one's
    static constexpr uint32_t BLOCK = HALVES ? SPLIT_HALVES : DIGITS * 256;
    static constexpr int COLUMNS = DIGITS;                   // of a token that carry digits; a fourth one repeats the third where there are three
    static constexpr uint32_t SUMS = HALVES ? 0 : 32;        // bytes of a (block, token) in `sums`
    static constexpr int RES = 16 * (TP == 1 ? 1 : NT * PER);  // results of a tile of 16 rows
    uint32_t frag;   // this lane's first B fragment
    uint32_t xs;     // block scale of this lane's token, block 0; blocks are TP floats apart
    uint32_t sums;   // this lane's sums of block 0 (the format's kind, see put_sums)
};

// ---- Q4_K and the repacked MLX-4: 144-byte blocks of 256 --------------------------------------------------------------------------
// SIGNED (MLX-4): a weight is 16 (n - 8), its group's offset goes into the low digits' sums alone; the arithmetic of gemv_tc.cu. Otherwise n, with 8 d less in the
// offsets: 15 % more error (their sums are larger than the result), 3 to 4 % less time for the routed experts, whose groups keep it.
template <bool MLX, bool SIGNED>
struct F4 {
    template <int TP>
    using X = XView<TP, false>;
    // IN_PAIRS: four slices' sums are added as gemv_tc.cu adds its four parts', so that a launch of several jobs there has the same bits (gemv_tc_jobs_supports).
    static constexpr bool HALVES = false, SUMS = true, PARTS = true, IN_PAIRS = true;
    static constexpr int BLOCK_K = 256, SLOTS = 2, MAX_BLOCKS = 2;  // a unit is one or two blocks
    static constexpr int BLOCK_BYTES = 16 * 144, UNIT_BYTES = MAX_BLOCKS * BLOCK_BYTES;
    static constexpr bool SUMS_BY_COLUMN = !MLX;
    // The chunk sums of a (block, token) in shared memory (32 bytes); s: the sum of chunk `lane` (lanes 0 .. 7 hold them).
    //   MLX: four sums of 64 times the block scale (f32).
    //   Q4_K: the sums in signed digits, [digit 0 .. 3][chunk], the B fragment of the instruction that multiplies them by the mins.
    __device__ static __forceinline__ void put_sums(uint8_t* e, float xs, int s, int lane) {
        if (MLX) {
            const int o = __shfl_xor_sync(0xffffffffu, s, 1);
            if (lane < 8 && (lane & 1) == 0) ((float*)e)[lane >> 1] = xs * (float)(s + o);
        } else if (lane < 8) {
            const uint32_t b = (uint32_t)(s + (int)0x80808080u) ^ 0x80808080u;  // |s| < 2^28
#pragma unroll
            for (int d = 0; d < 4; d++) e[8 * d + lane] = (uint8_t)(b >> (8 * d));
        }
    }
    __device__ static __forceinline__ uint32_t tag(const WeightDev&, const WeightDev&, size_t, size_t, int) { return 0; }
    // A slot holds [block][16 rows][144 bytes]. The tile's rows come as two halves of eight (each with a first row of its own, the
    // pair form's from two matrices); a lane's places in a half are the same for both.
    template <bool PAIR>
    struct Copy {
        const uint8_t *p0, *p1;
        uint32_t off[5], dst[5], row_bytes;
        int n;  // places of this lane
        __device__ __forceinline__ void init(const WeightDev& w, int blocks, int lane) {
            row_bytes = (uint32_t)(w.n_in / 256) * 144;
            n = blocks == 2 ? (lane < 16 ? 5 : 4) : (lane < 8 ? 3 : 2);
#pragma unroll
            for (int i = 0; i < 5; i++) {
                const int q = lane + 32 * i, blk = q / 72, in = q - 72 * blk, row = in / 9;
                off[i] = (uint32_t)min(row, (int)min((size_t)7, w.n_out - 1)) * row_bytes + (uint32_t)(blk * 144 + (in - 9 * row) * 16);
                dst[i] = (uint32_t)(blk * BLOCK_BYTES + in * 16);
            }
        }
        __device__ __forceinline__ void tile(const WeightDev& w, const WeightDev& w2, size_t r0, size_t r1, int) {
            p0 = w.p0 + r0 * row_bytes;
            p1 = (PAIR ? w2.p0 : w.p0) + r1 * row_bytes;
        }
        // `one`: the second block of the unit does not exist
        __device__ __forceinline__ void issue(uint32_t slot, int b, bool one, int) const {
            const uint32_t at = (uint32_t)b * 144;
#pragma unroll
            for (int i = 0; i < 5; i++) {
                if (i >= 2 && (i >= n || (one && dst[i] >= BLOCK_BYTES))) break;
                cp16(slot + dst[i], p0 + (at + off[i]));
                cp16(slot + dst[i] + 8 * 144, p1 + (at + off[i]));
            }
        }
    };
    // acc[n][row g | g + 8]: this lane's share (its two columns) of the results
    template <int TP>
    __device__ static __forceinline__ void block(uint32_t slot, int u, uint32_t, const WeightDev&, const WeightDev&, const X<TP>& x, int g, int t, float (&acc)[X<TP>::NT][2]) {
        constexpr int NT = X<TP>::NT;
        const uint32_t ra = slot + g * 144, rb = ra + 8 * 144;
        const uint4 ha = lds128(ra), hb = lds128(rb);
        uint32_t sa[2], sb[2];
        if (!MLX) {  // the eight 6-bit scales of a row as bytes (get_scale_min_k4, src/ggml.rs:501-509)
            sa[0] = ha.y & 0x3f3f3f3fu;
            sa[1] = (ha.w & 0x0f0f0f0fu) | ((ha.y >> 2) & 0x30303030u);
            sb[0] = hb.y & 0x3f3f3f3fu;
            sb[1] = (hb.w & 0x0f0f0f0fu) | ((hb.y >> 2) & 0x30303030u);
        }
        const uint32_t xf = x.frag + (uint32_t)u * (4 * X<TP>::STEP);
        const float w0 = (t & 1) ? 65536.0f : 1.0f, w1 = (t & 1) ? 0.0f : 256.0f;  // what this lane's two digits stand for
        int lo[NT][4], hi[NT][4];    // Q4_K: the chunks' sums times their scales; the high nibbles' are 16 times too large
        float f[NT][2];              // MLX: the groups' sums times d
#pragma unroll
        for (int n = 0; n < NT; n++) {
            f[n][0] = f[n][1] = 0.0f;
#pragma unroll
            for (int i = 0; i < 4; i++) lo[n][i] = hi[n][i] = 0;
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {  // groups of 64: chunk 2 j in the low nibbles, 2 j + 1 in the high ones
            const uint32_t a0 = lds32(ra + 16 + 32 * j + 4 * t), a2 = lds32(ra + 32 + 32 * j + 4 * t);
            const uint32_t a1 = lds32(rb + 16 + 32 * j + 4 * t), a3 = lds32(rb + 32 + 32 * j + 4 * t);
            constexpr uint32_t L = 0x0F0F0F0Fu, H = 0xF0F0F0F0u;
#pragma unroll
            for (int n = 0; n < NT; n++) {
                const uint4 b = lds128(xf + j * X<TP>::STEP + n * X<TP>::NEXT);
                int c[4], e[4];
                if (SIGNED) {
                    constexpr uint32_t M = 0x80808080u;
                    mma_ss_0(c, ((a0 << 4) & H) ^ M, ((a1 << 4) & H) ^ M, ((a2 << 4) & H) ^ M, ((a3 << 4) & H) ^ M, b.x, b.y);
                    mma_ss(c, (a0 & H) ^ M, (a1 & H) ^ M, (a2 & H) ^ M, (a3 & H) ^ M, b.z, b.w);
                } else {
                    mma_us_0(c, a0 & L, a1 & L, a2 & L, a3 & L, b.x, b.y);
                    mma_us_0(e, a0 & H, a1 & H, a2 & H, a3 & H, b.z, b.w);
                }
                if (MLX) {
                    const uint32_t da = j < 2 ? ha.x : ha.y, db = j < 2 ? hb.x : hb.y;
                    const float dA = (j & 1) ? half_hi(da) : half_lo(da), dB = (j & 1) ? half_hi(db) : half_lo(db);
#pragma unroll
                    for (int i = 0; i < 4 && !SIGNED; i++) c[i] = 16 * c[i] + e[i];
                    f[n][0] = fmaf(dA, fmaf((float)c[1], w1, (float)c[0] * w0), f[n][0]);
                    f[n][1] = fmaf(dB, fmaf((float)c[3], w1, (float)c[2] * w0), f[n][1]);
                } else {
                    const int s0 = (int)((sa[j >> 1] >> (16 * (j & 1))) & 0xffu), s1 = (int)((sa[j >> 1] >> (16 * (j & 1) + 8)) & 0xffu);
                    const int r0 = (int)((sb[j >> 1] >> (16 * (j & 1))) & 0xffu), r1 = (int)((sb[j >> 1] >> (16 * (j & 1) + 8)) & 0xffu);
                    lo[n][0] += s0 * c[0];
                    lo[n][1] += s0 * c[1];
                    lo[n][2] += r0 * c[2];
                    lo[n][3] += r0 * c[3];
                    hi[n][0] += s1 * e[0];
                    hi[n][1] += s1 * e[1];
                    hi[n][2] += r1 * e[2];
                    hi[n][3] += r1 * e[3];
                }
            }
        }
        if (MLX) {  // w = (n - 8) d + off per 64: off - 8 d times the sums of 64; a token's two lanes take two groups each
#pragma unroll
            for (int n = 0; n < NT; n++) {
                const float xs = ldsf(x.xs + (u * TP + 2 * n) * 4) * 0.0625f;
                if constexpr (SIGNED) {
                    const uint4 s = lds128(x.sums + (u * TP + 2 * n) * 32 - (t & 1) * 8);
                    const float s0 = __uint_as_float(s.x), s1 = __uint_as_float(s.y), s2 = __uint_as_float(s.z), s3 = __uint_as_float(s.w);
#pragma unroll
                    for (int r = 0; r < 2; r++) {
                        const uint2 o = r ? make_uint2(hb.z, hb.w) : make_uint2(ha.z, ha.w);
                        float v = fmaf(xs, f[n][r], acc[n][r]);
                        if (!(t & 1)) {
                            v = fmaf(__uint_as_float(o.x << 16), s0, v);
                            v = fmaf(__uint_as_float(o.x & 0xffff0000u), s1, v);
                            v = fmaf(__uint_as_float(o.y << 16), s2, v);
                            v = fmaf(__uint_as_float(o.y & 0xffff0000u), s3, v);
                        }
                        acc[n][r] = v;
                    }
                    continue;
                }
                const uint2 s = lds64(x.sums + (u * TP + 2 * n) * 32);
                const float s0 = __uint_as_float(s.x), s1 = __uint_as_float(s.y);
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const uint4 h = r ? hb : ha;
                    const uint32_t d = (t & 1) ? h.y : h.x, o = (t & 1) ? h.w : h.z;
                    float v = fmaf(xs, f[n][r], acc[n][r]);
                    v = fmaf(fmaf(-8.0f, half_lo(d), __uint_as_float(o << 16)), s0, v);
                    acc[n][r] = fmaf(fmaf(-8.0f, half_hi(d), __uint_as_float(o & 0xffff0000u)), s1, v);
                }
            }
        } else {
            // the mins: eight values of 6 bits times the chunk sums' digits
            const uint32_t ma = t == 0 ? ha.z & 0x3f3f3f3fu : t == 1 ? ((ha.w >> 4) & 0x0f0f0f0fu) | ((ha.z >> 2) & 0x30303030u) : 0u;
            const uint32_t mb = t == 0 ? hb.z & 0x3f3f3f3fu : t == 1 ? ((hb.w >> 4) & 0x0f0f0f0fu) | ((hb.z >> 2) & 0x30303030u) : 0u;
            const float dA = 0.0625f * half_lo(ha.x), mA = half_hi(ha.x), dB = 0.0625f * half_lo(hb.x), mB = half_hi(hb.x);
            const float m1 = (t & 1) ? 16777216.0f : 256.0f;
#pragma unroll
            for (int n = 0; n < NT; n++) {
                int e[4];
                mma_us16(e, ma, mb, lds32(x.sums + (u * TP + 2 * n) * 32));
                const float xs = ldsf(x.xs + (u * TP + 2 * n) * 4);
#pragma unroll
                for (int i = 0; i < 4; i++) lo[n][i] = 16 * lo[n][i] + hi[n][i];
                const float pa = fmaf((float)lo[n][1], w1, (float)lo[n][0] * w0), pb = fmaf((float)lo[n][3], w1, (float)lo[n][2] * w0);
                const float qa = fmaf((float)e[1], m1, (float)e[0] * w0), qb = fmaf((float)e[3], m1, (float)e[2] * w0);
                acc[n][0] = fmaf(xs, fmaf(dA, pa, -(mA * qa)), acc[n][0]);
                acc[n][1] = fmaf(xs, fmaf(dB, pb, -(mB * qb)), acc[n][1]);
            }
        }
    }
};

// ---- Q8_0: int8 rows and an f16 scale per 32; FP8: e4m3 rows and an f32 scale per 128 columns of a block of rows --------------------
// Blocks of 128 k. A slot holds [block][16 rows][144 bytes]: 128 weights, then four f16 scales (Q8_0) or one f32 (FP8).
// FP8: every instruction sums its 16 k from zero and its sums are added in f32. The instruction does not round to nearest when it adds to
// an accumulator: chained over a block's eight, a gate / up pair of N(0, 1) activations was 1.72e-7 of its norm from the f64 pair at
// K = 1024 and 1.95e-7 at 14336 (an f32 kernel 1.55e-7 and 2.04e-7), this way 1.48e-7 and 1.77e-7, at half a percent of a decoder
// step's time (a lone product of 4096 x 4096: 5.8 -> 5.9 us). A third f16 term of the activations would take another 0.1e-7 off and a
// sixth of the speed of two to four tokens.
template <bool FP8>
struct F8B {
    template <int TP>
    using X = XView<TP, FP8>;
    static constexpr bool HALVES = FP8, SUMS = false, SUMS_BY_COLUMN = false, PARTS = true, IN_PAIRS = false;
    static constexpr int BLOCK_K = 128, SLOTS = 2, MAX_BLOCKS = 2;
    static constexpr int BLOCK_BYTES = 16 * 144, UNIT_BYTES = MAX_BLOCKS * BLOCK_BYTES;
    __device__ static __forceinline__ void put_sums(uint8_t*, float, int, int) {}
    __device__ static __forceinline__ uint32_t tag(const WeightDev&, const WeightDev&, size_t, size_t, int) { return 0; }
    template <bool PAIR>
    struct Copy {
        const uint8_t *p0, *p1, *s0, *s1;
        size_t K;
        uint32_t rl, srow;   // this lane's row of the scales (limited to the matrix); bytes of a row of scales
        int rows, blocks;
        bool scaled;
        __device__ __forceinline__ void init(const WeightDev& w, int bpu, int lane) {
            K = w.n_in;
            rows = (int)min((size_t)8, w.n_out);
            blocks = bpu;
            scaled = w.p1 != nullptr;
            // Q8_0: lane = (row, block of the unit, 4-byte word of its scales); FP8: (row, block of the unit) for lanes below 16
            rl = (uint32_t)min(FP8 ? (lane >> 1) & 7 : lane >> 2, rows - 1);
            srow = FP8 ? (uint32_t)w.bs_ncb * 4 : (uint32_t)(K / 32) * 2;
        }
        __device__ __forceinline__ void tile(const WeightDev& w, const WeightDev& w2, size_t r0, size_t r1, int) {
            const WeightDev& o = PAIR ? w2 : w;
            p0 = w.p0 + r0 * K;
            p1 = o.p0 + r1 * K;
            if (FP8) {
                if (scaled) {
                    s0 = w.p1 + (w.bs_row0 + r0 + rl) / w.bs_rows * srow;
                    s1 = o.p1 + (o.bs_row0 + r1 + rl) / o.bs_rows * srow;
                }
            } else {
                s0 = w.p1 + (r0 + rl) * srow;
                s1 = o.p1 + (r1 + rl) * srow;
            }
        }
        __device__ __forceinline__ void issue(uint32_t slot, int b, bool, int lane) const {
            const uint32_t k0 = (uint32_t)b * 128;
#pragma unroll
            for (int i = 0; i < 4; i++) {  // half a tile's rows: 8 x (16 or 8) pieces of 16 bytes
                if (i >= 2 && blocks == 1) break;
                const int q = lane + 32 * i, row = blocks == 2 ? q >> 4 : q >> 3, c = blocks == 2 ? q & 15 : q & 7;
                const uint32_t k = k0 + c * 16, dst = slot + (c >> 3) * BLOCK_BYTES + row * 144 + (c & 7) * 16;
                const size_t at = (size_t)min(row, rows - 1) * K + k;
                cp16z(dst, p0 + at, k < K);
                cp16z(dst + 8 * 144, p1 + at, k < K);
            }
            if (FP8) {
                const int blk = lane & 1, row = (lane >> 1) & 7;
                if (scaled && lane < 16 && blk < blocks) {
                    const uint32_t k = k0 + blk * 128, dst = slot + blk * BLOCK_BYTES + row * 144 + 128;
                    cp4z(dst, s0 + k / 32, k < K);  // (four bytes per 128 k)
                    cp4z(dst + 8 * 144, s1 + k / 32, k < K);
                }
            } else {
                const int row = lane >> 2, blk = (lane >> 1) & 1, half = lane & 1;
                if (blk < blocks) {
                    const uint32_t k = k0 + blk * 128 + half * 64, dst = slot + blk * BLOCK_BYTES + row * 144 + 128 + half * 4;
                    cp4z(dst, s0 + k / 16, k < K);  // (two bytes per 32 k)
                    cp4z(dst + 8 * 144, s1 + k / 16, k < K);
                }
            }
        }
    };
    template <int TP>
    __device__ static __forceinline__ void block(uint32_t slot, int u, uint32_t, const WeightDev& w, const WeightDev&, const X<TP>& x, int g, int t, float (&acc)[X<TP>::NT][2]) {
        constexpr int NT = X<TP>::NT;
        const uint32_t ra = slot + g * 144, rb = ra + 8 * 144;
        if constexpr (FP8) {
            const uint32_t xf = x.frag + (uint32_t)u * (4 * X<TP>::STEP);
            float c[NT][2][4];
#pragma unroll
            for (int n = 0; n < NT; n++)
#pragma unroll
                for (int i = 0; i < 4; i++) c[n][0][i] = c[n][1][i] = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; j++) {  // chunks of 32: two instructions of 16 k
                uint32_t a[2][4];
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int r = 0; r < 2; r++) {
                        const uint32_t v = lds32((r ? rb : ra) + 32 * j + 16 * h + 4 * t);
                        const __half2_raw l = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(v & 0xffff), __NV_E4M3);
                        const __half2_raw m = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(v >> 16), __NV_E4M3);
                        a[h][r] = *(const uint32_t*)&l;
                        a[h][2 + r] = *(const uint32_t*)&m;
                    }
#pragma unroll
                for (int n = 0; n < NT; n++) {
                    const uint4 b = lds128(xf + j * X<TP>::STEP + n * X<TP>::NEXT);
                    float e0[4], e1[4];
                    mma_f16_0(e0, a[0][0], a[0][1], a[0][2], a[0][3], b.x, b.y);
                    mma_f16_0(e1, a[1][0], a[1][1], a[1][2], a[1][3], b.z, b.w);
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        c[n][0][i] += e0[i];
                        c[n][1][i] += e1[i];
                    }
                }
            }
            const float sA = w.p1 ? ldsf(ra + 128) : 1.0f, sB = w.p1 ? ldsf(rb + 128) : 1.0f;
#pragma unroll
            for (int n = 0; n < NT; n++) {
                const float xs = ldsf(x.xs + ((u >> 1) * TP + 4 * n) * 4);
                acc[n][0] = fmaf(sA * xs, (c[n][0][0] + c[n][1][0]) + (c[n][0][1] + c[n][1][1]), acc[n][0]);
                acc[n][1] = fmaf(sB * xs, (c[n][0][2] + c[n][1][2]) + (c[n][0][3] + c[n][1][3]), acc[n][1]);
            }
        } else {
            const uint32_t xf = x.frag + (uint32_t)u * (2 * X<TP>::STEP);
            const float w0 = (t & 1) ? 65536.0f : 1.0f, w1 = (t & 1) ? 0.0f : 256.0f;  // what this lane's two digits stand for
            const uint2 da = lds64(ra + 128), db = lds64(rb + 128);
            float f[NT][2];
#pragma unroll
            for (int n = 0; n < NT; n++) f[n][0] = f[n][1] = 0.0f;
#pragma unroll
            for (int j = 0; j < 2; j++) {  // pairs of chunks
                uint32_t a[2][4];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    a[h][0] = lds32(ra + 64 * j + 32 * h + 4 * t);
                    a[h][1] = lds32(rb + 64 * j + 32 * h + 4 * t);
                    a[h][2] = lds32(ra + 64 * j + 32 * h + 16 + 4 * t);
                    a[h][3] = lds32(rb + 64 * j + 32 * h + 16 + 4 * t);
                }
                const uint32_t dj = j ? da.y : da.x, ej = j ? db.y : db.x;
                const float d0 = half_lo(dj), d1 = half_hi(dj), e0 = half_lo(ej), e1 = half_hi(ej);
#pragma unroll
                for (int n = 0; n < NT; n++) {
                    const uint4 b = lds128(xf + j * X<TP>::STEP + n * X<TP>::NEXT);
                    int c[4], e[4];
                    mma_ss_0(c, a[0][0], a[0][1], a[0][2], a[0][3], b.x, b.y);
                    mma_ss_0(e, a[1][0], a[1][1], a[1][2], a[1][3], b.z, b.w);
                    f[n][0] = fmaf(d0, fmaf((float)c[1], w1, (float)c[0] * w0), f[n][0]);
                    f[n][1] = fmaf(e0, fmaf((float)c[3], w1, (float)c[2] * w0), f[n][1]);
                    f[n][0] = fmaf(d1, fmaf((float)e[1], w1, (float)e[0] * w0), f[n][0]);
                    f[n][1] = fmaf(e1, fmaf((float)e[3], w1, (float)e[2] * w0), f[n][1]);
                }
            }
#pragma unroll
            for (int n = 0; n < NT; n++) {
                const float xs = ldsf(x.xs + ((u >> 1) * TP + 2 * n) * 4);
                acc[n][0] = fmaf(xs, f[n][0], acc[n][0]);
                acc[n][1] = fmaf(xs, f[n][1], acc[n][1]);
            }
        }
    }
};

// ---- Q6_K: planes of low nibbles, high bit pairs, int8 scales per 16 and an f16 scale per 256 ----------------------------------------
// A slot holds [16 rows][208 bytes: 128 of nibbles, 64 of bit pairs, 16 scales], then a word per row that holds its f16 scale in one half.
struct F6 {
    template <int TP>
    using X = XView<TP, false>;
    static constexpr bool HALVES = false, SUMS = false, SUMS_BY_COLUMN = false, PARTS = true, IN_PAIRS = false;
    static constexpr int BLOCK_K = 256, SLOTS = 3, MAX_BLOCKS = 1;
    static constexpr int BLOCK_BYTES = 16 * 208 + 64, UNIT_BYTES = BLOCK_BYTES;
    __device__ static __forceinline__ void put_sums(uint8_t*, float, int, int) {}
    template <bool PAIR>
    struct Copy {
        const uint8_t *l0, *l1, *h0, *h1, *c0, *c1;  // this lane's first piece of each plane
        const uint16_t *d0, *d1;                     // this lane's row of the f16 scales
        uint32_t ldk;                                // bytes between this lane's two pieces of the nibble plane
        __device__ __forceinline__ void init(const WeightDev& w, int, int) { ldk = (uint32_t)(w.n_in / 2); }
        __device__ __forceinline__ void tile(const WeightDev& w, const WeightDev& w2, size_t r0, size_t r1, int lane) {
            const WeightDev& o = PAIR ? w2 : w;
            const size_t K = w.n_in, last = w.n_out - 1;
            // nibbles: pieces (row, 8 of 16 bytes), rows lane / 8 and 4 + lane / 8; bit pairs: (row, 4); scales: row = lane & 7
            const size_t rl = lane >> 3, rh = lane >> 2, rs = lane & 7;
            l0 = w.p0 + min(r0 + rl, last) * (K / 2) + (lane & 7) * 16;
            l1 = o.p0 + min(r1 + rl, last) * (K / 2) + (lane & 7) * 16;
            h0 = w.p1 + min(r0 + rh, last) * (K / 4) + (lane & 3) * 16;
            h1 = o.p1 + min(r1 + rh, last) * (K / 4) + (lane & 3) * 16;
            const size_t s0 = min(r0 + rs, last), s1 = min(r1 + rs, last);
            c0 = w.p2 + s0 * (K / 16);
            c1 = o.p2 + s1 * (K / 16);
            d0 = (const uint16_t*)w.p3 + s0 * (K / 256);
            d1 = (const uint16_t*)o.p3 + s1 * (K / 256);
            step = w.n_out >= 8 ? 4 : (uint32_t)min((size_t)4, w.n_out - 1 - min(rl, last));  // (a matrix of fewer rows than a half tile)
        }
        uint32_t step;
        __device__ __forceinline__ void issue(uint32_t slot, int b, bool, int lane) const {
            const uint32_t dl = slot + (lane >> 3) * 208 + (lane & 7) * 16, dh = slot + (lane >> 2) * 208 + 128 + (lane & 3) * 16;
            const size_t at = (size_t)b * 128, four = (size_t)step * ldk;
            cp16(dl, l0 + at);
            cp16(dl + 4 * 208, l0 + at + four);
            cp16(dl + 8 * 208, l1 + at);
            cp16(dl + 12 * 208, l1 + at + four);
            cp16(dh, h0 + (size_t)b * 64);
            cp16(dh + 8 * 208, h1 + (size_t)b * 64);
            if (lane < 8) {
                const uint32_t ds = slot + lane * 208 + 192;
                cp16(ds, c0 + (size_t)b * 16);
                cp16(ds + 8 * 208, c1 + (size_t)b * 16);
            } else if (lane < 16) {  // the aligned word that the scale lies in
                const uint32_t dd = slot + 16 * 208 + (lane & 7) * 4;
                cp4(dd, (const void*)((uintptr_t)(d0 + b) & ~(uintptr_t)3));
                cp4(dd + 32, (const void*)((uintptr_t)(d1 + b) & ~(uintptr_t)3));
            }
        }
    };
    // which half of its word the f16 scale of block 0 lies in, for rows g (bit 0) and g + 8 (bit 1) of a tile
    __device__ static __forceinline__ uint32_t tag(const WeightDev& w, const WeightDev& w2, size_t r0, size_t r1, int g) {
        const size_t nb = w.n_in / 256, last = w.n_out - 1;
        return (uint32_t)((((uintptr_t)w.p3 >> 1) + min(r0 + g, last) * nb) & 1) | (uint32_t)((((uintptr_t)w2.p3 >> 1) + min(r1 + g, last) * nb) & 1) << 1;
    }
    // Element 128 n + 32 k4 + e of a block: nibble k4 / 2 of ql[64 n + 32 (k4 & 1) + e] under bit pair k4 of qh[32 n + e], minus 32 (src/ggml.rs
    // Q6_K decode). As signed bytes of four times the value: the pair and the nibble shifted up by two, the sign bit turned.
    template <int TP>
    __device__ static __forceinline__ void block(uint32_t slot, int u, uint32_t tag, const WeightDev&, const WeightDev&, const X<TP>& x, int g, int t, float (&acc)[X<TP>::NT][2]) {
        constexpr int NT = X<TP>::NT;
        constexpr uint32_t N = 0x3C3C3C3Cu, P = 0xC0C0C0C0u, S = 0x80808080u;
        const uint32_t ra = slot + g * 208, rb = ra + 8 * 208;
        const uint4 sa = lds128(ra + 192), sb = lds128(rb + 192);
        const uint32_t wa = lds32(slot + 16 * 208 + g * 4), wb = lds32(slot + 16 * 208 + 32 + g * 4);
        const uint32_t scA[4] = {sa.x, sa.y, sa.z, sa.w}, scB[4] = {sb.x, sb.y, sb.z, sb.w};
        const uint32_t xf = x.frag + (uint32_t)u * (4 * X<TP>::STEP);
        int m[NT][4];
#pragma unroll
        for (int n = 0; n < NT; n++) m[n][0] = m[n][1] = m[n][2] = m[n][3] = 0;
#pragma unroll
        for (int n2 = 0; n2 < 2; n2++) {  // halves of the block
            uint32_t h[2][2], l[2][2][2];  // [row][half of 32]; [row][k4 & 1][half of 32]
#pragma unroll
            for (int e = 0; e < 2; e++)
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const uint32_t row = r ? rb : ra;
                    h[r][e] = lds32(row + 128 + 32 * n2 + 16 * e + 4 * t);
                    l[r][0][e] = lds32(row + 64 * n2 + 16 * e + 4 * t);
                    l[r][1][e] = lds32(row + 64 * n2 + 32 + 16 * e + 4 * t);
                }
#pragma unroll
            for (int kp = 0; kp < 2; kp++) {  // pairs of chunks: k4 = 2 kp, 2 kp + 1
                uint32_t a[2][2][2];  // [k4 & 1][half of 32][row]
#pragma unroll
                for (int o = 0; o < 2; o++)
#pragma unroll
                    for (int e = 0; e < 2; e++)
#pragma unroll
                        for (int r = 0; r < 2; r++) {
                            const uint32_t nib = ((kp ? l[r][o][e] >> 2 : l[r][o][e] << 2) & N) ^ S;
                            const int k4 = 2 * kp + o;
                            const uint32_t pr = k4 == 0 ? h[r][e] << 6 : k4 == 1 ? h[r][e] << 4 : k4 == 2 ? h[r][e] << 2 : h[r][e];
                            a[o][e][r] = (pr & P) ^ nib;
                        }
                const int c0 = 8 * n2 + 4 * kp;  // this pair's first scale (of 16 values)
#pragma unroll
                for (int n = 0; n < NT; n++) {
                    const uint4 b = lds128(xf + (2 * n2 + kp) * X<TP>::STEP + n * X<TP>::NEXT);
                    const uint32_t bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                    for (int i = 0; i < 4; i++) {  // runs of 16
                        int c[4];
                        mma_ss16(c, a[i >> 1][i & 1][0], a[i >> 1][i & 1][1], bw[i]);
                        const int si = (int)(int8_t)(scA[(c0 + i) >> 2] >> (8 * ((c0 + i) & 3))), ti = (int)(int8_t)(scB[(c0 + i) >> 2] >> (8 * ((c0 + i) & 3)));
                        m[n][0] += si * c[0];
                        m[n][1] += si * c[1];
                        m[n][2] += ti * c[2];
                        m[n][3] += ti * c[3];
                    }
                }
            }
        }
        const float w0 = (t & 1) ? 65536.0f : 1.0f, w1 = (t & 1) ? 0.0f : 256.0f;
        const float dA = 0.25f * ((tag & 1) ? half_hi(wa) : half_lo(wa)), dB = 0.25f * ((tag & 2) ? half_hi(wb) : half_lo(wb));
#pragma unroll
        for (int n = 0; n < NT; n++) {
            const float xs = ldsf(x.xs + (u * TP + 2 * n) * 4);
            acc[n][0] = fmaf(dA * xs, fmaf((float)m[n][1], w1, (float)m[n][0] * w0), acc[n][0]);
            acc[n][1] = fmaf(dB * xs, fmaf((float)m[n][3], w1, (float)m[n][2] * w0), acc[n][1]);
        }
    }
};

}  // namespace gmma
}  // namespace b2
