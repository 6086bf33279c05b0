// The other GGUF block formats (dq_other.cuh) in the small-batch products of gemv_mma.cu: rows of whole 256-value runs, read as they are
// in the file. Every format's values are small integers under an integer or float scale per 16 or 32 (and a minimum, some): the
// integers become signed or unsigned bytes in a few instructions on whole words, the integer tensor cores do the rest.
//
// The generic kernel of gemv_other.cu reads single bytes from shared memory and multiplies floats: four passes of the shared-memory
// pipe per 32 weights, 39 us for Q5_K 14336 x 4096. This form is bound like the tuned formats; what it measures stands at launch_gemv_other.
#pragma once
#include "dq_other.cuh"
#include "gemv_mma.cuh"

namespace b2 {
namespace gmma {

__host__ __device__ constexpr uint32_t pack4(int a, int b, int c, int d) {
    return ((uint32_t)a & 255u) | ((uint32_t)b & 255u) << 8 | ((uint32_t)c & 255u) << 16 | ((uint32_t)d & 255u) << 24;
}
// Four indices into the code book (IQ4: ggml's non-linear 4-bit one, else the doubled E2M1 values): nibbles 0 .. 3 of `sel` hold their
// low three bits, those of `hi` 0, 1, 2, 3, plus four where the index's fourth bit is set.
template <bool IQ4>
__device__ __forceinline__ uint32_t lut4(uint32_t sel, uint32_t hi) {
    constexpr uint32_t T0 = IQ4 ? pack4(-127, -104, -83, -65) : pack4(0, 1, 2, 3), T1 = IQ4 ? pack4(-49, -35, -22, -10) : pack4(4, 6, 8, 12);
    constexpr uint32_t T2 = IQ4 ? pack4(1, 13, 25, 38) : pack4(0, -1, -2, -3), T3 = IQ4 ? pack4(53, 69, 89, 113) : pack4(-4, -6, -8, -12);
    return __byte_perm(__byte_perm(T0, T1, sel), __byte_perm(T2, T3, sel), hi);
}
// The eight nibbles of w through the table: the low nibbles of its four bytes to `lo`, the high ones to `hi`.
template <bool IQ4>
__device__ __forceinline__ void lut8(uint32_t w, uint32_t& lo, uint32_t& hi) {
    const uint32_t s = w & 0x77777777u, h = 0x32103210u | ((w & 0x88888888u) >> 1);
    const uint32_t a = lut4<IQ4>(s & 0xffffu, h & 0xffffu), b = lut4<IQ4>(s >> 16, h >> 16);
    lo = __byte_perm(a, b, 0x6420);
    hi = __byte_perm(a, b, 0x7531);
}
// The low nibbles of w's bytes (the high ones are zero) through the table.
template <bool IQ4>
__device__ __forceinline__ uint32_t lut4_bytes(uint32_t w) {
    const uint32_t p = __byte_perm(w | (w >> 4), 0, 0x4420);
    return lut4<IQ4>(p & 0x7777u, 0x3210u | ((p & 0x8888u) >> 1));
}
// bits 0 .. 3 of x to bit 0 of bytes 0 .. 3
__device__ __forceinline__ uint32_t spread4(uint32_t x) { return (x * 0x00204081u) & 0x01010101u; }

__device__ __forceinline__ void cp8(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}

template <int FMT>
struct Fo {
    template <int TP>
    using X = XView<TP, false, 4>;  // (four digits: the float kernel, which these formats had before, rounds nothing of x)
    static constexpr bool ONE = FMT == B2_FMT_Q4_1 || FMT == B2_FMT_Q5_1;  // a float minimum per 32
    static constexpr bool HALVES = false, SUMS = ONE || FMT == B2_FMT_Q5_K, SUMS_BY_COLUMN = FMT == B2_FMT_Q5_K, IN_PAIRS = false;
    static constexpr int BS = FMT == B2_FMT_Q2_K || FMT == B2_FMT_Q3_K || FMT == B2_FMT_Q5_K || FMT == B2_FMT_IQ4_XS ? 256 : FMT == B2_FMT_NVFP4 ? 64 : 32;
    static constexpr int TS = FMT == B2_FMT_NVFP4 ? 36 : FMT == B2_FMT_Q4_0 || FMT == B2_FMT_IQ4_NL ? 18 : FMT == B2_FMT_Q4_1 ? 20 : FMT == B2_FMT_Q5_0 ? 22 : FMT == B2_FMT_Q5_1 ? 24
                              : FMT == B2_FMT_Q2_K ? 84 : FMT == B2_FMT_Q3_K ? 110 : FMT == B2_FMT_Q5_K ? 176 : FMT == B2_FMT_IQ4_XS ? 136 : 17;
    static constexpr int RUN = 256 / BS * TS;                                     // bytes of 256 values
    static constexpr int PIECE = RUN % 16 == 0 ? 16 : RUN % 8 == 0 ? 8 : 4;       // a copy's bytes; Q3_K runs are 2-byte aligned: the words around them
    static constexpr int NP = (RUN + 3) / 4 * 4 / PIECE;                          // copies of a run
    // of a row in a slot: an odd multiple of 16 bytes, so that eight rows of four words each fall on 32 banks
    static constexpr int STRIDE = RUN <= 112 ? 112 : RUN <= 144 ? 144 : RUN <= 176 ? 176 : 208;
    static constexpr bool PARTS = false;  // long rows of several tokens go token by token instead
    static constexpr int BLOCK_K = 256, SLOTS = STRIDE > 176 ? 2 : 3, MAX_BLOCKS = 1;
    static constexpr int BLOCK_BYTES = 16 * STRIDE, UNIT_BYTES = BLOCK_BYTES;
    // One: eight sums of 32 times the block scale. Q5_K: as for Q4_K.
    __device__ static __forceinline__ void put_sums(uint8_t* e, float xs, int s, int lane) {
        if (FMT == B2_FMT_Q5_K) F4<false, false>::put_sums(e, xs, s, lane);
        else if (ONE && lane < 8) ((float*)e)[lane] = xs * (float)s;
    }
    // Q3_K: whether block 0 of rows g (bit 0) and g + 8 (bit 1) starts in the middle of a word
    __device__ static __forceinline__ uint32_t tag(const WeightDev& w, const WeightDev& w2, size_t r0, size_t r1, int g) {
        if (FMT != B2_FMT_Q3_K) return 0;
        const size_t rb = w.n_in / 256 * RUN, last = w.n_out - 1;
        return (uint32_t)((((uintptr_t)w.p0 + min(r0 + g, last) * rb) >> 1) & 1) | (uint32_t)((((uintptr_t)w2.p0 + min(r1 + g, last) * rb) >> 1) & 1) << 1;
    }
    template <bool PAIR>
    struct Copy {
        static constexpr int N = (8 * NP + 31) / 32;
        const uint8_t *p0, *p1;
        uint32_t off[N], dst[N];
        size_t rb;
        __device__ __forceinline__ void init(const WeightDev& w, int, int lane) {
            rb = w.n_in / 256 * RUN;
#pragma unroll
            for (int i = 0; i < N; i++) {
                const int q = lane + 32 * i, row = q / NP, in = q - row * NP;
                off[i] = (uint32_t)min(row, (int)min((size_t)7, w.n_out - 1)) * (uint32_t)rb + (uint32_t)(in * PIECE);
                dst[i] = (uint32_t)(row * STRIDE + in * PIECE);
            }
        }
        __device__ __forceinline__ void tile(const WeightDev& w, const WeightDev& w2, size_t r0, size_t r1, int) {
            p0 = w.p0 + r0 * rb;
            p1 = (PAIR ? w2.p0 : w.p0) + r1 * rb;
        }
        __device__ __forceinline__ void issue(uint32_t slot, int b, bool, int lane) const {
            const uint32_t at = (uint32_t)b * RUN;
#pragma unroll
            for (int i = 0; i < N; i++) {
                if (32 * i + 32 > 8 * NP && lane + 32 * i >= 8 * NP) break;
                const uint8_t *s0 = p0 + (at + off[i]), *s1 = p1 + (at + off[i]);
                if (PIECE == 16) {
                    cp16(slot + dst[i], s0);
                    cp16(slot + dst[i] + 8 * STRIDE, s1);
                } else if (PIECE == 8) {
                    cp8(slot + dst[i], s0);
                    cp8(slot + dst[i] + 8 * STRIDE, s1);
                } else {
                    cp4(slot + dst[i], (const void*)((uintptr_t)s0 & ~(uintptr_t)3));
                    cp4(slot + dst[i] + 8 * STRIDE, (const void*)((uintptr_t)s1 & ~(uintptr_t)3));
                }
            }
        }
    };

    // The word at `row + at`, at the row's own alignment of 4 (at: a constant).
    __device__ static __forceinline__ uint32_t word(uint32_t row, int at) {
        if (at % 4 == 0) return lds32(row + at);
        const uint32_t sel = at % 4 == 1 ? 0x4321 : at % 4 == 2 ? 0x5432 : 0x6543;
        return __byte_perm(lds32(row + at / 4 * 4), lds32(row + at / 4 * 4 + 4), sel);
    }
    __device__ static __forceinline__ float half_at(uint32_t row, int at) {
        const uint32_t w = lds32(row + at / 4 * 4);
        return at % 4 ? half_hi(w) : half_lo(w);
    }
    // Chunk c of a row's run: the bytes of values 4 t .. and 16 + 4 t .., and what they are multiplied by: d[0] for all, or d[0] / d[1]
    // for the halves. `r`: the row plus 4 t. For the formats of 32- and 64-value blocks.
    __device__ static __forceinline__ void chunk(uint32_t row, uint32_t r, int c, int t, uint32_t& a, uint32_t& b, float (&d)[2], float& m) {
        constexpr uint32_t L = 0x0F0F0F0Fu;
        const int at = c * TS;
        m = 0.0f;
        if constexpr (FMT == B2_FMT_Q4_0) {  // 16 (n - 8) as signed bytes
            const uint32_t w = word(r, at + 2);
            a = ((w << 4) & 0xF0F0F0F0u) ^ 0x80808080u;
            b = (w & 0xF0F0F0F0u) ^ 0x80808080u;
            d[0] = 0.0625f * half_at(row, at);
        } else if constexpr (FMT == B2_FMT_Q4_1) {
            const uint32_t w = word(r, at + 4), h = lds32(row + at);
            a = w & L;
            b = (w >> 4) & L;
            d[0] = half_lo(h);
            m = half_hi(h);
        } else if constexpr (FMT == B2_FMT_Q5_0) {  // 8 (n - 16) as signed bytes
            const uint32_t w = word(r, at + 6), qh = word(row, at + 2) >> (4 * t);
            a = (((w << 3) & 0x78787878u) | spread4(qh & 15u) << 7) ^ 0x80808080u;
            b = (((w >> 1) & 0x78787878u) | spread4((qh >> 16) & 15u) << 7) ^ 0x80808080u;
            d[0] = 0.125f * half_at(row, at);
        } else if constexpr (FMT == B2_FMT_Q5_1) {
            const uint32_t w = word(r, at + 8), h = lds32(row + at), qh = lds32(row + at + 4) >> (4 * t);
            a = (w & L) | spread4(qh & 15u) << 4;
            b = ((w >> 4) & L) | spread4((qh >> 16) & 15u) << 4;
            d[0] = half_lo(h);
            m = half_hi(h);
        } else if constexpr (FMT == B2_FMT_IQ4_NL) {
            lut8<true>(word(r, at + 2), a, b);
            d[0] = half_at(row, at);
        } else if constexpr (FMT == B2_FMT_MXFP4) {
            lut8<false>(word(r, at + 1), a, b);
            const uint32_t w = lds32(row + at / 4 * 4);
            d[0] = e8m0_half((w >> (8 * (at % 4))) & 0xffu);
        } else if constexpr (FMT == B2_FMT_NVFP4) {
            // sub-blocks of 16: the low nibbles of eight bytes, then the high ones
            const int blk = (c >> 1) * 36, s = 2 * (c & 1);
            const uint32_t at4 = row + blk + 4 + 8 * s + 4 * (t & 1);
            a = lut4_bytes<false>((lds32(at4) >> (4 * (t >> 1))) & L);
            b = lut4_bytes<false>((lds32(at4 + 8) >> (4 * (t >> 1))) & L);
            const uint32_t sc = lds32(row + blk) >> (8 * s);
            d[0] = ue4m3_half(sc & 0xffu);
            d[1] = ue4m3_half((sc >> 8) & 0xffu);
        }
    }

    // Q5_K: as Q4_K with a fifth bit. Q2_K: the 4-bit scale multiplies the 2-bit values in their bytes. Q3_K, IQ4_XS: integer scales.
    template <int TP>
    __device__ static __forceinline__ void block(uint32_t slot, int u, uint32_t tag, const WeightDev& w, const WeightDev& w2, const X<TP>& x, int g, int t,
                                                 float (&acc)[X<TP>::NT][2]) {
        constexpr int NT = X<TP>::NT;
        const uint32_t row[2] = {slot + g * STRIDE, slot + (g + 8) * STRIDE};
        const uint32_t xf = x.frag + (uint32_t)u * (4 * X<TP>::STEP);
        const float w0 = (t & 1) ? 65536.0f : 1.0f, w1 = (t & 1) ? 16777216.0f : 256.0f;  // what this lane's two digits stand for
        if constexpr (BS != 256) {
            float f[NT][2], mins[2][4] = {};  // mins: of the four chunks that this lane of its token's two takes
#pragma unroll
            for (int n = 0; n < NT; n++) f[n][0] = f[n][1] = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                uint4 bq[NT];
#pragma unroll
                for (int n = 0; n < NT; n++) bq[n] = lds128(xf + j * X<TP>::STEP + n * X<TP>::NEXT);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    uint32_t a[2][2];
                    float d[2][2], m[2];
#pragma unroll
                    for (int r = 0; r < 2; r++) {
                        chunk(row[r], row[r] + 4 * t, 2 * j + h, t, a[r][0], a[r][1], d[r], m[r]);
                        if (ONE && ((t & 1) == (2 * j + h) / 4)) mins[r][(2 * j + h) % 4] = m[r];
                    }
#pragma unroll
                    for (int n = 0; n < NT; n++) {
                        const uint32_t b0 = h ? bq[n].z : bq[n].x, b1 = h ? bq[n].w : bq[n].y;
                        int c[4];
                        if constexpr (FMT == B2_FMT_NVFP4) {
                            int e[4];
                            mma_ss16(c, a[0][0], a[1][0], b0);
                            mma_ss16(e, a[0][1], a[1][1], b1);
                            f[n][0] = fmaf(d[0][1], fmaf((float)e[1], w1, (float)e[0] * w0), fmaf(d[0][0], fmaf((float)c[1], w1, (float)c[0] * w0), f[n][0]));
                            f[n][1] = fmaf(d[1][1], fmaf((float)e[3], w1, (float)e[2] * w0), fmaf(d[1][0], fmaf((float)c[3], w1, (float)c[2] * w0), f[n][1]));
                        } else {
                            if constexpr (ONE) mma_us_0(c, a[0][0], a[1][0], a[0][1], a[1][1], b0, b1);
                            else mma_ss_0(c, a[0][0], a[1][0], a[0][1], a[1][1], b0, b1);
                            f[n][0] = fmaf(d[0][0], fmaf((float)c[1], w1, (float)c[0] * w0), f[n][0]);
                            f[n][1] = fmaf(d[1][0], fmaf((float)c[3], w1, (float)c[2] * w0), f[n][1]);
                        }
                    }
                }
            }
            const float gs[2] = {FMT == B2_FMT_NVFP4 && w.p1 ? __ldg((const float*)w.p1) : 1.0f, FMT == B2_FMT_NVFP4 && w2.p1 ? __ldg((const float*)w2.p1) : 1.0f};
#pragma unroll
            for (int n = 0; n < NT; n++) {
                const float xs = ldsf(x.xs + (u * TP + 2 * n) * 4);
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    acc[n][r] = fmaf(FMT == B2_FMT_NVFP4 ? xs * gs[r] : xs, f[n][r], acc[n][r]);
                    if constexpr (ONE) {
                        const uint4 s = lds128(x.sums + (t & 1) * 8 + (u * TP + 2 * n) * 32);
                        float v = acc[n][r];
                        v = fmaf(mins[r][0], __uint_as_float(s.x), v);
                        v = fmaf(mins[r][1], __uint_as_float(s.y), v);
                        v = fmaf(mins[r][2], __uint_as_float(s.z), v);
                        acc[n][r] = fmaf(mins[r][3], __uint_as_float(s.w), v);
                    }
                }
            }
        } else {
            int lo[NT][4], e[NT][4];
#pragma unroll
            for (int n = 0; n < NT; n++)
#pragma unroll
                for (int i = 0; i < 4; i++) lo[n][i] = e[n][i] = 0;
            float dd[2], dm[2] = {0.0f, 0.0f};  // of the rows
            // the word at `at` of row r (Q3_K rows may start in the middle of a word)
            auto rw = [&](int r, int at) {
                if constexpr (FMT == B2_FMT_Q3_K) {
                    const uint32_t p = row[r] + at;
                    return (tag >> r) & 1 ? __byte_perm(lds32(p), lds32(p + 4), 0x5432) : lds32(p);
                } else {
                    return lds32(row[r] + at);
                }
            };
            if constexpr (FMT == B2_FMT_Q2_K) {
                uint4 sc[2];
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    sc[r] = lds128(row[r]);
                    const uint32_t h = lds32(row[r] + 80);
                    dd[r] = half_lo(h);
                    dm[r] = half_hi(h);
                }
#pragma unroll
                for (int n2 = 0; n2 < 2; n2++) {
                    uint32_t q[2][2];
#pragma unroll
                    for (int r = 0; r < 2; r++) {
                        q[r][0] = lds32(row[r] + 16 + 32 * n2 + 4 * t);
                        q[r][1] = lds32(row[r] + 32 + 32 * n2 + 4 * t);
                    }
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        uint32_t a[2][2], mn[2][2];
#pragma unroll
                        for (int r = 0; r < 2; r++) {
                            const uint32_t s4 = n2 ? (j < 2 ? sc[r].z : sc[r].w) : (j < 2 ? sc[r].x : sc[r].y), s2 = s4 >> (16 * (j & 1));
#pragma unroll
                            for (int h = 0; h < 2; h++) {
                                const uint32_t s = (s2 >> (8 * h)) & 0xffu;
                                a[r][h] = ((q[r][h] >> (2 * j)) & 0x03030303u) * (s & 15u);
                                mn[r][h] = (s >> 4) * 0x01010101u;
                            }
                        }
#pragma unroll
                        for (int n = 0; n < NT; n++) {
                            const uint4 b = lds128(xf + (2 * n2 + (j >> 1)) * X<TP>::STEP + n * X<TP>::NEXT);
                            const uint32_t b0 = (j & 1) ? b.z : b.x, b1 = (j & 1) ? b.w : b.y;
                            mma_us(lo[n], a[0][0], a[1][0], a[0][1], a[1][1], b0, b1);
                            mma_us(e[n], mn[0][0], mn[1][0], mn[0][1], mn[1][1], b0, b1);
                        }
                    }
                }
            } else if constexpr (FMT == B2_FMT_Q3_K) {  // 32 (q - 4) as signed bytes
                uint32_t sc[2][4], hm[2][2];
#pragma unroll
                for (int r = 0; r < 2; r++) {  // the sixteen 6-bit scales as bytes (q3k_scales, src/ggml.rs:513-531)
                    const uint32_t a0 = rw(r, 96), a1 = rw(r, 100), tm = rw(r, 104);
                    sc[r][0] = (a0 & 0x0f0f0f0fu) | ((tm & 0x03030303u) << 4);
                    sc[r][1] = (a1 & 0x0f0f0f0fu) | (((tm >> 2) & 0x03030303u) << 4);
                    sc[r][2] = ((a0 >> 4) & 0x0f0f0f0fu) | (((tm >> 4) & 0x03030303u) << 4);
                    sc[r][3] = ((a1 >> 4) & 0x0f0f0f0fu) | (((tm >> 6) & 0x03030303u) << 4);
                    const uint32_t dw = lds32(row[r] + 108);  // the two bytes at 108, or 110 where the row starts in the middle of a word
                    dd[r] = 0.03125f * ((tag >> r) & 1 ? half_hi(dw) : half_lo(dw));
                    hm[r][0] = rw(r, 4 * t);
                    hm[r][1] = rw(r, 16 + 4 * t);
                }
#pragma unroll
                for (int n2 = 0; n2 < 2; n2++) {
                    uint32_t q[2][2];
#pragma unroll
                    for (int r = 0; r < 2; r++) {
                        q[r][0] = rw(r, 32 + 32 * n2 + 4 * t);
                        q[r][1] = rw(r, 48 + 32 * n2 + 4 * t);
                    }
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        uint32_t a[2][2];
                        int s[2][2];
#pragma unroll
                        for (int r = 0; r < 2; r++)
#pragma unroll
                            for (int h = 0; h < 2; h++) {
                                a[r][h] = ((((q[r][h] >> (2 * j)) & 0x03030303u) << 5) | (((hm[r][h] >> (4 * n2 + j)) & 0x01010101u) << 7)) ^ 0x80808080u;
                                const int si = 8 * n2 + 2 * j + h;
                                s[r][h] = (int)((sc[r][si >> 2] >> (8 * (si & 3))) & 0xffu) - 32;
                            }
#pragma unroll
                        for (int n = 0; n < NT; n++) {
                            const uint4 b = lds128(xf + (2 * n2 + (j >> 1)) * X<TP>::STEP + n * X<TP>::NEXT);
#pragma unroll
                            for (int h = 0; h < 2; h++) {
                                int c[4];
                                mma_ss16(c, a[0][h], a[1][h], h ? ((j & 1) ? b.w : b.y) : ((j & 1) ? b.z : b.x));
                                lo[n][0] += s[0][h] * c[0];
                                lo[n][1] += s[0][h] * c[1];
                                lo[n][2] += s[1][h] * c[2];
                                lo[n][3] += s[1][h] * c[3];
                            }
                        }
                    }
                }
            } else {  // Q5_K, IQ4_XS: an integer scale per 32
                uint32_t s8[2][2], qh[2][2], mb[2] = {0u, 0u};
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    if constexpr (FMT == B2_FMT_Q5_K) {  // the header is Q4_K's (get_scale_min_k4, src/ggml.rs:501-509)
                        const uint4 h = lds128(row[r]);
                        s8[r][0] = h.y & 0x3f3f3f3fu;
                        s8[r][1] = (h.w & 0x0f0f0f0fu) | ((h.y >> 2) & 0x30303030u);
                        mb[r] = t == 0 ? h.z & 0x3f3f3f3fu : t == 1 ? ((h.w >> 4) & 0x0f0f0f0fu) | ((h.z >> 2) & 0x30303030u) : 0u;
                        dd[r] = half_lo(h.x);
                        dm[r] = half_hi(h.x);
                        qh[r][0] = lds32(row[r] + 16 + 4 * t);
                        qh[r][1] = lds32(row[r] + 32 + 4 * t);
                    } else {  // low nibbles of the scales in s8[0], high pairs in s8[1]
                        const uint32_t h = lds32(row[r]);
                        dd[r] = half_lo(h);
                        s8[r][0] = lds32(row[r] + 4);
                        s8[r][1] = h >> 16;
                    }
                }
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    uint32_t a[2][2][2];  // [chunk][row][half]
                    int s[2][2];          // [chunk][row]
#pragma unroll
                    for (int r = 0; r < 2; r++) {
                        if constexpr (FMT == B2_FMT_Q5_K) {
#pragma unroll
                            for (int h = 0; h < 2; h++) {
                                const uint32_t q = lds32(row[r] + 48 + 32 * j + 16 * h + 4 * t);
                                a[0][r][h] = (q & 0x0f0f0f0fu) | (((qh[r][h] >> (2 * j)) & 0x01010101u) << 4);
                                a[1][r][h] = ((q >> 4) & 0x0f0f0f0fu) | (((qh[r][h] >> (2 * j + 1)) & 0x01010101u) << 4);
                            }
                            s[0][r] = (int)((s8[r][j >> 1] >> (16 * (j & 1))) & 0xffu);
                            s[1][r] = (int)((s8[r][j >> 1] >> (16 * (j & 1) + 8)) & 0xffu);
                        } else {
#pragma unroll
                            for (int k = 0; k < 2; k++) {
                                const int c = 2 * j + k;
                                lut8<true>(lds32(row[r] + 8 + 16 * c + 4 * t), a[k][r][0], a[k][r][1]);
                                s[k][r] = (int)(((s8[r][0] >> (4 * c)) & 15u) | (((s8[r][1] >> (2 * c)) & 3u) << 4)) - 32;
                            }
                        }
                    }
#pragma unroll
                    for (int n = 0; n < NT; n++) {
                        const uint4 b = lds128(xf + j * X<TP>::STEP + n * X<TP>::NEXT);
#pragma unroll
                        for (int k = 0; k < 2; k++) {
                            int c[4];
                            if constexpr (FMT == B2_FMT_Q5_K) mma_us_0(c, a[k][0][0], a[k][1][0], a[k][0][1], a[k][1][1], k ? b.z : b.x, k ? b.w : b.y);
                            else mma_ss_0(c, a[k][0][0], a[k][1][0], a[k][0][1], a[k][1][1], k ? b.z : b.x, k ? b.w : b.y);
                            lo[n][0] += s[k][0] * c[0];
                            lo[n][1] += s[k][0] * c[1];
                            lo[n][2] += s[k][1] * c[2];
                            lo[n][3] += s[k][1] * c[3];
                        }
                    }
                }
                if constexpr (FMT == B2_FMT_Q5_K)
#pragma unroll
                    for (int n = 0; n < NT; n++) mma_us16(e[n], mb[0], mb[1], lds32(x.sums + (u * TP + 2 * n) * 32));  // mins times the chunk sums' digits
            }
#pragma unroll
            for (int n = 0; n < NT; n++) {
                const float xs = ldsf(x.xs + (u * TP + 2 * n) * 4);
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const float p = fmaf((float)lo[n][2 * r + 1], w1, (float)lo[n][2 * r] * w0);
                    float v = dd[r] * p;
                    if constexpr (FMT == B2_FMT_Q2_K || FMT == B2_FMT_Q5_K) v = fmaf(dd[r], p, -(dm[r] * fmaf((float)e[n][2 * r + 1], w1, (float)e[n][2 * r] * w0)));
                    acc[n][r] = fmaf(xs, v, acc[n][r]);
                }
            }
        }
    }
};

}  // namespace gmma
}  // namespace b2
