// Packed weights to f16 operands in tensor memory: 64 weights of a row a call, as 32 words of two (gemm_wt.cu, gemm_wp.cu).
#pragma once
#include <cuda_fp8.h>

#include "tcgen05.cuh"

namespace b2 {
namespace {

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
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, "
        "%21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
          "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]),
          "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]),
          "=r"(v[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ __half2 as_h2(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }
// The second terms of Q4_K weights in the place of their first: the exact f32 weight of the reference's decode, d1 * q - m1 with both
// roundings (src/ggml.rs:750-773), minus the first term.
__device__ __forceinline__ void expand_4bit_rest(const uint4& hdr, const uint32_t (&qw)[8], int j, uint32_t (&o)[32]) {
    uint32_t sc0, mn0, sc1, mn1;
    q4k_scale_min(2 * j, hdr.y, hdr.z, hdr.w, sc0, mn0);
    q4k_scale_min(2 * j + 1, hdr.y, hdr.z, hdr.w, sc1, mn1);
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

// 64 weights of a 4-bit block: 32 bytes, low nibbles = elements 0..31, high nibbles = 32..63 (see gemm_tc.cu for the arithmetic).
// hdr: the block's 16 bytes in front; j: which of its four groups of 64.
template <int FMT>
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
}

constexpr float WT_PRE = 256.0f;  // power of two in the f16 weights of Q6_K, Q8_0 and FP8: small scales stay out of f16's subnormals

// 64 bytes of a Q8_0 row and the f16 scales of its two blocks of 32: q exactly, times f16(256 d).
__device__ __forceinline__ void expand_q8_0(const uint4 (&q)[4], uint32_t d2, uint32_t (&o)[32]) {
    const __half2 m0 = __float2half2_rn(__half2float(__ushort_as_half((unsigned short)(d2 & 0xffffu))) * WT_PRE);
    const __half2 m1 = __float2half2_rn(__half2float(__ushort_as_half((unsigned short)(d2 >> 16))) * WT_PRE);
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
}

// 64 e4m3 bytes and their block scale.
__device__ __forceinline__ void expand_f8(const uint4 (&q)[4], float scale, uint32_t (&o)[32]) {
    const __half2 sc2 = __float2half2_rn(scale * WT_PRE);
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

// 64 weights of a Q6_K super-block's half: its 64 bytes of low nibbles (odd: the high nibbles of them), 32 bytes of bit pairs and the
// group's four i8 scales: (q - 32) exactly, times f16(256 d sc).
__device__ __forceinline__ void expand_q6k(const uint4 (&ql4)[4], const uint4 (&qh4)[2], float d, uint32_t sc4, bool odd, uint32_t (&o)[32]) {
    const uint32_t qlw[16] = {ql4[0].x, ql4[0].y, ql4[0].z, ql4[0].w, ql4[1].x, ql4[1].y, ql4[1].z, ql4[1].w,
                              ql4[2].x, ql4[2].y, ql4[2].z, ql4[2].w, ql4[3].x, ql4[3].y, ql4[3].z, ql4[3].w};
    const uint32_t qhw[8] = {qh4[0].x, qh4[0].y, qh4[0].z, qh4[0].w, qh4[1].x, qh4[1].y, qh4[1].z, qh4[1].w};
    const __half2 bias = __float2half2_rn(1056.0f);  // 1024 under the exponent byte 0x64, and 32
    __half2 mul[4];
#pragma unroll
    for (int i = 0; i < 4; i++) mul[i] = __float2half2_rn(d * (float)(int8_t)(sc4 >> (8 * i)) * WT_PRE);
#pragma unroll
    for (int i = 0; i < 16; i++) {  // word i: elements 4 i .. 4 i + 3 of the group; its bit pairs go to bits 4 and 5 of their bytes
        const uint32_t nib = (odd ? qlw[i] >> 4 : qlw[i]) & 0x0F0F0F0Fu;
        const uint32_t hb = (odd ? qhw[i & 7] >> (2 * (i >> 3)) : qhw[i & 7] << (4 - 2 * (i >> 3))) & 0x30303030u;
        const uint32_t q4 = nib | hb;
        o[2 * i] = h2_bits(__hmul2(__hsub2(as_h2(__byte_perm(q4, 0x64646464u, 0x4140)), bias), mul[i >> 2]));
        o[2 * i + 1] = h2_bits(__hmul2(__hsub2(as_h2(__byte_perm(q4, 0x64646464u, 0x4342)), bias), mul[i >> 2]));
    }
}

}  // namespace
}  // namespace b2
