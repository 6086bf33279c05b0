// The activation split of the small-batch products (gemv_mma.cu). A vector is cut into blocks of 256 values, one warp per block: lane
// l holds values 4 l .. 4 l + 3 and 128 + 4 l ... Two forms, chosen by the weights' format:
//
// Digits (integer weights). x ~ xs q with xs a power of two per block and |q| <= 8355711 = 127 (1 + 256 + 65536), 23 to 24 bits of
// the block's largest value (other GGUF formats: a fourth digit, 25 to 26 bits); q = q0 + 256 q1 + 65536 q2 in signed bytes. The products run on the integer tensor cores, exactly.
//   Record of a block: [pair of chunks of 32 k: 4][digit: 3][lane-in-four t][16 bytes] (the B fragments of two mma.m16n8k32: bytes
//   4 t .. of either half of the one chunk, then of the other), then SPLIT_AUX bytes of {xs, sum of squares of x, 0, 0, the sums of
//   q over the eight chunks (int32)}.
// Halves (FP8 weights). x = xs (hi + lo) with xs the power of two that brings the block's largest value into [2^14, 2^15), hi = f16(x / xs)
// and lo = f16 of what that left: 22 bits of every value.
//   Record of a block: [chunk of 32 k: 8][hi | lo][t][16 bytes] (two mma.m16n8k16: values 4 t .. 4 t + 3 of either half of the chunk), then SPLIT_AUX bytes as above without the sums.
#pragma once
#include "kernels.h"
#include "pdl.cuh"

namespace b2 {

constexpr float SPLIT_QMAX = 8355711.0f;
constexpr int SPLIT_AUX = 48;
constexpr int SPLIT_DIGITS = 768, SPLIT_HALVES = 1024;  // bytes of a block's values
__host__ __device__ inline size_t split_blocks(size_t K) { return (K + 255) / 256; }
__host__ __device__ inline size_t split_bytes(size_t K, bool halves) { return split_blocks(K) * ((halves ? SPLIT_HALVES : SPLIT_DIGITS) + SPLIT_AUX); }

struct SplitIn {  // a lane's eight values and their norm weights
    float4 x[2], w[2];
};
// x: the block's values, `n` of them from here to the end of the vector (a multiple of 4); w: norm weights or null.
__device__ __forceinline__ SplitIn split_load(const float* x, const float* w, int n, int lane) {
    SplitIn r;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int k = 128 * h + 4 * lane;
        r.x[h] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        r.w[h] = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
        if (k < n) {
            if (((uintptr_t)x & 15) == 0) r.x[h] = __ldcg((const float4*)(x + k));
            else r.x[h] = make_float4(__ldcg(x + k), __ldcg(x + k + 1), __ldcg(x + k + 2), __ldcg(x + k + 3));
            if (w) r.w[h] = __ldg((const float4*)(w + k));
        }
    }
    return r;
}

// The values times pre and the weights, their largest magnitude's bits over the warp, and the sum of squares before the weights.
__device__ __forceinline__ void split_values(const SplitIn& in, float pre, float (&v)[8], uint32_t& max_bits, float& ssq) {
    float q = 0.0f;
    uint32_t mx = 0;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const float a[4] = {in.x[h].x * pre, in.x[h].y * pre, in.x[h].z * pre, in.x[h].w * pre};
        const float b[4] = {in.w[h].x, in.w[h].y, in.w[h].z, in.w[h].w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            q = fmaf(a[i], a[i], q);
            v[4 * h + i] = a[i] * b[i];
            mx = max(mx, __float_as_uint(v[4 * h + i]) & 0x7fffffffu);  // non-negative floats order like their bit patterns, NaN last
        }
    }
    max_bits = __reduce_max_sync(0xffffffffu, mx);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
    ssq = q;
}

template <int DIGITS>
struct SplitDigits {
    uint32_t d[2][DIGITS];  // of each digit, a lane's four bytes for either half of the block
    int s[2];          // sums of q over chunks lane / 8 and 4 + lane / 8
    float xs, ssq;
};
// fast: the upper 18 of the 24 bits of every value
// Four digits: |q| <= 2^25, so that a chunk's sum stays inside 31 bits; the largest values are exact then.
template <int DIGITS = 3>
__device__ __forceinline__ SplitDigits<DIGITS> split_digits(const SplitIn& in, float pre, bool fast) {
    SplitDigits<DIGITS> r;
    float v[8];
    uint32_t mb;
    split_values(in, pre, v, mb, r.ssq);
    // the largest scales into (2^22, QMAX], or one power lower when it would exceed it
    const int up = mb == 0 ? 0 : min(126, max(-126, (DIGITS == 4 ? 151 : 149 - ((mb & 0x7fffffu) > 0x7efefeu ? 1 : 0)) - (int)(mb >> 23)));
    const float k = __uint_as_float((uint32_t)(127 + up) << 23);
    r.xs = mb >= 0x7f800000u ? __uint_as_float(0x7fffffffu) : __uint_as_float((uint32_t)(127 - up) << 23);  // (digits cannot hold an infinity or a NaN)
#pragma unroll
    for (int h = 0; h < 2; h++) {
        uint32_t u[4];
        int s = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            int q = __float2int_rn(v[4 * h + i] * k);
            if (DIGITS == 3 && fast) q = min((q + 32) & ~63, 0x7f7f40);  // (the next multiple of 64 has no three signed digits)
            s += q;
            u[i] = (uint32_t)q + (DIGITS == 4 ? 0x80808080u : 0x808080u);  // q + 128 (1 + 256 + 65536 ..): its bytes are the digits plus 128
        }
        const uint32_t a = __byte_perm(u[0], u[1], 0x5140), b = __byte_perm(u[2], u[3], 0x5140);
        r.d[h][0] = __byte_perm(a, b, 0x5410) ^ 0x80808080u;
        r.d[h][1] = __byte_perm(a, b, 0x7632) ^ 0x80808080u;
        if constexpr (DIGITS == 4) {
            const uint32_t c = __byte_perm(u[0], u[1], 0x7362), e = __byte_perm(u[2], u[3], 0x7362);
            r.d[h][2] = __byte_perm(c, e, 0x5410) ^ 0x80808080u;
            r.d[h][3] = __byte_perm(c, e, 0x7632) ^ 0x80808080u;
        } else {
            r.d[h][2] = __byte_perm(__byte_perm(u[0], u[1], 0x0062), __byte_perm(u[2], u[3], 0x0062), 0x5410) ^ 0x80808080u;
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        r.s[h] = s;
    }
    return r;
}
// Where a lane's digits go in the block's record: half h at split_digit_at(h, lane) + 64 * digit.
__device__ __forceinline__ void split_digit_at(int h, int lane, int& pair, int& in16) {
    const int chunk = 4 * h + (lane >> 3);
    pair = chunk >> 1;
    in16 = (lane & 3) * 16 + (chunk & 1) * 8 + ((lane >> 2) & 1) * 4;
}

__device__ __forceinline__ uint32_t split_pack(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *(const uint32_t*)&h;
}
struct SplitHalves {
    uint2 hi[2], lo[2];
    float xs, ssq;
};
__device__ __forceinline__ SplitHalves split_halves(const SplitIn& in, float pre) {
    SplitHalves r;
    float v[8];
    uint32_t mb;
    split_values(in, pre, v, mb, r.ssq);
    const int up = mb == 0 ? 0 : min(126, max(-126, 141 - (int)(mb >> 23)));
    const float k = __uint_as_float((uint32_t)(127 + up) << 23);
    r.xs = __uint_as_float((uint32_t)(127 - up) << 23);
#pragma unroll
    for (int h = 0; h < 2; h++) {
        float a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            a[i] = v[4 * h + i] * k;
            b[i] = a[i] - __half2float(__float2half_rn(a[i]));
        }
        r.hi[h] = make_uint2(split_pack(a[0], a[1]), split_pack(a[2], a[3]));
        r.lo[h] = make_uint2(split_pack(b[0], b[1]), split_pack(b[2], b[3]));
    }
    return r;
}

}  // namespace b2
