// Per-head norm, RoPE and cache append of one token (rope_head), and a CTA's sum.
#pragma once
#include <cuda_fp16.h>

#include "kernels.h"
#include "pdl.cuh"

namespace b2 {
namespace attend_core {

// Sum over the CTA (every thread calls it; threads with nothing to add pass 0). red: 32 floats of shared memory.
__device__ __forceinline__ float block_sum(float v, float* red) {  // red: 32 floats of shared memory
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
    __syncthreads();  // red may still be read from an earlier call
    if (lane == 0) red[warp] = v;
    __syncthreads();
    float s = 0.0f;
    for (int i = 0; i < nw; i++) s += red[i];  // same order in every thread
    return s;
}


// One head of the token's attention inputs: h < nh a query head, then nkv key heads, then nkv value heads. Every thread
// of the CTA calls this (it uses the CTA barrier); thread i < hd owns dimension i. Optional per-head RMS norm, RoPE on
// the first 2 * half_rot dimensions (unfused multiplies and adds, as the CPU's apply_rope), queries to `qo`, keys and
// values to row `pos` of the caches [nkv][max_len][hd]. buf: 256 floats of shared memory.
template <typename T>
__device__ __forceinline__ void rope_head(const uint32_t h, const uint32_t i, const uint32_t pos, const uint32_t table_pos0,
                                          const float* qkv, float* qo, T* kc, T* vc,
                                          const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ cs_table,
                                          const DecRope& p, float* buf, float* red) {
    const uint32_t hd = p.hd;
    const bool on = i < hd;
    const uint32_t kind = h < p.nh ? 0 : (h < p.nh + p.nkv ? 1 : 2);
    const uint32_t hh = kind == 0 ? h : (kind == 1 ? h - p.nh : h - p.nh - p.nkv);
    float v = 0.0f;
    // the vector is rewritten between calls by other SMs (persistent kernel): read it from L2
    if (on) v = __ldcg(kind == 0 ? qkv + hh * p.q_stride + i : (kind == 1 || p.v_from_k) ? qkv + p.k_off + hh * hd + i : qkv + p.v_off + hh * hd + i);
    const bool norm = kind == 0 ? qn != nullptr : (kind == 1 ? kn != nullptr : p.v_norm != 0);
    if (norm) {
        float s = block_sum(v * v, red);
        v = v * (1.0f / sqrtf(s / (float)hd + p.eps));
        if (on && kind == 0) v *= qn[i];
        else if (on && kind == 1) v *= kn[i];
    }
    const bool room = pos < p.max_len;  // a full cache: nothing is written (the host refuses the step before this)
    const size_t at = ((size_t)hh * p.max_len + pos) * hd + i;
    if (on && kind != 2) buf[i] = v;
    __syncthreads();
    if (on && room) {
        if (kind == 2) {
            vc[at] = (T)v;
        } else {
            const uint32_t hr = p.half_rot;
            const float* cs = cs_table + (size_t)(pos - table_pos0) * p.cs_stride + p.cs_off;  // cos[hr] then sin[hr] of this position
            if (i < 2 * hr) {
                if (p.interleaved) {
                    uint32_t j = i >> 1;
                    float c = cs[j], s = cs[hr + j];
                    float x1 = buf[2 * j], x2 = buf[2 * j + 1];
                    v = (i & 1) == 0 ? __fsub_rn(__fmul_rn(x1, c), __fmul_rn(x2, s)) : __fadd_rn(__fmul_rn(x2, c), __fmul_rn(x1, s));
                } else {
                    uint32_t j = i < hr ? i : i - hr;
                    float c = cs[j], s = cs[hr + j];
                    float x1 = buf[j], x2 = buf[j + hr];
                    v = i < hr ? __fsub_rn(__fmul_rn(x1, c), __fmul_rn(x2, s)) : __fadd_rn(__fmul_rn(x2, c), __fmul_rn(x1, s));
                }
            }
            if (kind == 0) qo[hh * hd + i] = v;
            else kc[at] = (T)v;
        }
    }
    __syncthreads();  // buf may be reused by the caller's next head
}

}  // namespace attend_core
}  // namespace b2
