// The non-matmul kernels of a prefill step: the ops of decode_ops.cu over many token rows at once
// (Backend::decode_plan_prefill, src/gpu.rs:283-289: "steps of up to `tokens` tokens on batched kernels, the activations
// kept on the device for the whole step"). Token row r of every activation sits `stride` floats behind row r - 1.
//
//   qk_rope_rows : per-head q / k norm, RoPE and cache append of every token (rope_head, the one-token arithmetic)
//   glu_rows, rows_op : the element-wise ops
#include <cuda_fp16.h>

#include <algorithm>

#include "attend_core.cuh"

namespace b2 {

using namespace attend_core;

namespace {

__device__ __forceinline__ uint32_t pack_h2f(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *(const uint32_t*)&h;
}

template <typename T>
__global__ void __launch_bounds__(256) qk_rope_rows_kernel(const float* __restrict__ qkv, float* __restrict__ qo, size_t stride, T* __restrict__ kc,
                                                           T* __restrict__ vc, const float* __restrict__ qn, const float* __restrict__ kn,
                                                           const float* __restrict__ cs_table, const uint32_t* __restrict__ sp, DecRope p) {
    __shared__ float buf[256];
    __shared__ float red[32];
    pdl_launch_dependents();
    const size_t off = (size_t)blockIdx.y * stride;
    rope_head<T>(blockIdx.x, threadIdx.x, sp[0] + blockIdx.y, sp[1], qkv + off, qo + off, kc, vc, qn, kn, cs_table, p, buf, red);
}

// RoPE and cache append without per-head norms: a warp per head of a token, lane l owning dimensions 4 l .. 4 l + 3 (and
// 128 + 4 l .. for heads of 256). The rotation is rope_head's arithmetic (unfused multiplies and adds), so the rows that
// reach the caches equal the one-token kernel's bit for bit. hd and half_rot are multiples of 4.
template <typename T>
__device__ __forceinline__ void store4(T* p, float4 v);
template <>
__device__ __forceinline__ void store4<float>(float* p, float4 v) { *(float4*)p = v; }
template <>
__device__ __forceinline__ void store4<__half>(__half* p, float4 v) {
    const __half2 a = __floats2half2_rn(v.x, v.y), b = __floats2half2_rn(v.z, v.w);
    *(uint2*)p = make_uint2(*(const uint32_t*)&a, *(const uint32_t*)&b);
}

template <typename T>
__global__ void __launch_bounds__(256) qk_rope_fast_kernel(const float* __restrict__ qkv, float* __restrict__ qo, size_t stride, uint32_t rows,
                                                           T* __restrict__ kc, T* __restrict__ vc, const float* __restrict__ cs_table,
                                                           const uint32_t* __restrict__ sp, DecRope p) {
    pdl_launch_dependents();
    const uint32_t heads = p.nh + 2 * p.nkv;
    const uint32_t unit = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (unit >= rows * heads) return;
    const uint32_t tok = unit / heads, h = unit - tok * heads;
    const uint32_t kind = h < p.nh ? 0 : (h < p.nh + p.nkv ? 1 : 2);
    const uint32_t hh = kind == 0 ? h : (kind == 1 ? h - p.nh : h - p.nh - p.nkv);
    const uint32_t pos = sp[0] + tok, hd = p.hd, hr = p.half_rot;
    if (pos >= p.max_len) return;
    const float* src = qkv + (size_t)tok * stride + (kind == 0 ? hh * p.q_stride : (kind == 1 || p.v_from_k) ? p.k_off + hh * hd : p.v_off + hh * hd);
    const float* cs = cs_table + (size_t)(pos - sp[1]) * p.cs_stride + p.cs_off;
    const size_t at = ((size_t)hh * p.max_len + pos) * hd;
    for (uint32_t d0 = 4 * lane; d0 < hd; d0 += 128) {
        float4 v = *(const float4*)(src + d0);
        if (kind != 2 && d0 < 2 * hr) {
            if (p.interleaved) {  // pairs (2 j, 2 j + 1): both in this lane
                const uint32_t j = d0 >> 1;
                const float c0 = cs[j], s0 = cs[hr + j], c1 = cs[j + 1], s1 = cs[hr + j + 1];
                v = make_float4(__fsub_rn(__fmul_rn(v.x, c0), __fmul_rn(v.y, s0)), __fadd_rn(__fmul_rn(v.y, c0), __fmul_rn(v.x, s0)),
                                __fsub_rn(__fmul_rn(v.z, c1), __fmul_rn(v.w, s1)), __fadd_rn(__fmul_rn(v.w, c1), __fmul_rn(v.z, s1)));
            } else {  // pairs (j, j + hr): the partner's four values come from global memory again (L1)
                const bool first = d0 < hr;
                const uint32_t j = first ? d0 : d0 - hr;
                const float4 o = *(const float4*)(src + (first ? d0 + hr : d0 - hr));
                const float4 c = *(const float4*)(cs + j), s = *(const float4*)(cs + hr + j);
                if (first)
                    v = make_float4(__fsub_rn(__fmul_rn(v.x, c.x), __fmul_rn(o.x, s.x)), __fsub_rn(__fmul_rn(v.y, c.y), __fmul_rn(o.y, s.y)),
                                    __fsub_rn(__fmul_rn(v.z, c.z), __fmul_rn(o.z, s.z)), __fsub_rn(__fmul_rn(v.w, c.w), __fmul_rn(o.w, s.w)));
                else
                    v = make_float4(__fadd_rn(__fmul_rn(v.x, c.x), __fmul_rn(o.x, s.x)), __fadd_rn(__fmul_rn(v.y, c.y), __fmul_rn(o.y, s.y)),
                                    __fadd_rn(__fmul_rn(v.z, c.z), __fmul_rn(o.z, s.z)), __fadd_rn(__fmul_rn(v.w, c.w), __fmul_rn(o.w, s.w)));
            }
        }
        if (kind == 0) *(float4*)(qo + (size_t)tok * stride + hh * hd + d0) = v;
        else store4<T>((kind == 1 ? kc : vc) + at + d0, v);
    }
}

// RMS norm of many rows, one CTA of 256 threads per row, the row in registers between the passes (n <= 8192). With x16 the
// row also leaves as f16 operands of the GEMM behind it: multiplied by the power of two that brings its largest magnitude
// into [2^14, 2^15), the inverse factor in unscale[row] (what to_f16_rows_kernel makes of the f32 row); `out` may be null then.
// addend: dense rows that are added to x first (the residual add of the product ahead; x is written back). The three are one pass
// because they are bound by memory: 2048 x 4096 rows take two reads, a write and the f16 rows instead of four reads and three writes.
constexpr int NORM_ROWS_V = 8;
__global__ void __launch_bounds__(256) norm_rows_kernel(float* x, size_t x_stride, float* out, size_t out_stride,
                                                        const float* __restrict__ w, uint32_t n, float pre, float eps, int add,
                                                        __half* __restrict__ x16, float* __restrict__ unscale, const float* __restrict__ addend) {
    __shared__ float red[32];
    const size_t row = blockIdx.x;
    float4* xr = (float4*)(x + row * x_stride);
    float4* o = (float4*)(out + row * out_stride);
    const float4* ar = (const float4*)(addend + row * n);
    const uint32_t n4 = n / 4;
    float4 v[NORM_ROWS_V];
#pragma unroll
    for (int j = 0; j < NORM_ROWS_V; j++) {
        const uint32_t i = threadIdx.x + 256 * j;
        v[j] = i < n4 ? xr[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    if (addend) {
        float4 a[NORM_ROWS_V];
#pragma unroll
        for (int j = 0; j < NORM_ROWS_V; j++) {
            const uint32_t i = threadIdx.x + 256 * j;
            if (i < n4) a[j] = ar[i];
        }
#pragma unroll
        for (int j = 0; j < NORM_ROWS_V; j++) {
            const uint32_t i = threadIdx.x + 256 * j;
            if (i < n4) xr[i] = v[j] = make_float4(v[j].x + a[j].x, v[j].y + a[j].y, v[j].z + a[j].z, v[j].w + a[j].w);
        }
    }
    float s = 0.0f;
#pragma unroll
    for (int j = 0; j < NORM_ROWS_V; j++) {
        const uint32_t i = threadIdx.x + 256 * j;
        if (i < n4) {
            const float4 t = v[j];
            v[j] = make_float4(t.x * pre, t.y * pre, t.z * pre, t.w * pre);
            s += v[j].x * v[j].x + v[j].y * v[j].y + v[j].z * v[j].z + v[j].w * v[j].w;
        }
    }
    const float k = 1.0f / sqrtf(block_sum(s, red) / (float)n + eps);
    float mx = 0.0f;
#pragma unroll
    for (int j = 0; j < NORM_ROWS_V; j++) {
        const uint32_t i = threadIdx.x + 256 * j;
        if (i < n4) {
            float4 t = make_float4(v[j].x * k, v[j].y * k, v[j].z * k, v[j].w * k);
            if (w) {
                const float4 ww = ((const float4*)w)[i];
                t = make_float4(t.x * ww.x, t.y * ww.y, t.z * ww.z, t.w * ww.w);
            }
            if (add) {
                const float4 a = o[i];
                t = make_float4(t.x + a.x, t.y + a.y, t.z + a.z, t.w + a.w);
            }
            if (out) o[i] = t;
            v[j] = t;
            mx = fmaxf(fmaxf(mx, fmaxf(fabsf(t.x), fabsf(t.y))), fmaxf(fabsf(t.z), fabsf(t.w)));
        }
    }
    if (!x16) return;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, d));
    __syncthreads();  // red is read by every thread in block_sum above
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
    __syncthreads();
    mx = red[0];
#pragma unroll
    for (int i = 1; i < 8; i++) mx = fmaxf(mx, red[i]);
    float sc = 1.0f, inv = 1.0f;
    if (mx > 0.0f && mx < INFINITY) {
        int e;
        frexpf(mx, &e);
        const int up = min(100, max(-100, 15 - e));
        sc = ldexpf(1.0f, up);
        inv = ldexpf(1.0f, -up);
    }
    __half* h = x16 + row * n;
#pragma unroll
    for (int j = 0; j < NORM_ROWS_V; j++) {
        const uint32_t i = threadIdx.x + 256 * j;
        if (i < n4) *(uint2*)(h + 4 * (size_t)i) = make_uint2(pack_h2f(v[j].x * sc, v[j].y * sc), pack_h2f(v[j].z * sc, v[j].w * sc));
    }
    if (threadIdx.x == 0) unscale[row] = inv;
}

__global__ void __launch_bounds__(256) glu_rows_kernel(const float* __restrict__ g, size_t g_stride, const float* __restrict__ u, size_t u_stride,
                                                       float* __restrict__ out, size_t out_stride, uint32_t n, int gelu) {
    const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (i >= n) return;
    const size_t r = blockIdx.y;
    const float4 a4 = *(const float4*)(g + r * g_stride + i), u4 = *(const float4*)(u + r * u_stride + i);
    const float a[4] = {a4.x, a4.y, a4.z, a4.w}, uu[4] = {u4.x, u4.y, u4.z, u4.w};
    float o[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {  // the arithmetic of glu_kernel (decode_ops.cu)
        float v;
        if (gelu) {
            const float K2 = 2.0f * 0.7978846f;
            const float t = K2 * (a[j] + 0.044715f * a[j] * a[j] * a[j]);
            v = a[j] / (1.0f + expf(-t));
        } else {
            v = a[j] / (1.0f + expf(-a[j]));
        }
        o[j] = v * uu[j];
    }
    *(float4*)(out + r * out_stride + i) = make_float4(o[0], o[1], o[2], o[3]);
}

// act(g) * u of a whole row by one CTA, the row in registers (n <= 16384): the f32 result and, with x16, the f16 operand
// rows of the product behind it with their power-of-two row factor (what to_f16_rows_kernel makes of the f32 row), so that
// product needs no conversion launch and the row is not read again.
// `out` may be null. Bound by memory: 512 threads with half of their loads at a time ahead of the arithmetic, so that 64 registers are enough for two
// CTAs an SM, one's loads under the other's stores (all loads at once, 79 registers, one CTA: 76 us for 2048 x 14336, this way 53; the bytes take 45), and no f32 rows where nobody reads them
// (256 threads, load by load, with the f32 rows: 107 us for 2048 x 14336). With the residual adds in the norms: 20.9 -> 20.0 ms a step of
// 2048 tokens through 16 layers of hidden size 4096.
constexpr int GLU_ROW_V = 8, GLU_THREADS = 512, GLU_BATCH = 4;
__global__ void __launch_bounds__(GLU_THREADS, 2) glu_rows_f16_kernel(const float* __restrict__ g, size_t g_stride, const float* __restrict__ u, size_t u_stride,
                                                                   float* __restrict__ out, size_t out_stride, uint32_t n, int gelu,
                                                                   __half* __restrict__ x16, float* __restrict__ unscale) {
    __shared__ float red[GLU_THREADS / 32];
    const size_t r = blockIdx.x;
    const uint32_t n4 = n / 4;
    float4 v[GLU_ROW_V];
    float mx = 0.0f;
#pragma unroll
    for (int j0 = 0; j0 < GLU_ROW_V; j0 += GLU_BATCH) {
        float4 w[GLU_BATCH];
#pragma unroll
        for (int j = 0; j < GLU_BATCH; j++) {
            const uint32_t i = threadIdx.x + GLU_THREADS * (j0 + j);
            v[j0 + j] = w[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (i < n4) {
                v[j0 + j] = ((const float4*)(g + r * g_stride))[i];
                w[j] = ((const float4*)(u + r * u_stride))[i];
            }
        }
#pragma unroll
        for (int j = 0; j < GLU_BATCH; j++) {
            const uint32_t i = threadIdx.x + GLU_THREADS * (j0 + j);
            if (i < n4) {
                float4& x = v[j0 + j];
                const float a[4] = {x.x, x.y, x.z, x.w}, uu[4] = {w[j].x, w[j].y, w[j].z, w[j].w};
                float o[4];
#pragma unroll
                for (int e = 0; e < 4; e++) {  // the arithmetic of glu_rows_kernel
                    float t;
                    if (gelu) {
                        const float K2 = 2.0f * 0.7978846f;
                        const float z = K2 * (a[e] + 0.044715f * a[e] * a[e] * a[e]);
                        t = a[e] / (1.0f + expf(-z));
                    } else {
                        t = a[e] / (1.0f + expf(-a[e]));
                    }
                    o[e] = t * uu[e];
                    mx = fmaxf(mx, fabsf(o[e]));
                }
                x = make_float4(o[0], o[1], o[2], o[3]);
                if (out) ((float4*)(out + r * out_stride))[i] = x;
            }
        }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, d));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
    __syncthreads();
    mx = red[0];
#pragma unroll
    for (int i = 1; i < GLU_THREADS / 32; i++) mx = fmaxf(mx, red[i]);
    float sc = 1.0f, inv = 1.0f;
    if (mx > 0.0f && mx < INFINITY) {
        int e;
        frexpf(mx, &e);
        const int up = min(100, max(-100, 15 - e));
        sc = ldexpf(1.0f, up);
        inv = ldexpf(1.0f, -up);
    }
    __half* h = x16 + r * n;
#pragma unroll
    for (int j = 0; j < GLU_ROW_V; j++) {
        const uint32_t i = threadIdx.x + GLU_THREADS * j;
        if (i < n4) *(uint2*)(h + 4 * (size_t)i) = make_uint2(pack_h2f(v[j].x * sc, v[j].y * sc), pack_h2f(v[j].z * sc, v[j].w * sc));
    }
    if (threadIdx.x == 0) unscale[r] = inv;
}

template <bool ADD>
__global__ void __launch_bounds__(256) rows_op_kernel(float* __restrict__ dst, size_t dst_stride, const float* __restrict__ src, size_t src_stride,
                                                      uint32_t n) {
    const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (i >= n) return;
    const size_t r = blockIdx.y;
    float4 s = *(const float4*)(src + r * src_stride + i);
    float4* d = (float4*)(dst + r * dst_stride + i);
    if (ADD) {
        const float4 o = *d;
        s = make_float4(o.x + s.x, o.y + s.y, o.z + s.z, o.w + s.w);
    }
    *d = s;
}

}  // namespace

cudaError_t launch_qk_rope_rows(const float* qkv, float* qo, size_t stride, uint32_t rows, void* kc, void* vc, int kv_f16, const float* qn,
                                const float* kn, const float* cs, const uint32_t* sp, const DecRope& p, cudaStream_t st) {
    if (p.hd > 256 || p.hd % 32 || 2 * p.half_rot > p.hd || rows == 0 || rows > 65535) return cudaErrorInvalidValue;
    // (the fast kernel reads a rotation partner's values from the input again: input and output must not overlap)
    const size_t in_extent = std::max<size_t>((size_t)(p.nh - 1) * p.q_stride + p.hd, std::max<size_t>(p.k_off, p.v_off) + (size_t)p.nkv * p.hd);
    const bool apart = qo + (size_t)p.nh * p.hd <= qkv || qkv + in_extent <= qo;
    if (apart && !qn && !kn && !p.v_norm && p.half_rot % 4 == 0 && stride % 4 == 0 && p.q_stride % 4 == 0 && p.k_off % 4 == 0 && p.v_off % 4 == 0 &&
        p.cs_off % 4 == 0 && p.cs_stride % 4 == 0 && (((uintptr_t)qkv | (uintptr_t)qo | (uintptr_t)cs) & 15) == 0) {
        const size_t units = (size_t)rows * (p.nh + 2 * p.nkv);
        const unsigned grid = (unsigned)((units + 7) / 8);
        if (kv_f16)
            qk_rope_fast_kernel<__half><<<grid, 256, 0, st>>>(qkv, qo, stride, rows, (__half*)kc, (__half*)vc, cs, sp, p);
        else
            qk_rope_fast_kernel<float><<<grid, 256, 0, st>>>(qkv, qo, stride, rows, (float*)kc, (float*)vc, cs, sp, p);
        return cudaGetLastError();
    }
    const dim3 grid(p.nh + 2 * p.nkv, rows);
    if (kv_f16)
        qk_rope_rows_kernel<__half><<<grid, p.hd, 0, st>>>(qkv, qo, stride, (__half*)kc, (__half*)vc, qn, kn, cs, sp, p);
    else
        qk_rope_rows_kernel<float><<<grid, p.hd, 0, st>>>(qkv, qo, stride, (float*)kc, (float*)vc, qn, kn, cs, sp, p);
    return cudaGetLastError();
}

bool norm_rows_supports(uint32_t n, const float* x, const float* out, const float* w, size_t x_stride, size_t out_stride) {
    return n % 4 == 0 && n <= 1024 * NORM_ROWS_V && x_stride % 4 == 0 && out_stride % 4 == 0 && (((uintptr_t)x | (uintptr_t)out | (uintptr_t)w) & 15) == 0;
}

cudaError_t launch_norm_rows(float* x, size_t x_stride, float* out, size_t out_stride, const float* w, const DecNorm& p, uint32_t rows,
                             void* x16, float* unscale, const float* addend, cudaStream_t st) {
    if (((uintptr_t)addend & 15) || (!out && (p.add || !x16))) return cudaErrorInvalidValue;
    if (!norm_rows_supports(p.n, x, out, w, x_stride, out_stride) || rows == 0 || (x16 && (p.n % 8 || ((uintptr_t)x16 & 15)))) return cudaErrorInvalidValue;
    norm_rows_kernel<<<rows, 256, 0, st>>>(x, x_stride, out, out_stride, w, p.n, p.pre, p.eps, (int)p.add, (__half*)x16, unscale, addend);
    return cudaGetLastError();
}

bool glu_rows_f16_supports(uint32_t n) { return n % 8 == 0 && n <= 4 * GLU_THREADS * GLU_ROW_V; }

cudaError_t launch_glu_rows(const float* g, size_t g_stride, const float* u, size_t u_stride, float* out, size_t out_stride, uint32_t n,
                            uint32_t rows, int gelu, cudaStream_t st, void* x16, float* unscale) {
    if (n % 4 || g_stride % 4 || u_stride % 4 || out_stride % 4 || rows == 0 || rows > 65535 || (((uintptr_t)g | (uintptr_t)u | (uintptr_t)out) & 15))
        return cudaErrorInvalidValue;
    if (!out && !x16) return cudaErrorInvalidValue;
    if (x16) {
        if (!glu_rows_f16_supports(n) || ((uintptr_t)x16 & 15)) return cudaErrorInvalidValue;
        glu_rows_f16_kernel<<<rows, GLU_THREADS, 0, st>>>(g, g_stride, u, u_stride, out, out_stride, n, gelu, (__half*)x16, unscale);
        return cudaGetLastError();
    }
    glu_rows_kernel<<<dim3((n / 4 + 255) / 256, rows), 256, 0, st>>>(g, g_stride, u, u_stride, out, out_stride, n, gelu);
    return cudaGetLastError();
}

cudaError_t launch_rows_op(float* dst, size_t dst_stride, const float* src, size_t src_stride, uint32_t n, uint32_t rows, bool add,
                           cudaStream_t st) {
    if (n % 4 || dst_stride % 4 || src_stride % 4 || rows == 0 || rows > 65535 || (((uintptr_t)dst | (uintptr_t)src) & 15)) return cudaErrorInvalidValue;
    const dim3 grid((n / 4 + 255) / 256, rows);
    if (add)
        rows_op_kernel<true><<<grid, 256, 0, st>>>(dst, dst_stride, src, src_stride, n);
    else
        rows_op_kernel<false><<<grid, 256, 0, st>>>(dst, dst_stride, src, src_stride, n);
    return cudaGetLastError();
}

}  // namespace b2
