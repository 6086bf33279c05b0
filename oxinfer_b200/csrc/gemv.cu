// One-token products of FP8 matrices whose scale blocks the small-batch kernel (gemv_mma.cu) does not take: other widths than 128
// columns. Hardware e4m3x2 -> f16x2 conversion and f32 multiply-adds with the f32 vector.
//
// A warp owns two weight rows at a time (or, for the fused SiLU / GELU pair, the same row of the gate and the up matrix): every lane
// issues the 16-byte loads of both before using either, and reads its slice of the vector from shared memory once for both. The vector
// is staged once per CTA, with its 16-byte slots permuted so that the eight lanes of a shared-memory phase, which read 64 bytes each
// at a 64-byte stride, fall on different banks.
#include <cuda_fp8.h>

#include <algorithm>
#include <atomic>
#include <cstdio>

#include "gemv_core.cuh"

namespace b2 {

using namespace gemv_core;

namespace {

constexpr int GEMV_THREADS = 256;
constexpr int GEMV_WARPS = GEMV_THREADS / 32;
constexpr int ITER_K = 512;  // 16 e4m3 bytes per lane

struct Regs {
    uint4 q;
    float s;
};
__device__ __forceinline__ void load_row(const WeightDev& w, size_t row, int k0, Regs& r) {
    r.q = ldg_stream(w.p0 + row * w.n_in + k0);
    r.s = w.p1 ? __ldg((const float*)w.p1 + ((w.bs_row0 + row) / w.bs_rows) * w.bs_ncb + k0 / w.bs_cols) : 1.0f;
}
__device__ __forceinline__ float part(uint32_t q, float4 xx, float acc) {
    __half2_raw h01 = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(q & 0xffff), __NV_E4M3);
    __half2_raw h23 = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(q >> 16), __NV_E4M3);
    float2 f01 = __half22float2(*(const __half2*)&h01), f23 = __half22float2(*(const __half2*)&h23);
    acc = fmaf(f01.x, xx.x, acc);
    acc = fmaf(f01.y, xx.y, acc);
    acc = fmaf(f23.x, xx.z, acc);
    return fmaf(f23.y, xx.w, acc);
}
// Slot g -> g with its low two bits xor-ed by bits 3 and 4: lanes L = 0..7 of a phase that read slots 4 L + i (a 64-byte
// stride) then cover all eight 16-byte bank groups for every i.
__device__ __forceinline__ int swizzle(int g) { return g ^ ((((g >> 3) & 1) << 1) | ((g >> 4) & 1)); }

template <bool PAIR>
__global__ void __launch_bounds__(GEMV_THREADS, 3)
gemv_f8_kernel(WeightDev w, WeightDev w2, const float* __restrict__ x, float* __restrict__ y, int mode, const float* __restrict__ gate) {
    extern __shared__ __align__(128) uint8_t smem[];
    pdl_launch_dependents();
    const int K = (int)w.n_in;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t n_out = w.n_out;
    constexpr int RW = PAIR ? 1 : 2;  // output rows per warp pass
    const size_t r_first = ((size_t)blockIdx.x * GEMV_WARPS + warp) * RW, r_step = (size_t)gridDim.x * GEMV_WARPS * RW;
    Regs na, nb;
    auto fetch = [&](size_t r0, int k0) {
        if (k0 < K) {
            load_row(w, r0, k0, na);
            load_row(PAIR ? w2 : w, PAIR ? r0 : min(r0 + 1, n_out - 1), k0, nb);
        }
    };
    if (r_first < n_out) fetch(r_first, lane * 16);
    pdl_wait();
    float* xf = (float*)smem;
    for (int g = threadIdx.x; g < K / 4; g += GEMV_THREADS) ((float4*)xf)[swizzle(g)] = ((const float4*)x)[g];
    __syncthreads();
    for (size_t r0 = r_first; r0 < n_out; r0 += r_step) {
        float acc_a = 0.0f, acc_b = 0.0f;
        for (int k0 = lane * 16; k0 < K; k0 += ITER_K) {
            if (k0 >= ITER_K || r0 != r_first) fetch(r0, k0);  // the first step's loads were issued before the wait
            const uint32_t qa[4] = {na.q.x, na.q.y, na.q.z, na.q.w}, qb[4] = {nb.q.x, nb.q.y, nb.q.z, nb.q.w};
            float pa = 0.0f, pb = 0.0f;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float4 xx = ((const float4*)xf)[swizzle((k0 >> 2) + i)];
                pa = part(qa[i], xx, pa);
                pb = part(qb[i], xx, pb);
            }
            acc_a = fmaf(pa, na.s, acc_a);
            acc_b = fmaf(pb, nb.s, acc_b);
        }
        const float sa = warp_sum(acc_a), sb = warp_sum(acc_b);
        if (lane) continue;
        if (PAIR) {
            y[r0] = (mode == B2_MODE_SILU_PAIR ? silu(sa) : gelu_tanh(sa)) * sb;
            continue;
        }
#pragma unroll
        for (int r = 0; r < 2; r++) {
            if (r0 + r >= n_out) break;
            const float a = r ? sb : sa;
            float* o = y + r0 + r;
            if (mode == B2_MODE_STORE) *o = a;
            else if (mode == B2_MODE_ADD) *o += a;
            else *o += a * (1.0f / (1.0f + __expf(-gate[0])));
        }
    }
}

}  // namespace

bool gemv_supports(const WeightDev& w) {
    return gemv_mma_supports(w) ||
           (w.fmt == B2_FMT_F8E4M3 && w.n_in % 16 == 0 && w.n_in * 4 <= 200 * 1024 && (w.p1 == nullptr || w.bs_cols % 16 == 0));
}

cudaError_t launch_gemv_f8_float(const WeightDev& w, const WeightDev* up, const float* x, float* y, int mode, const float* gate, int sm_count,
                                 cudaStream_t st, bool pdl) {
    if (w.fmt != B2_FMT_F8E4M3) return cudaErrorInvalidValue;
    const bool pair = mode == B2_MODE_SILU_PAIR || mode == B2_MODE_GELU_PAIR;
    auto kern = pair ? gemv_f8_kernel<true> : gemv_f8_kernel<false>;
    const size_t smem = (w.n_in * 4 + 127) / 128 * 128;
    if (cudaError_t e = ensure_dynamic_smem((const void*)kern, smem); e != cudaSuccess) return e;
    const size_t rows_per_cta = (size_t)GEMV_WARPS * (pair ? 1 : 2), groups = (w.n_out + rows_per_cta - 1) / rows_per_cta;
    const size_t per_sm = std::min<size_t>(3, std::max<size_t>(1, (size_t)(220 * 1024) / (smem + 1024)));
    const size_t grid = std::min(groups, (size_t)sm_count * per_sm);
    return launch_k(kern, dim3((unsigned)grid), dim3(GEMV_THREADS), smem, st, pdl, w, pair ? *up : w, x, y, mode, gate);
}

}  // namespace b2

// =============================================================================================
// b2_matvec_q4k_noalloc: the Q4_K matrix-vector product for callers that must not allocate.
//
// Some hosts of this library cannot call cudaMalloc at the moment they need a product: a serving
// process that handed the whole device to its own arena at start-up (oxinfer's decode plans carve
// every buffer out of one arena they own, src/cuda_decode.rs:372-383) has nothing left for the
// runtime to give, and a latency-critical decode loop must not enter the allocator at all. The
// product splits its vector in shared memory, so the call needs no device memory of its own, and
// calls on different streams do not meet. A call whose y overlaps x reads x from a copy in a fixed
// array of the library (every CTA reads x for itself, while others may already store y); all such
// calls share the array. n_in is limited to its B2_NOALLOC_MAX_K = 16384 values.
// =============================================================================================
namespace b2 {
namespace {
constexpr size_t NOALLOC_MAX_K = 16384;
constexpr int NOALLOC_MAX_DEVICES = 64;
std::atomic<int> g_noalloc_sms[NOALLOC_MAX_DEVICES];
static __device__ __align__(256) float g_noalloc_x[NOALLOC_MAX_K];
std::atomic<float*> g_noalloc_ptr[NOALLOC_MAX_DEVICES];  // its address on each device

int noalloc_fail(char* err, size_t err_len, int code, const char* text, cudaError_t e = cudaSuccess) {
    if (err && err_len) {
        if (e != cudaSuccess)
            snprintf(err, err_len, "[b200qmm: matvec_q4k_noalloc: %s: %s]", text, cudaGetErrorString(e));
        else
            snprintf(err, err_len, "[b200qmm: matvec_q4k_noalloc: %s]", text);
    }
    return code;
}
}  // namespace
}  // namespace b2

extern "C" __attribute__((visibility("default"))) int b2_matvec_q4k_noalloc(const void* w_blocks_dev, size_t n_out, size_t n_in,
                                                                             const float* x_dev, float* y_dev, void* cuda_stream,
                                                                             char* err, size_t err_len) {
    using namespace b2;
    if (!w_blocks_dev || !x_dev || !y_dev || n_out == 0) return noalloc_fail(err, err_len, B2_ERR_ARG, "null pointer or empty matrix");
    if (n_in == 0 || n_in % 256 != 0) return noalloc_fail(err, err_len, B2_ERR_ARG, "n_in must be a positive multiple of 256 (Q4_K super-blocks)");
    if (n_in > NOALLOC_MAX_K) {
        if (err && err_len)
            snprintf(err, err_len, "[b200qmm: matvec_q4k_noalloc: n_in = %zu exceeds the built-in scratch (at most %zu); use b2_matvec_dev]", n_in,
                     NOALLOC_MAX_K);
        return B2_ERR_ARG;
    }
    if (((uintptr_t)w_blocks_dev & 15) || ((uintptr_t)x_dev & 3) || ((uintptr_t)y_dev & 3))
        return noalloc_fail(err, err_len, B2_ERR_ARG, "weights must be 16-byte aligned, x and y 4-byte aligned");
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return noalloc_fail(err, err_len, B2_ERR_CUDA, "cudaGetDevice", e);
    if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) return noalloc_fail(err, err_len, B2_ERR_ARG, "device ordinal out of range");
    int sms = g_noalloc_sms[dev].load(std::memory_order_acquire);
    if (!sms) {
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess || sms <= 0) return noalloc_fail(err, err_len, B2_ERR_CUDA, "cudaDeviceGetAttribute", e);
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_x);
        if (e != cudaSuccess || !p) return noalloc_fail(err, err_len, B2_ERR_CUDA, "cudaGetSymbolAddress(scratch)", e);
        g_noalloc_ptr[dev].store((float*)p, std::memory_order_relaxed);
        g_noalloc_sms[dev].store(sms, std::memory_order_release);
    }
    WeightDev w{};
    w.fmt = B2_FMT_Q4_K;
    w.n_out = n_out;
    w.n_in = n_in;
    w.p0 = (const uint8_t*)w_blocks_dev;
    GemvIn in;
    in.x = x_dev;
    if ((uintptr_t)(y_dev + n_out) > (uintptr_t)x_dev && (uintptr_t)(x_dev + n_in) > (uintptr_t)y_dev) {
        float* copy = g_noalloc_ptr[dev].load(std::memory_order_relaxed);
        e = cudaMemcpyAsync(copy, x_dev, n_in * sizeof(float), cudaMemcpyDeviceToDevice, (cudaStream_t)cuda_stream);
        if (e != cudaSuccess) return noalloc_fail(err, err_len, B2_ERR_CUDA, "copy of x", e);
        in.x = copy;
    }
    e = launch_gemv_mma(w, nullptr, in, 1, y_dev, 0, B2_MODE_STORE, nullptr, 0, sms, (cudaStream_t)cuda_stream, false);
    if (e != cudaSuccess) return noalloc_fail(err, err_len, B2_ERR_CUDA, "gemv kernel", e);
    return B2_OK;
}
