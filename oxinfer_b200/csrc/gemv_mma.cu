// The products of one to eight tokens of the five tuned formats, and the activation split's own kernel (gemv_mma_kernel.cuh).
#include "gemv_mma_kernel.cuh"

namespace b2 {

namespace {

__global__ void __launch_bounds__(256) split_kernel(const float* __restrict__ x, size_t x_stride, const float* __restrict__ w, float pre, int K, uint8_t* out,
                                                    size_t out_stride, int fast, int halves) {
    pdl_launch_dependents();
    pdl_wait();
    // (the tokens along x: there may be more than the 65,535 that y holds)
    const int blk = blockIdx.y * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31, nb = (K + 255) / 256;
    if (blk >= nb) return;
    const int k = blk * 256;
    const SplitIn in = split_load(x + (size_t)blockIdx.x * x_stride + k, w ? w + k : nullptr, K - k, lane);
    uint8_t* r = out + (size_t)blockIdx.x * out_stride;
    if (halves) {
        const SplitHalves d = split_halves(in, pre);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            uint8_t* o = r + (size_t)blk * SPLIT_HALVES + (4 * h + (lane >> 3)) * 128 + (lane & 3) * 16 + ((lane >> 2) & 1) * 8;
            *(uint2*)o = d.hi[h];
            *(uint2*)(o + 64) = d.lo[h];
        }
        if (lane == 0) *(float4*)(r + (size_t)nb * SPLIT_HALVES + (size_t)blk * SPLIT_AUX) = make_float4(d.xs, d.ssq, 0.0f, 0.0f);
        return;
    }
    const SplitDigits<3> d = split_digits(in, pre, fast);
#pragma unroll
    for (int h = 0; h < 2; h++) {
        int pair, in16;
        split_digit_at(h, lane, pair, in16);
#pragma unroll
        for (int p = 0; p < 3; p++) *(uint32_t*)(r + (size_t)blk * SPLIT_DIGITS + pair * 192 + p * 64 + in16) = d.d[h][p];
    }
    uint8_t* aux = r + (size_t)nb * SPLIT_DIGITS + (size_t)blk * SPLIT_AUX;
    if (lane == 0) *(float4*)aux = make_float4(d.xs, d.ssq, 0.0f, 0.0f);
    if ((lane & 7) == 0) {
        ((int*)(aux + 16))[lane >> 3] = d.s[0];
        ((int*)(aux + 16))[4 + (lane >> 3)] = d.s[1];
    }
}

template <class F>
cudaError_t launch_f(Args& a, bool pair, int sm_count, cudaStream_t st, bool pdl, const GemvGroups* gt = nullptr) {
    if (a.T == 1) return pair ? launch_t<F, true, 1>(a, sm_count, st, pdl, gt) : launch_t<F, false, 1>(a, sm_count, st, pdl, gt);
    if (a.T <= 4) return pair ? launch_t<F, true, 4>(a, sm_count, st, pdl, gt) : launch_t<F, false, 4>(a, sm_count, st, pdl, gt);
    if (a.T <= 6) return pair ? launch_t<F, true, 6>(a, sm_count, st, pdl, gt) : launch_t<F, false, 6>(a, sm_count, st, pdl, gt);
    return pair ? launch_t<F, true, 8>(a, sm_count, st, pdl, gt) : launch_t<F, false, 8>(a, sm_count, st, pdl, gt);
}

}  // namespace

bool gemv_mma_supports(const WeightDev& w) {
    // (the longest rows: a unit of eight tokens' activations has to fit beside the rings and the norm's sums, launch_t)
    if (((uintptr_t)w.p0 & 15) || w.n_in > (w.fmt == B2_FMT_F8E4M3 ? 51200 : 58512)) return false;
    switch (w.fmt) {
        case B2_FMT_MLX4:
        case B2_FMT_Q4_K: return w.n_in % 256 == 0;
        case B2_FMT_Q6_K: return w.n_in % 256 == 0 && (((uintptr_t)w.p1 | (uintptr_t)w.p2) & 15) == 0;
        case B2_FMT_Q8_0: return w.n_in % 64 == 0 && ((uintptr_t)w.p1 & 3) == 0;
        // (its scales have to be per 128 columns: other block shapes take the float kernel of gemv.cu)
        case B2_FMT_F8E4M3: return w.n_in % 16 == 0 && (w.p1 == nullptr || w.bs_cols == 128);
        default: return false;
    }
}
size_t split_blocks_of(size_t K) { return split_blocks(K); }
size_t split_bytes_of(size_t K, bool halves) { return split_bytes(K, halves); }
bool gemv_mma_halves(const WeightDev& w) { return w.fmt == B2_FMT_F8E4M3; }

cudaError_t launch_gemv_mma(const WeightDev& w, const WeightDev* up, const GemvIn& in, int T, float* y, size_t y_stride, int mode, const float* gate,
                            size_t gate_stride, int sm_count, cudaStream_t st, bool pdl) {
    if (!gemv_mma_supports(w) || T < 1 || T > 8) return cudaErrorInvalidValue;
    if (in.status && gemv_tc_supports(w)) return launch_gemv_tc(w, up, in, T, y, y_stride, mode, gate, gate_stride, sm_count, st, pdl);
    const bool pair = mode == B2_MODE_SILU_PAIR || mode == B2_MODE_GELU_PAIR;
    Args a{};
    a.w = w;
    a.w2 = pair ? *up : w;
    a.x = in.x;
    a.x_stride = in.x_stride;
    a.nw = in.norm_w;
    a.pre = in.pre;
    a.norm = in.norm;
    a.eps = in.eps;
    a.rec = in.rec;
    a.rec_stride = in.rec_stride;
    a.fast = in.fast;
    a.y = y;
    a.y_stride = y_stride;
    a.gate = gate;
    a.gate_stride = gate_stride;
    a.mode = mode;
    a.T = T;
    switch (w.fmt) {
        case B2_FMT_MLX4: return launch_f<F4<true, true>>(a, pair, sm_count, st, pdl);
        case B2_FMT_Q4_K: return launch_f<F4<false, false>>(a, pair, sm_count, st, pdl);
        case B2_FMT_Q6_K: return launch_f<F6>(a, pair, sm_count, st, pdl);
        case B2_FMT_Q8_0: return launch_f<F8B<false>>(a, pair, sm_count, st, pdl);
        case B2_FMT_F8E4M3: return launch_f<F8B<true>>(a, pair, sm_count, st, pdl);
        default: return cudaErrorInvalidValue;
    }
}

// The most rows of K values that a group's activations fit for beside the rings (launch_t: two warp groups' sums are 16 KB).
int gemv_groups_most(size_t K) {
    const size_t nb = split_blocks(K), fixed = (size_t)WARPS * F4<false, false>::SLOTS * F4<false, false>::UNIT_BYTES + 16384 + 512;
    for (size_t tp : {8, 4, 1})
        if (fixed + nb * tp * (SPLIT_DIGITS + 4 + 4 + 32) <= SMEM_MAX) return (int)tp;
    return 0;
}
cudaError_t launch_gemv_groups(const WeightDev& w, const WeightDev* up, const float* x, size_t x_stride, const GemvGroups& groups, int most, float* y,
                               size_t y_stride, int mode, bool fast, int sm_count, cudaStream_t st) {
    if (!gemv_mma_supports(w) || groups.n < 1 || most < 1 || most > 8) return cudaErrorInvalidValue;
    const bool pair = mode == B2_MODE_SILU_PAIR || mode == B2_MODE_GELU_PAIR;
    Args a{};
    a.w = w;
    a.w2 = pair ? *up : w;
    a.x = x;
    a.x_stride = x_stride;
    a.pre = 1.0f;
    a.fast = fast;
    a.y = y;
    a.y_stride = y_stride;
    a.mode = mode;
    a.T = most;
    if (w.fmt == B2_FMT_MLX4) return launch_f<F4<true, false>>(a, pair, sm_count, st, true, &groups);
    if (w.fmt == B2_FMT_Q4_K) return launch_f<F4<false, false>>(a, pair, sm_count, st, true, &groups);
    return cudaErrorInvalidValue;
}

cudaError_t launch_split(const float* x, size_t x_stride, const float* norm_w, float pre, size_t K, int tokens, uint8_t* rec, size_t rec_stride, bool halves,
                         bool fast, cudaStream_t st, bool pdl) {
    if (tokens < 1 || K == 0 || K % 4) return cudaErrorInvalidValue;
    const unsigned nb = (unsigned)split_blocks(K);
    return launch_k(split_kernel, dim3((unsigned)tokens, (nb + 7) / 8), dim3(256), 0, st, pdl, x, x_stride, norm_w, pre, (int)K, rec, rec_stride, (int)fast, (int)halves);
}

}  // namespace b2
