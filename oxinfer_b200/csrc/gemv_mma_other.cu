// The products of one to four tokens of the other GGUF block formats, for rows of whole runs of 256 values (gemv_mma_other.cuh).
#include "gemv_mma_kernel.cuh"
#include "gemv_mma_other.cuh"

namespace b2 {

namespace {

template <int FMT>
bool fits(const WeightDev& w, int T) {
    using F = Fo<FMT>;
    const uintptr_t align = FMT == B2_FMT_Q3_K ? 2 : F::PIECE;
    const size_t tp = T == 1 ? 1 : 4, fixed = (size_t)WARPS * F::SLOTS * F::UNIT_BYTES + 16384 + 512;
    return w.n_in % 256 == 0 && (uintptr_t)w.p0 % align == 0 && fixed + split_blocks(w.n_in) * tp * (4 * 256 + 32 + 4 + 4) <= SMEM_MAX;
}

template <int FMT>
cudaError_t launch(Args& a, bool pair, int sm_count, cudaStream_t st) {
    if (a.T == 1) return pair ? launch_t<Fo<FMT>, true, 1>(a, sm_count, st, true) : launch_t<Fo<FMT>, false, 1>(a, sm_count, st, true);
    return pair ? launch_t<Fo<FMT>, true, 4>(a, sm_count, st, true) : launch_t<Fo<FMT>, false, 4>(a, sm_count, st, true);
}

bool fits_any(const WeightDev& w, int T) {
    switch (w.fmt) {
#define B2_FITS(F) \
    case F: return fits<F>(w, T);
        B2_FITS(B2_FMT_Q4_0) B2_FITS(B2_FMT_Q4_1) B2_FITS(B2_FMT_Q5_0) B2_FITS(B2_FMT_Q5_1) B2_FITS(B2_FMT_Q2_K) B2_FITS(B2_FMT_Q3_K) B2_FITS(B2_FMT_Q5_K)
        B2_FITS(B2_FMT_IQ4_NL) B2_FITS(B2_FMT_IQ4_XS) B2_FITS(B2_FMT_MXFP4) B2_FITS(B2_FMT_NVFP4)
#undef B2_FITS
        default: return false;
    }
}

cudaError_t launch_any(Args& a, bool pair, int sm_count, cudaStream_t st) {
    B2_OTHER_SWITCH(a.w.fmt, launch<FMT>(a, pair, sm_count, st))
}

}  // namespace

int gemv_mma_other_tokens(const WeightDev& w) { return fits_any(w, 4) ? 4 : fits_any(w, 1) ? 1 : 0; }

cudaError_t launch_gemv_mma_other(const WeightDev& w, const WeightDev* up, const float* x, size_t x_stride, float* y, size_t y_stride, int nt, int mode,
                                  const float* gate, int sm_count, cudaStream_t st) {
    const int most = gemv_mma_other_tokens(w);
    if (!most || nt < 1) return cudaErrorInvalidValue;
    const bool pair = mode == B2_MODE_SILU_PAIR || mode == B2_MODE_GELU_PAIR;
    for (int i = 0; i < nt; i += most) {
        Args a{};
        a.w = w;
        a.w2 = pair ? *up : w;
        a.x = x + (size_t)i * x_stride;
        a.x_stride = x_stride;
        a.pre = 1.0f;
        a.y = y + (size_t)i * y_stride;
        a.y_stride = y_stride;
        a.gate = gate;
        a.mode = mode;
        a.T = std::min(most, nt - i);
        if (cudaError_t e = launch_any(a, pair, sm_count, st); e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace b2
