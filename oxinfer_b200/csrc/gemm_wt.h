// Host side of gemm_wt.cu and gemm_wp.cu: dequant-GEMM with the weights in tensor memory and the tokens on the instruction's N side.
#pragma once
#include <cuda.h>

#include "kernels.h"

namespace b2 {

typedef CUresult (*TensorMapEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                      const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
TensorMapEncodeFn tensor_map_encode();  // cuTensorMapEncodeTiled, or null (gemm_tc.cu)

// Maps of f16 activations [rows][n_in] as [n_in / 64][rows][64]: map i copies 16 (i + 1) rows of one or two groups of 64 k, group by group.
// (One copy a stage: the copying warp issues one in about 100 cycles.)
struct XMaps {
    CUtensorMap m[8];
};
struct GemmWt {
    XMaps x;
    CUtensorMap w, w2;  // (w2: Q6_K's second plane)
    int n_max = 0, splits = 1, x_terms = 1, lo_row0 = 0, n_raw = 0, n_b = 0, n_a = 0, groups = 1;
    size_t smem = 0;
};
// Parts of K of a dense product.
int wt_splits(size_t K);
// x16: f16 [x_rows][n_in], `tokens` of them in the longest tile (at most 128 a tile). x_terms 2: the second terms lo_row0 rows below.
// grouped: w.p0 stacks `experts` matrices of n_out rows. false: no tensor map could be made.
bool gemm_wt_encode(GemmWt* g, const WeightDev& w, size_t experts, const void* x16, size_t x_rows, size_t tokens, int x_terms, size_t lo_row0, bool grouped);
// tiles (device; grouped launches): n_tiles of them; null: `t` tokens in order. y rows y_ld elements apart; more[0 .. n_more): other ranks'
// copies of an f32 y.
cudaError_t launch_gemm_wt(const GemmWt& g, const WeightDev& w, size_t t, const WtTile* tiles, int n_tiles, void* y, int y_dtype, size_t y_ld, float* const* more, int n_more,
                           GemmStatus* status, const float* row_unscale, cudaStream_t st);
// Maps first .. last of a set, `groups` of 64 k a copy.
bool gemm_x_maps(XMaps* x, int first, int last, const void* x16, size_t rows, size_t n_in, int groups);

// The CTA-pair form (gemm_wp.cu), one-term operands, or grouped Q4_K with two-term ones. A grouped launch's tiles hold up to WP_TILE_ROWS rows
// (two-term: 128).
constexpr int WP_MOST_ROWS = 256, WP_TILE_ROWS = 160;
struct WpShare {  // how a dense launch is shared out (Segments in gemm_wp.cu)
    int pieces, snap, whole, split;
    int units, longer;  // a piece's units of 32 tokens, and how many of the first pieces have one more
};
struct GemmWp {
    XMaps x;
    CUtensorMap w, w2, y;
    int pairs = 0;
    int busy = 0;                         // a dense launch's pairs that have segments
    WpShare share = {};
    int lo_row0 = 0;                      // grouped Q4_K launches with two-term operands: the activations' second terms, rows below the first
    bool staged = false;                  // the results can leave through the copy engine
};
// Fills in how a dense launch is shared out and returns an estimate of its time in cycles.
double gemm_wp_share(GemmWp* g, size_t n_out, size_t t, size_t n_in, int sm_count);
// x_rows: the tokens (grouped: the rows of all segments). Dense: after gemm_wp_share.
bool gemm_wp_encode(GemmWp* g, const WeightDev& w, size_t experts, bool grouped, const void* x16, size_t x_rows, int sm_count, void* y, int y_dtype, size_t y_ld,
                    size_t lo_row0 = 0);
cudaError_t launch_gemm_wp(const GemmWp& g, const WeightDev& w, size_t t, const WtTile* tiles, int n_tiles, void* y, int y_dtype, size_t y_ld,
                           GemmStatus* status, const float* row_unscale, cudaStream_t st);

}  // namespace b2
