// Dequant products of one to eight tokens: the role of dmv_* and dmvk_* in the reference (src/cuda_decode.cu:139-232). See
// gemv_mma.cuh for the arithmetic and split.cuh for the activations.
//
// One CTA of 16 warps per SM. K is summed in eight slices (units of one or two blocks in turn, so that neighbouring warps read
// neighbouring bytes; fewer where there are fewer units), a warp each; the two groups of eight warps take tiles of 16 rows of their own.
// Each warp keeps units of packed weights in flight in a ring of shared memory of its own (cp.async), filled before the
// kernel waits for the one ahead of it in the stream. The slices' sums of a few tiles wait in shared memory and are then added, in the
// order of the slices, by all threads of the group. The number of tokens does not change the order of a sum, so every row equals its
// one-token row bit for bit, in a row shard too.
//
// The activations come as f32 vectors and are split by the CTA itself (an RMS norm in front of the product runs in the same pass: the
// weights multiply before the split, the factor multiplies the results), or as records that launch_split made. Where the split vectors
// of all tokens do not fit beside the rings, K is taken in parts and the slices' sums wait in shared memory between them. Records are copied
// asynchronously, all pieces at once (loaded and stored one block and token after the other they were a chain of up to 21 L2 latencies: six
// Q8_0 tokens, 4096 x 14336, 36.1 -> 30.7 us; four tokens through 16 decoder layers 1761 -> 1718).
#pragma once
#include <algorithm>
#include <type_traits>

#include "gemv_mma.cuh"

namespace b2 {

using namespace gmma;

namespace {

constexpr int WARPS = 16, THREADS = WARPS * 32;
constexpr int MAX_TILES = 8;           // most tiles of a group whose sums wait between parts
constexpr size_t SMEM_MAX = 226 * 1024;

__device__ __forceinline__ float silu(float a) { return a / (1.0f + __expf(-a)); }
__device__ __forceinline__ float gelu_tanh(float a) {
    const float t = 0.7978845608f * (a + 0.044715f * a * a * a);
    return 0.5f * a * (1.0f + tanhf(t));
}

struct Args {
    WeightDev w, w2;
    const float* x;        // token i at x + i * x_stride
    size_t x_stride;
    const float* nw;       // norm weights (null: none)
    float pre;
    int norm;              // multiply the results by 1 / sqrt(mean square + eps)
    float eps;
    const uint8_t* rec;    // or token i's record at rec + i * rec_stride
    size_t rec_stride;
    float* y;
    size_t y_stride;
    const float* gate;     // token i's gate at gate + i * gate_stride
    size_t gate_stride;
    int mode, T, fast;
    int units, part_units;  // units of k in all, and in a part
    int blocks, bpu, slice_log, batch, bufs;  // blocks of the format, blocks per unit, log2 of the slices, tiles whose sums are added together, buffers for them
    int hold_tiles;
    uint32_t frag_off, xs_off, ssq_off, sums_off, hold_off, comb_off;  // shared memory
};

struct NoGroups {};

// G: NoGroups, or GemvGroups (a stack of matrices, each times the rows of its groups of up to TP). The tiles of all groups are one list
// then, and every CTA takes a run of it: neighbouring tiles of a group split its activations once, and no CTA waits for a longer one.
template <class F, bool PAIR, int TP, bool PARTS, class G>
__global__ void __launch_bounds__(THREADS, 1) gemv_mma_kernel(const __grid_constant__ Args a, const __grid_constant__ G gt) {
    constexpr bool GROUPED = !std::is_same<G, NoGroups>::value;
    static_assert(!GROUPED || !PARTS);
    extern __shared__ __align__(128) uint8_t smem[];
    using X = typename F::template X<TP>;
    constexpr int ROWS = PAIR ? 8 : 16, S = F::SLOTS, BPX = 256 / F::BLOCK_K, NT = X::NT;  // BPX: blocks of the format per block of the split
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int sl_log = a.slice_log, slices = 1 << sl_log, bpu = a.bpu;
    // (uniform over the warp, and the compiler should know) q: the warp's slice
    const int wq = __shfl_sync(0xffffffffu, warp, 0), group = wq >> sl_log, q = wq & (slices - 1), groups = WARPS >> sl_log;
    const size_t n_out = a.w.n_out;
    const int tiles = (int)((n_out + ROWS - 1) / ROWS);
    // this group of warps: tiles tile0, tile0 + tile_step, ... below tile_end
    int tile0 = group * (int)gridDim.x + (int)blockIdx.x, tile_step = groups * (int)gridDim.x, tile_end = tiles;
    int seg0 = 0, segs = 1;  // the CTA's first group of tokens, how many it has tiles of
    if constexpr (GROUPED) {
        const long long total = (long long)tiles * gt.n;
        const int lo = (int)(total * blockIdx.x / gridDim.x);
        tile_end = (int)(total * (blockIdx.x + 1) / gridDim.x);
        tile0 = lo + group;
        tile_step = groups;
        seg0 = lo / tiles;
        segs = (tile_end - 1) / tiles - seg0 + 1;
    }
    const int my_tiles = tile0 < tile_end ? (tile_end - tile0 + tile_step - 1) / tile_step : 0;
    // unit u, of `bpu` blocks, belongs to slice u % slices (a power of two)
    const int parts = PARTS ? (a.units + a.part_units - 1) / a.part_units : 1;
    auto j_at = [&](int u) { return (u - q + slices - 1) >> sl_log; };  // the slice's units below u
    auto j_beg = [&](int p) { return PARTS ? j_at(p * a.part_units) : 0; };
    auto j_end = [&](int p) { return j_at(PARTS ? min(a.units, (p + 1) * a.part_units) : a.units); };
    const size_t last_row0 = n_out > 8 ? n_out - 8 : 0;
    auto tile_of = [&](int i) { return GROUPED ? (tile0 + i * tile_step) % tiles : tile0 + i * tile_step; };
    auto row_of = [&](int i, int half) { return min((size_t)tile_of(i) * ROWS + (PAIR ? 0 : 8 * half), last_row0); };
    const uint32_t smem0 = (uint32_t)__cvta_generic_to_shared(smem);
    const uint32_t ring = smem0 + (uint32_t)wq * (S * F::UNIT_BYTES), ring_end = ring + S * F::UNIT_BYTES;
    uint32_t islot = ring, slot = ring;

    // the copies run ahead of the arithmetic in the same order: parts, tiles, units
    typename F::template Copy<PAIR> cp;
    cp.init(a.w, bpu, lane);
    int ip = 0, it = 0, ij = 0, ije = j_end(0);
    bool more = my_tiles > 0 && q < a.units;
    auto copy_tile = [&](int i) {
        if constexpr (GROUPED) {
            const size_t at = gt.expert[min((tile0 + i * tile_step) / tiles, gt.n - 1)] * gt.w_stride;
            WeightDev w = a.w, w2 = a.w2;
            w.p0 += at;
            w2.p0 += at;
            cp.tile(w, w2, row_of(i, 0), row_of(i, 1), lane);
        } else {
            cp.tile(a.w, a.w2, row_of(i, 0), row_of(i, 1), lane);
        }
    };
    if (more) copy_tile(0);
    auto next_run = [&] {  // the next tile of a part, part
        if (++it == my_tiles) {
            it = 0;
            ip++;
        }
        copy_tile(it);
        more = ip < parts;
        ij = j_beg(ip);
        ije = j_end(ip);
    };
    if (PARTS)
        while (more && ij >= ije) next_run();
    auto issue = [&] {
        if (more) {
            const int b = (q + (ij << sl_log)) * bpu;
            cp.issue(islot, b, b + 2 > a.blocks, lane);
            islot = islot + F::UNIT_BYTES == ring_end ? ring : islot + F::UNIT_BYTES;
            if (++ij >= ije) do next_run();
                while (more && ij >= ije);
        }
        cp_commit();
    };
#pragma unroll
    for (int s = 0; s < S; s++) issue();
    pdl_wait();

    float* const xs_s = (float*)(smem + a.xs_off);
    float* const ssq_s = (float*)(smem + a.ssq_off);
    float2* const hold = (float2*)(smem + a.hold_off);
    // the slices' sums of `batch` tiles, `bufs` times: [tile][slice][instruction's tokens][row 16][token]
    constexpr int RES = X::RES;
    float* const comb = (float*)(smem + a.comb_off) + (size_t)group * a.bufs * a.batch * slices * RES;
    X xv;
    {
        if constexpr (F::HALVES) {
            const int ct = TP == 1 ? 0 : g >> 1, rt = TP == 1 ? 0 : t;
            xv.frag = smem0 + a.frag_off + (uint32_t)(ct * 128 + (g & 1) * 64 + t * 16);
            xv.xs = smem0 + a.xs_off + 4u * (uint32_t)rt;
            xv.sums = 0;
        } else {
            const int ct = TP == 1 ? 0 : g >> 2, cd = min(g & 3, X::COLUMNS - 1), rt = TP == 1 ? 0 : t >> 1;
            xv.frag = smem0 + a.frag_off + ct * X::TOKEN + (uint32_t)(cd * 64 + t * 16);
            xv.xs = smem0 + a.xs_off + 4u * (uint32_t)rt;
            xv.sums = smem0 + a.sums_off + (F::SUMS_BY_COLUMN ? (uint32_t)(ct * 32 + (g & 3) * 8 + t * 4) : (uint32_t)(rt * 32 + (t & 1) * 8));
        }
    }
    const int xblocks = (a.blocks + BPX - 1) / BPX;  // of the split
    int tile_at = 0;
    for (int p = 0; p < (GROUPED ? segs : parts); p++) {
        const int seg = seg0 + p, row0 = [&] { if constexpr (GROUPED) return (int)gt.row0[seg]; else return 0; }();
        const int T = [&] { if constexpr (GROUPED) return (int)gt.count[seg]; else return a.T; }();
        const int i_end = GROUPED ? min(my_tiles, max(0, ((seg + 1) * tiles - tile0 + tile_step - 1) / tile_step)) : my_tiles;
        const int b0 = PARTS ? p * (a.part_units * bpu / BPX) : 0, nb = PARTS ? min(xblocks, b0 + a.part_units * bpu / BPX) - b0 : xblocks;
        if ((PARTS || GROUPED) && p > 0) __syncthreads();  // every warp is done with the part before
        auto block_of = [&](int i) { return TP == 1 ? i : i / T; };
        auto load = [&](int i) {
            const int b = block_of(i), tk = TP == 1 ? 0 : i - b * T, k = (b0 + b) * 256;
            size_t xr = (size_t)tk;
            if constexpr (GROUPED) xr = gt.gather ? gt.src[row0 + tk] : row0 + tk;
            return split_load(a.x + xr * a.x_stride + k, a.nw ? a.nw + k : nullptr, (int)a.w.n_in - k, lane);
        };
        SplitIn next;
        constexpr bool RECORDS = X::COLUMNS <= 3;  // (there are none of four digits)
        if (!(RECORDS && a.rec) && wq < nb * T) next = load(wq);
        for (int i = RECORDS && a.rec ? nb * T : wq; i < nb * T; i += WARPS) {
            const int b = block_of(i), tk = TP == 1 ? 0 : i - b * T, blk = b0 + b;
            uint8_t* f0 = smem + a.frag_off + (size_t)b * (X::BLOCK * TP) + tk * X::TOKEN;
            int s;
            float xs, ssq;
            {
                const SplitIn in = next;
                if (i + WARPS < nb * T) next = load(i + WARPS);
                if constexpr (F::HALVES) {
                    const SplitHalves d = split_halves(in, a.pre);
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        uint8_t* o = f0 + (size_t)(4 * h + (lane >> 3)) * X::STEP + (lane & 3) * 16 + ((lane >> 2) & 1) * 8;
                        *(uint2*)o = d.hi[h];
                        *(uint2*)(o + 64) = d.lo[h];
                    }
                    xs = d.xs;
                    ssq = d.ssq;
                    s = 0;
                } else {
                    const auto d = split_digits<X::COLUMNS>(in, a.pre, a.fast);
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        int pair, in16;
                        split_digit_at(h, lane, pair, in16);
                        uint8_t* o = f0 + (size_t)pair * X::STEP + in16;
#pragma unroll
                        for (int pl = 0; pl < X::COLUMNS; pl++) *(uint32_t*)(o + 64 * pl) = d.d[h][pl];
                    }
                    xs = d.xs;
                    ssq = d.ssq;
                    const int from = (lane & 3) * 8, sl = __shfl_sync(0xffffffffu, d.s[0], from), sh = __shfl_sync(0xffffffffu, d.s[1], from);
                    s = (lane & 4) ? sh : sl;
                }
            }
            if (lane == 0) {
                xs_s[b * TP + tk] = xs;
                ssq_s[blk * TP + tk] = ssq;
            }
            F::put_sums(smem + a.sums_off + (size_t)(b * TP + tk) * X::SUMS, xs, s, lane);
        }
        // Records: the fragments lie there as they lie here; nobody waits for a copy before all are on their way. (Apart from the other path, whose first
        // run through its code counts: inside its loop, and with divisions by one token, Q5_K 14336 x 4096 took 12.05 us, this way 11.70.)
        if (RECORDS && __builtin_expect(a.rec != nullptr, 0)) {
            for (int i = wq; i < nb * T; i += WARPS) {
                const int b = block_of(i), tk = TP == 1 ? 0 : i - b * T, blk = b0 + b;
                const uint8_t* src = a.rec + (size_t)tk * a.rec_stride + (size_t)blk * X::BLOCK;
                constexpr int PIECES = X::BLOCK / 16, PER = X::TOKEN / 16;  // pieces of 16 bytes
                const uint32_t dst = smem0 + a.frag_off + (uint32_t)(b * (X::BLOCK * TP) + tk * X::TOKEN);
                cp16(dst + (lane / PER) * X::STEP + (lane % PER) * 16, src + lane * 16);
                if (lane + 32 < PIECES) cp16(dst + ((lane + 32) / PER) * X::STEP + ((lane + 32) % PER) * 16, src + (lane + 32) * 16);
            }
            cp_commit();
            // the scales, and the chunk sums of which every lane takes one
            constexpr int LANES = F::SUMS ? 8 : 1;
            for (int e0 = wq * 32; e0 < nb * T * LANES; e0 += THREADS) {
                const int i = (e0 + lane) / LANES, sub = lane % LANES, at = min(i, nb * T - 1), b = at / T, tk = at - b * T, blk = b0 + b;
                const uint8_t* aux = a.rec + (size_t)tk * a.rec_stride + (size_t)xblocks * X::BLOCK + (size_t)blk * SPLIT_AUX;
                const float2 h0 = __ldcg((const float2*)aux);
                const int s = F::SUMS ? __ldcg((const int*)(aux + 16) + sub) : 0;
                if (i < nb * T && sub == 0) {
                    xs_s[b * TP + tk] = h0.x;
                    ssq_s[blk * TP + tk] = h0.y;
                }
                if constexpr (F::SUMS) F::put_sums(smem + a.sums_off + (size_t)(b * TP + tk) * X::SUMS, h0.x, s, i < nb * T ? sub : 8 + sub);
            }
            cp_wait<0>();  // (and with them the weights' first units, which were asked for long before)
        }
        __syncthreads();
        int in_batch = 0, buf = 0, batch0 = GROUPED ? tile_at : 0;
        for (int i = batch0; i < i_end; i++) {
            float* cb = comb + (size_t)(buf * a.batch + in_batch) * slices * RES;
            const uint32_t tag = F::tag(a.w, a.w2, row_of(i, 0), row_of(i, 1), g);
            float acc[NT][2];
            float2* h = PARTS ? hold + (size_t)(wq * a.hold_tiles + i) * NT * 32 + lane : nullptr;
#pragma unroll
            for (int n = 0; n < NT; n++) {
                float2 v = make_float2(0.0f, 0.0f);
                if (PARTS && p > 0) v = h[n * 32];
                acc[n][0] = v.x;
                acc[n][1] = v.y;
            }
            const int b_part = PARTS ? p * a.part_units * bpu : 0, j1 = j_end(p);
            for (int j = j_beg(p); j < j1; j++) {
                cp_wait<S - 1>();
                __syncwarp();
                const int b = (q + (j << sl_log)) * bpu;
                const int bn = min(bpu, a.blocks - b);
                for (int k = 0; k < bn; k++) F::template block<TP>(slot + k * F::BLOCK_BYTES, b + k - b_part, ((b + k) & 1) ? ~tag : tag, a.w, a.w2, xv, g, t, acc);
                __syncwarp();
                issue();  // into the slot just used
                slot = slot + F::UNIT_BYTES == ring_end ? ring : slot + F::UNIT_BYTES;
            }
            if (PARTS && p + 1 < parts) {
#pragma unroll
                for (int n = 0; n < NT; n++) h[n * 32] = make_float2(acc[n][0], acc[n][1]);
            } else {
#pragma unroll
                for (int n = 0; n < NT; n++) {
                    float* cr = cb + q * RES + n * 16 * X::PER;
                    if constexpr (F::HALVES) {
                        if (TP > 1) cr[g * 4 + t] = acc[n][0], cr[(g + 8) * 4 + t] = acc[n][1];
                        else if (t == 0) cr[g] = acc[n][0], cr[g + 8] = acc[n][1];
                    } else {  // a token's two lanes together; one keeps row g, the other row g + 8
                        const float v0 = acc[n][0] + __shfl_xor_sync(0xffffffffu, acc[n][0], 1), v1 = acc[n][1] + __shfl_xor_sync(0xffffffffu, acc[n][1], 1);
                        const float v = (t & 1) ? v1 : v0;
                        const int row = g + 8 * (t & 1);
                        if (TP > 1) cr[row * 2 + (t >> 1)] = v;
                        else if (t < 2) cr[row] = v;
                    }
                }
            }
            if (PARTS && p + 1 < parts) continue;
            if (++in_batch < a.batch && i + 1 < i_end) continue;
            if (slices == 1) __syncwarp();
            else asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(slices * 32) : "memory");
            // one thread per result (per pair of results in the pair form): the sums in the order of the slices
            constexpr int PER = PAIR ? 8 : 16;
            const float* c0 = comb + (size_t)buf * a.batch * slices * RES;
            for (int e = q * 32 + lane; e < in_batch * PER * T; e += slices * 32) {
                const int r = e % PER, et = e / PER, token = et % T, tl = et / T;
                const size_t first = (size_t)tile_of(batch0 + tl) * ROWS + (r & 8), row = row_of(batch0 + tl, r >> 3) + (r & 7);
                if (row < first || row >= n_out) continue;  // (the last tile's halves overlap the rows before them)
                const float* pv = c0 + (size_t)tl * slices * RES + (TP == 1 ? r : token / X::PER * 16 * X::PER + r * X::PER + token % X::PER);
                float v = 0.0f, v2 = 0.0f;
                constexpr int SECOND = 8 * (TP == 1 ? 1 : X::PER);  // (of a pair)
                if (!GROUPED && F::IN_PAIRS && slices == 4) {
                    v = (pv[0] + pv[RES]) + (pv[2 * RES] + pv[3 * RES]);
                    if (PAIR) v2 = (pv[SECOND] + pv[RES + SECOND]) + (pv[2 * RES + SECOND] + pv[3 * RES + SECOND]);
                } else {
                    for (int s = 0; s < slices; s++) {
                        v += pv[s * RES];
                        if (PAIR) v2 += pv[s * RES + SECOND];
                    }
                }
                if (a.norm) {
                    float sq = 0.0f;
                    for (int b = 0; b < xblocks; b++) sq += ssq_s[b * TP + token];
                    const float k = 1.0f / sqrtf(sq / (float)a.w.n_in + a.eps);
                    v *= k;
                    v2 *= k;
                }
                float* o = a.y + (size_t)(row0 + token) * a.y_stride + row;
                if (PAIR) *o = (a.mode == B2_MODE_SILU_PAIR ? silu(v) : gelu_tanh(v)) * v2;
                else if (a.mode == B2_MODE_STORE) *o = v;
                else if (a.mode == B2_MODE_ADD) *o += v;
                else *o += v * (1.0f / (1.0f + __expf(-a.gate[(size_t)token * a.gate_stride])));
            }
            batch0 = i + 1;
            in_batch = 0;
            if (a.bufs == 2) buf ^= 1;
            else if (slices == 1) __syncwarp();
            else asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(slices * 32) : "memory");
        }
        tile_at = i_end;
    }
    cp_wait<0>();
}

template <class F, bool PAIR, int TP>
cudaError_t launch_t(Args& a, int sm_count, cudaStream_t st, bool pdl, const GemvGroups* gt = nullptr) {
    using X = typename F::template X<TP>;
    constexpr int ROWS = PAIR ? 8 : 16, BPX = 256 / F::BLOCK_K, NT = X::NT, RES = X::RES;
    a.blocks = (int)((a.w.n_in + F::BLOCK_K - 1) / F::BLOCK_K);
    // The order of a row's sum depends on K alone (a row shard has other tiles): eight slices, or as many as there are units, of units
    // of two blocks where that leaves a unit per slice.
    a.bpu = a.blocks >= 8 * F::MAX_BLOCKS ? F::MAX_BLOCKS : 1;
    a.units = (a.blocks + a.bpu - 1) / a.bpu;
    a.slice_log = 3;
    while ((1 << a.slice_log) > a.units) a.slice_log--;
    const int slices = 1 << a.slice_log;
    const size_t tiles = (a.w.n_out + ROWS - 1) / ROWS;
    const int groups = WARPS / slices;
    const int span = std::max(slices, BPX), xblocks = (a.blocks + BPX - 1) / BPX;
    // the sums of a few tiles wait for one barrier: 8 KB of them, twice, over all groups
    a.batch = std::max(1, std::min(8, 8192 / (groups * slices * RES * 4)));
    a.bufs = 2;
    const size_t ring = (size_t)WARPS * F::SLOTS * F::UNIT_BYTES;
    size_t comb = (size_t)groups * a.bufs * a.batch * slices * RES * 4;
    size_t grid = std::min(gt ? tiles * gt->n : tiles, (size_t)sm_count);
    const size_t ssq = xblocks * TP * 4, per_block = TP * (X::BLOCK + 4 + X::SUMS), slack = 512;
    size_t fixed = ring + comb + ssq + slack, hold = 0, part = xblocks;
    if (fixed + xblocks * per_block > SMEM_MAX) {
        if (gt || !F::PARTS) return cudaErrorInvalidValue;
        a.batch = a.bufs = 1;  // (a tile's arithmetic is long here: the second barrier costs little and the room holds activations)
        fixed -= comb;
        comb = (size_t)groups * slices * RES * 4;
        fixed += comb;
        // parts of whole rounds of the slices where one fits, else of as many units as fit
        size_t step = (size_t)std::max(1, span * a.bpu / BPX);  // in blocks of the split
        const size_t least = (size_t)std::max(1, a.bpu / BPX), per_tile = (size_t)WARPS * NT * 256;
        if (fixed + per_tile + least * per_block > SMEM_MAX) return cudaErrorInvalidValue;
        // The waiting sums may take the room that a round leaves; a group that has more tiles than that goes in several waves of CTAs.
        const size_t room = SMEM_MAX - fixed - (fixed + per_tile + step * per_block <= SMEM_MAX ? step : least) * per_block;
        const size_t most = std::min<size_t>(MAX_TILES, room / per_tile), wave = (size_t)sm_count * groups;
        const size_t waves = (tiles + wave * most - 1) / (wave * most);
        if (waves > 1) grid = waves * sm_count;
        a.hold_tiles = (int)((tiles + grid * groups - 1) / (grid * groups));
        hold = a.hold_tiles * per_tile;
        part = (SMEM_MAX - fixed - hold) / per_block;
        if (part < step) step = least;
        part = part / step * step;
    }
    const bool parts = part < (size_t)xblocks;
    a.part_units = parts ? (int)part * BPX / a.bpu : a.units;
    size_t at = ring;
    auto take = [&](size_t n) {
        const size_t r = at;
        at += (n + 15) / 16 * 16;
        return (uint32_t)r;
    };
    a.frag_off = take(part * TP * X::BLOCK);
    a.comb_off = take(comb);
    a.hold_off = take(hold);
    a.sums_off = take(part * TP * X::SUMS + 64);
    a.ssq_off = take(ssq);
    a.xs_off = take(part * TP * 4 + 64);
    if constexpr (std::is_same<F, F4<true, false>>::value || std::is_same<F, F4<false, false>>::value) {
        if (gt) {
            auto kern = gemv_mma_kernel<F, PAIR, TP, false, GemvGroups>;
            if (cudaError_t e = ensure_dynamic_smem((const void*)kern, at); e != cudaSuccess) return e;
            return launch_k(kern, dim3((unsigned)grid), dim3(THREADS), at, st, pdl, a, *gt);
        }
    }
    auto kern = gemv_mma_kernel<F, PAIR, TP, false, NoGroups>;
    if constexpr (F::PARTS) {
        if (parts) kern = gemv_mma_kernel<F, PAIR, TP, true, NoGroups>;
    }
    if (cudaError_t e = ensure_dynamic_smem((const void*)kern, at); e != cudaSuccess) return e;
    return launch_k(kern, dim3((unsigned)grid), dim3(THREADS), at, st, pdl, a, NoGroups{});
}

}  // namespace
}  // namespace b2
