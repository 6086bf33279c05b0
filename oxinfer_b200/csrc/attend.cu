// The decode attention: one query per head over the cache (dattn / dattn_combine, src/cuda_decode.cu:396-536), for the one to four
// tokens of a step at once.
//
// A cluster of CTAs takes up to four rows (query heads of one KV head, of one or several of the step's tokens) over all keys. Tile t of
// 64 keys belongs to part t % 16, keys 8 w .. 8 w + 7 of a tile to warp w, so the division depends on the absolute position of a key alone, and a
// row's sums are the same whatever rows stand beside it (keys that it may not see do not enter them). A cluster has 16 CTAs, a part each, while
// no more than 14 of them are wanted, which is what the chip holds at two CTAs an SM (seven at one); otherwise eight, two parts each. Over long caches
// several clusters share a KV head's keys, 1024 at a time in turn (attend_shares); the last to finish adds their sums.
// Every warp runs on its own: a ring of batches of eight keys or values in shared memory (bulk copies, started before the kernel waits for the one
// ahead: those rows were written by earlier steps), a running softmax, and no CTA barrier between batches. The warps' sums are added in
// shared memory, every CTA stores them into the CTAs of the cluster, a share of the outputs to each, and those add them, in a fixed order.
//
// What bounds it: latency. A launch over an empty cache takes half of its time at 2048 keys: the step words, the factors and the
// heads' values one behind the other, the two barriers of the cluster. At 2048 f32 keys of 8 heads of 128 a layer's caches take 2.6 us at the HBM rate.
// Chained behind launches of a whole SM each, 32 query heads, one token, context 16 / 500 / 2048 / 8000: 5.1 / 6.0 / 10.2 / 18.6 us a launch; four
// tokens 9.8 / 10.7 / 20.0 / 49. The form before, a CTA per 64 keys, partial sums through global memory and a last CTA that added
// them behind a fence and a counter: 8.7 / 9.6 / 13.5 / 29.0, and four tokens, each over the caches for itself, 9.6 / 12.0 / 25.1 / 57.4 beside
// a launch that turned and appended. Sixteen rows a warp: 17 us over an empty cache. cp.async by the lanes instead of bulk copies, queries
// in registers: 5.6 / 6.6 / 10.4 / 20.0.
#include <cuda_fp16.h>

#include <algorithm>

#include "async_copy.cuh"
#include "kernels.h"
#include "pdl.cuh"

namespace b2 {

using namespace acopy;

namespace {

constexpr int ATT_WARPS = 8, ATT_THREADS = ATT_WARPS * 32;
constexpr int ATT_BATCH = 8;                        // keys a warp takes at a time: eight lanes take two of them
constexpr int ATT_TILE = ATT_WARPS * ATT_BATCH;     // keys
constexpr int ATT_MOST_ROWS = 4;
constexpr int ATT_PARTS = 16;                       // of the keys
constexpr int ATT_SPAN = ATT_PARTS * ATT_TILE;      // keys: a tile of every part
constexpr int ATT_MOST_SHARES = 16;

template <int HD, int R, typename T>
struct AttShared {  // bytes
    static constexpr uint32_t SLOT = ATT_BATCH * HD * sizeof(T);                              // the keys or the values of a batch
    static constexpr int SLOTS = 12 * 1024 / SLOT < 8 ? 12 * 1024 / SLOT : 8;                 // of a warp: 96 KB a CTA, and two CTAs fit an SM
    static constexpr uint32_t RING = SLOTS * SLOT, F4 = R * HD / 4;                           // (outputs by fours)
    static constexpr uint32_t Q = ATT_WARPS * RING, P = Q + R * HD * 4, M = P + ATT_WARPS * (ATT_BATCH + 1) * 16, X = M + 2 * R * ATT_WARPS * 4,
                              XM = X + F4 * ATT_PARTS / 8 * 16, XL = XM + F4 * ATT_PARTS / 8 * 4, OWN = XL + F4 * ATT_PARTS / 8 * 4,
                              BARS = OWN + ATT_STEP_TOKENS * 2 * HD * (uint32_t)sizeof(T), BYTES = BARS + ATT_WARPS * SLOTS * 8 + 8;
    static_assert(BYTES + 1024 <= 228 * 1024 / 2);
    static_assert(RING >= R * HD * 4, "a warp's sums take its ring's place");
};

// (a.x b.x + c.x, a.y b.y + c.y), each rounded as fmaf rounds it: one instruction for two.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\tfma.rn.f32x2 a, a, b, c;\n\tmov.b64 {%0, %1}, a;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}

// Two keys' products with R queries (in shared memory) over a lane's HD / 8 dimensions, the even and the odd ones' sums apart.
template <int HD, int R>
__device__ __forceinline__ void score(float2 (&a)[R], float2 (&b)[R], const float* ka, const float* kb, const float* qs, int l8) {
#pragma unroll
    for (int i = 0; i < HD / 32; i++) {
        const int d = l8 * 4 + 32 * i;
        const float4 x = *(const float4*)(ka + d), y = *(const float4*)(kb + d);
#pragma unroll
        for (int r = 0; r < R; r++) {
            const float4 q = *(const float4*)(qs + r * HD + d);
            a[r] = fma2(make_float2(x.x, x.y), make_float2(q.x, q.y), a[r]);
            b[r] = fma2(make_float2(y.x, y.y), make_float2(q.x, q.y), b[r]);
            a[r] = fma2(make_float2(x.z, x.w), make_float2(q.z, q.w), a[r]);
            b[r] = fma2(make_float2(y.z, y.w), make_float2(q.z, q.w), b[r]);
        }
    }
}
template <int HD, int R>
__device__ __forceinline__ void score(float2 (&a)[R], float2 (&b)[R], const __half* ka, const __half* kb, const float* qs, int l8) {
#pragma unroll
    for (int i = 0; i < HD / 64; i++) {
        const int d = l8 * 8 + 64 * i;
        const uint4 u = *(const uint4*)(ka + d), v = *(const uint4*)(kb + d);
        const uint32_t uw[4] = {u.x, u.y, u.z, u.w}, vw[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const float2 x0 = __half22float2(*(const __half2*)&uw[2 * h]), x1 = __half22float2(*(const __half2*)&uw[2 * h + 1]);
            const float2 y0 = __half22float2(*(const __half2*)&vw[2 * h]), y1 = __half22float2(*(const __half2*)&vw[2 * h + 1]);
#pragma unroll
            for (int r = 0; r < R; r++) {
                const float4 q = *(const float4*)(qs + r * HD + 64 * i + 32 * h + 4 * l8);  // (q_at)
                a[r] = fma2(x0, make_float2(q.x, q.y), a[r]);
                b[r] = fma2(y0, make_float2(q.x, q.y), b[r]);
                a[r] = fma2(x1, make_float2(q.z, q.w), a[r]);
                b[r] = fma2(y1, make_float2(q.z, q.w), b[r]);
            }
        }
    }
}

// Where the queries' dimension d lies in shared memory: eight lanes' quads side by side as they read them. (f16 keys come eight dimensions a lane; with the
// queries in order two lanes met in a bank: 32 heads of 8 KV heads of 128, one / four tokens, 8200 keys 22.0 / 38.9 us, this way 18.3 / 36.6, 16000
// keys 37.3 / 72.7 and 31.8 / 61.1.)
template <typename T>
__device__ __forceinline__ uint32_t q_at(uint32_t d) { return sizeof(T) == 2 ? (d & ~63u) + 32 * ((d >> 2) & 1) + 4 * ((d >> 3) & 7) + (d & 3) : d; }

template <int V>
__device__ __forceinline__ void load_values(float (&v)[V], const float* p) {
    if constexpr (V == 4) {
        const float4 a = *(const float4*)p;
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
    } else {
        const float2 a = *(const float2*)p;
        v[0] = a.x, v[1] = a.y;
    }
}
template <int V>
__device__ __forceinline__ void load_values(float (&v)[V], const __half* p) {
    uint32_t w[V / 2];
    if constexpr (V == 4) {
        const uint2 a = *(const uint2*)p;
        w[0] = a.x, w[1] = a.y;
    } else {
        w[0] = *(const uint32_t*)p;
    }
#pragma unroll
    for (int j = 0; j < V / 2; j++) {
        const float2 f = __half22float2(*(const __half2*)&w[j]);
        v[2 * j] = f.x, v[2 * j + 1] = f.y;
    }
}

// The sum over eight lanes of each of R values, one of them left to a lane: s[row_of(l8)] to lane l8. The pairs that are added are the same for every R.
template <int R>
__device__ __forceinline__ float reduce8(float (&s)[R], int l8) {
    if constexpr (R == 4) {
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const float keep = (l8 & 1) ? s[2 + i] : s[i], give = (l8 & 1) ? s[i] : s[2 + i];
            s[i] = keep + __shfl_xor_sync(0xffffffffu, give, 1);
        }
        const float keep = (l8 & 2) ? s[1] : s[0], give = (l8 & 2) ? s[0] : s[1];
        s[0] = keep + __shfl_xor_sync(0xffffffffu, give, 2);
    } else if constexpr (R == 2) {
        const float keep = (l8 & 1) ? s[1] : s[0], give = (l8 & 1) ? s[0] : s[1];
        s[0] = keep + __shfl_xor_sync(0xffffffffu, give, 1);
        s[0] += __shfl_xor_sync(0xffffffffu, s[0], 2);
    } else {
        s[0] += __shfl_xor_sync(0xffffffffu, s[0], 1);
        s[0] += __shfl_xor_sync(0xffffffffu, s[0], 2);
    }
    return s[0] + __shfl_xor_sync(0xffffffffu, s[0], 4);
}
template <int R>
__device__ __forceinline__ int row_of(int l8) { return R == 4 ? 2 * (l8 & 1) + ((l8 >> 1) & 1) : R == 2 ? l8 & 1 : 0; }

__device__ __forceinline__ uint32_t peer_addr(const void* p, uint32_t cta) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr(p)), "r"(cta));
    return r;
}
// Into another CTA's shared memory, counted on its barrier: data and signal in one. (A cluster barrier with release semantics behind plain
// stores took 1500 cycles.)
__device__ __forceinline__ void peer_store(uint32_t a, float4 v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(a), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(bar) : "memory");
}
__device__ __forceinline__ void peer_store(uint32_t a, float v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(a), "f"(v), "r"(bar) : "memory");
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// 2^(m - most), 0 where there was nothing (m = -inf)
__device__ __forceinline__ float weight_of(float m, float most) { return exp2f(m - (most == -INFINITY ? 0.0f : most)); }
__device__ __forceinline__ float shfl_x(float v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }

// Two dimensions of a head that RoPE turns together (or, behind the rotated ones, leaves): the arithmetic of rope_head, attend_core.cuh.
// The factors are known before the kernel ahead ends, the head's values after it.
struct Turn {
    float c, s;
    uint32_t a, b;
    bool on;
    __device__ __forceinline__ Turn(uint32_t j, const float* cs, const DecRope& r) {
        on = j < r.half_rot;
        a = on && !r.interleaved ? j : 2 * j;
        b = on && !r.interleaved ? j + r.half_rot : 2 * j + 1;
        c = on ? cs[j] : 1.0f;
        s = on ? cs[r.half_rot + j] : 0.0f;
    }
    __device__ __forceinline__ float2 of(float x, float y) const {
        return on ? make_float2(__fsub_rn(__fmul_rn(x, c), __fmul_rn(y, s)), __fadd_rn(__fmul_rn(y, c), __fmul_rn(x, s))) : make_float2(x, y);
    }
};

// Clusters that share a KV head's keys: 1 << log of them, span j of the keys to cluster j % shares.
struct AttShares {
    int log;
    uint32_t groups, groups_inv;  // ceil(2^16 / groups)
    float4* part;      // [unit][share][4 outputs]{sums, {largest score, denominator, -, -}}
    uint32_t* counts;  // [unit][CTA], zero
};

// Grid (C, KV heads, shares x groups of R rows), a cluster along x. Row r of a KV head: query head r % G of token r / G. sp[0]: the position of the
// step's first token.
template <int HD, int R, typename T, bool SHARED>
__global__ void __launch_bounds__(ATT_THREADS, 2) attend_kernel(const float* __restrict__ q, T* kc, T* vc, float* __restrict__ out,
                                                                const uint32_t* __restrict__ sp, DecAttn p, uint32_t* status, FusedRope fr, AttnTokens at,
                                                                int g_log, AttShares sh) {
    using L = AttShared<HD, R, T>;
    constexpr int V = HD / 32, S = L::SLOTS;
    extern __shared__ __align__(128) uint8_t smem[];
    pdl_launch_dependents();
    const uint32_t pos0 = sp[0], table0 = sp[1];
    const uint32_t C = gridDim.x, c = blockIdx.x, kvh = blockIdx.y, my_share = SHARED ? blockIdx.z * sh.groups_inv >> 16 : 0, group = blockIdx.z - my_share * sh.groups, row0 = group * R;
    const uint32_t all = (uint32_t)max(1, at.n) << g_log, g_mask = (1u << g_log) - 1;
    const uint32_t tok_a = row0 >> g_log, tok_z = (min(row0 + R, all) - 1) >> g_log;  // the group's tokens
    const uint32_t len = min(pos0 + tok_z + 1, p.max_len);                            // keys below len are seen by some row
    const uint32_t lo = p.window != 0 && pos0 + tok_a + 1 > p.window ? pos0 + tok_a + 1 - p.window : 0;
    const uint32_t span0 = lo / ATT_SPAN, shares_mask = SHARED ? (1u << sh.log) - 1 : 0;
    __shared__ uint32_t active_s[1];  // shares that have keys
    if constexpr (SHARED) {
        const uint32_t spans = (len - 1) / ATT_SPAN + 1 - span0;
        if (((my_share - span0) & shares_mask) >= spans) return;
        if (threadIdx.x == 0) *active_s = min(spans, shares_mask + 1);
    }
    constexpr int F4_LOG = L::F4 == 16 ? 4 : L::F4 == 32 ? 5 : L::F4 == 64 ? 6 : 7;
    static_assert(L::F4 == 1u << F4_LOG);
    const uint32_t share_log = F4_LOG - (gridDim.x == 16 ? 4 : 3), share = 1u << share_log;  // of the outputs
    uint64_t* const all_in = (uint64_t*)(smem + L::BARS) + ATT_WARPS * S;  // the parts' sums have come
    if (threadIdx.x == 0) {
        bar_init(all_in, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        bar_expect_tx(all_in, share * ATT_PARTS * 24);
    }
    __syncwarp();
    cluster_arrive();  // (the CTAs store into one another's shared memory: all of them have to be there)
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, l8 = lane & 7;
    uint8_t* const ring = smem + warp * L::RING;
    float* const qs = (float*)(smem + L::Q);                                // [R][HD]
    float* const pw = (float*)(smem + L::P) + warp * (ATT_BATCH + 1) * 4;   // the warp's probabilities [key][4], and what its sums shrink by
    float* const wm = (float*)(smem + L::M);                                // the warps' largest scores and denominators [R][warp]
    float* const wl = wm + R * ATT_WARPS;
    float4* const xo = (float4*)(smem + L::X);                              // the parts' sums of this CTA's share: [share][part]
    float* const xm = (float*)(smem + L::XM);
    float* const xl = (float*)(smem + L::XL);
    T* const own = (T*)(smem + L::OWN);                                     // the step's own keys and values [token][k | v][HD]
    uint64_t* const bars = (uint64_t*)(smem + L::BARS) + warp * S;

    const bool fused = fr.qkv != nullptr;
    const float q_scale = p.scale * 1.44269504f;  // scores in powers of two
    const uint32_t first_pos = pos0 + tok_a, last_pos = pos0 + tok_z;
    const uint32_t lo_all = p.window != 0 && last_pos + 1 > p.window ? last_pos + 1 - p.window : 0;  // keys from here to first_pos are seen by every row
    const uint32_t t_beg = lo / ATT_TILE;
    const uint32_t w_key = (tid >> 5) * ATT_BATCH, t_end = len > w_key ? (len - w_key + ATT_TILE - 1) / ATT_TILE : 0;  // (this warp's tiles end there)
    const uint32_t copied = fused ? min(len, pos0) : len;  // rows that come from the caches
    // A warp's batches: those of part c, then (eight CTAs) of part c + 8. A part's first tile of this share at or above t_beg, and from one to the next:
    auto first_of = [&](uint32_t part) {
        if constexpr (!SHARED) return t_beg + ((part - t_beg) & (ATT_PARTS - 1));
        const uint32_t span = (t_beg + ATT_PARTS - 1 - part) / ATT_PARTS;
        return (span + ((my_share - span) & shares_mask)) * ATT_PARTS + part;
    };
    const uint32_t t_step = SHARED ? ATT_PARTS << sh.log : ATT_PARTS;
    // copies run ahead: the batch at tile `it` of the part, its keys or its values next (one lane)
    uint32_t it = first_of(c), in_flight = 0, is = 0;
    bool iv = false;
    const T* const k_head = kc + (size_t)kvh * p.max_len * HD;
    const T* const v_head = vc + (size_t)kvh * p.max_len * HD;
    auto issue = [&] {
        const uint32_t key = it * ATT_TILE + w_key, bytes = key < copied ? min((uint32_t)ATT_BATCH, copied - key) * HD * (uint32_t)sizeof(T) : 0u;
        bar_expect_tx(&bars[is], bytes);  // with no bytes to wait for this alone completes the phase
        if (bytes) bulk_load(ring + is * L::SLOT, (iv ? v_head : k_head) + (size_t)key * HD, bytes, &bars[is]);
        is = is + 1 == S ? 0 : is + 1;
        in_flight++;
        if (iv) it += t_step;
        iv = !iv;
    };
    if (lane == 0) {
        for (int s = 0; s < S; s++) bar_init(&bars[s], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        // Rows of earlier steps do not wait for the kernel ahead; the step's own come from it. (The first keys only: the copies would hold
        // up the loads below by 2000 cycles.)
        if (it < t_end && (fused || it * ATT_TILE + w_key + ATT_BATCH <= pos0)) issue();
    }
    if (fused) {
        constexpr uint32_t PAIRS = HD / 2;
        static_assert(ATT_THREADS / PAIRS >= R);
        const uint32_t j = tid % PAIRS, r = tid / PAIRS, ra = min(row0 + r, all - 1), tok = ra >> g_log;
        const float* cs = fr.cs_table + (size_t)(pos0 - table0) * fr.r.cs_stride + fr.r.cs_off;
        const Turn turn(j, cs + tok * fr.r.cs_stride, fr.r);
        pdl_wait();
        const float* const at_q = fr.qkv + tok * at.act_stride + ((kvh << g_log) + (ra & g_mask)) * fr.r.q_stride;
        const float x = __ldcg(at_q + turn.a), y = __ldcg(at_q + turn.b);
        if (lane == 0)
            while (in_flight < S && it < t_end) issue();
        if (r < R) {
            const float2 v = turn.of(x, y);
            qs[r * HD + q_at<T>(turn.a)] = v.x * q_scale;
            qs[r * HD + q_at<T>(turn.b)] = v.y * q_scale;
        }
        // The step's own keys and values up to the group's last token: turned, appended to the caches and kept for the warp that
        // takes them, all by the CTA that has their tile.
        for (uint32_t i = tid; i < 2 * PAIRS * (tok_z + 1); i += ATT_THREADS) {
            const uint32_t t = i / (2 * PAIRS), e = i % (2 * PAIRS), jj = e % PAIRS, pos = pos0 + t;
            if (pos >= len || ((pos / ATT_TILE) & (C - 1)) != c || (SHARED && ((pos / ATT_SPAN) & shares_mask) != my_share)) continue;
            const float* base = fr.qkv + t * at.act_stride;
            const size_t row = ((size_t)kvh * p.max_len + pos) * HD;
            if (e < PAIRS) {
                const Turn k(jj, cs + t * fr.r.cs_stride, fr.r);
                const float* const at_k = base + fr.r.k_off + (size_t)kvh * HD;
                const float2 v = k.of(__ldcg(at_k + k.a), __ldcg(at_k + k.b));
                kc[row + k.a] = own[t * 2 * HD + k.a] = (T)v.x;
                kc[row + k.b] = own[t * 2 * HD + k.b] = (T)v.y;
            } else {
                const float* v = base + fr.r.v_off + (size_t)kvh * HD + 2 * jj;
                vc[row + 2 * jj] = own[t * 2 * HD + HD + 2 * jj] = (T)__ldcg(v);
                vc[row + 2 * jj + 1] = own[t * 2 * HD + HD + 2 * jj + 1] = (T)__ldcg(v + 1);
            }
        }
    } else {
        pdl_wait();
        if (lane == 0)
            while (in_flight < S && it < t_end) issue();
        for (uint32_t i = tid; i < R * HD; i += ATT_THREADS) {
            const uint32_t r = min(row0 + i / HD, all - 1);
            qs[i / HD * HD + q_at<T>(i % HD)] = __ldcg(q + (r >> g_log) * at.act_stride + (size_t)((kvh << g_log) + (r & g_mask)) * HD + i % HD) * q_scale;
        }
    }
    __syncthreads();

    const int my_row = row_of<R>(l8);
    const uint32_t my_pos = pos0 + (min(row0 + my_row, all - 1) >> g_log);  // the position of the row whose scores this lane keeps
    bool ok = true;
    uint32_t s = 0, phase = 0;  // the slot that is next, and its barrier's parity
    auto arrived = [&] {
        ok = ok && __all_sync(0xffffffffu, bar_wait(&bars[s], phase));
        return ok;
    };
    auto next_slot = [&] {  // the slot has been read by the whole warp
        __syncwarp();
        if (lane == 0) {
            in_flight--;
            if (it < t_end) issue();
        }
        if (++s == S) {
            s = 0;
            phase ^= 1;
        }
    };
    for (uint32_t part = c; part < ATT_PARTS; part += C) {
        float2 o[R][V / 2];
        float m = -INFINITY, l = 0.0f;
#pragma unroll
        for (int r = 0; r < R; r++)
#pragma unroll
            for (int i = 0; i < V / 2; i++) o[r][i] = make_float2(0.0f, 0.0f);
        for (uint32_t t = first_of(part); t < t_end && ok; t += t_step) {
            const uint32_t key0 = t * ATT_TILE + w_key;
            // some of the batch's rows are the step's own
            auto put_own = [&](T* slot, int which) {
                if (!fused || key0 + ATT_BATCH <= pos0) return;
                for (uint32_t pos = max(key0, pos0); pos < min(key0 + ATT_BATCH, len); pos++)
#pragma unroll
                    for (int d = lane; d < HD; d += 32) slot[(pos - key0) * HD + d] = own[(2 * (pos - pos0) + which) * HD + d];
                __syncwarp();
            };
            if (!arrived()) break;
            T* const Ks = (T*)(ring + s * L::SLOT);
            put_own(Ks, 0);
            float a[R], b[R];
            {
                float2 a2[R], b2[R];
#pragma unroll
                for (int r = 0; r < R; r++) a2[r] = b2[r] = make_float2(0.0f, 0.0f);
                score<HD, R>(a2, b2, Ks + (lane >> 3) * HD, Ks + (4 + (lane >> 3)) * HD, qs, l8);
#pragma unroll
                for (int r = 0; r < R; r++) {
                    a[r] = a2[r].x + a2[r].y;
                    b[r] = b2[r].x + b2[r].y;
                }
            }
            next_slot();
            const float sa = reduce8<R>(a, l8), sb = reduce8<R>(b, l8);
            const uint32_t ka = key0 + (lane >> 3), kb = ka + 4;
            const bool see_a = ka <= my_pos && ka < len && (p.window == 0 || my_pos - ka < p.window);
            const bool see_b = kb <= my_pos && kb < len && (p.window == 0 || my_pos - kb < p.window);
            float mx = fmaxf(see_a ? sa : -INFINITY, see_b ? sb : -INFINITY);
            mx = fmaxf(mx, shfl_x(mx, 8));
            mx = fmaxf(mx, shfl_x(mx, 16));
            const float mn = fmaxf(m, mx), base = mn == -INFINITY ? 0.0f : mn;
            const float pa = see_a ? exp2f(sa - base) : 0.0f, pb = see_b ? exp2f(sb - base) : 0.0f, al = exp2f(m - base);
            const bool shrink = __any_sync(0xffffffffu, mn > m);
            m = mn;
            l = fmaf(l, al, pa + pb);
            pw[(lane >> 3) * 4 + my_row] = pa;
            pw[((lane >> 3) + 4) * 4 + my_row] = pb;
            if (lane < 8) pw[ATT_BATCH * 4 + my_row] = al;
            if (!arrived()) break;
            T* const Vs = (T*)(ring + s * L::SLOT);
            put_own(Vs, 1);
            __syncwarp();
            if (shrink) {
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const float k = pw[ATT_BATCH * 4 + r];
#pragma unroll
                    for (int e = 0; e < V / 2; e++) o[r][e] = make_float2(o[r][e].x * k, o[r][e].y * k);
                }
            }
            if (key0 + ATT_BATCH <= first_pos + 1 && key0 >= lo_all) {  // every row sees every key
#pragma unroll
                for (int kk = 0; kk < ATT_BATCH; kk++) {
                    float v[V];
                    load_values<V>(v, Vs + kk * HD + lane * V);
                    const float4 pr = *(const float4*)(pw + kk * 4);
                    const float e[4] = {pr.x, pr.y, pr.z, pr.w};
#pragma unroll
                    for (int r = 0; r < R; r++)
#pragma unroll
                        for (int d = 0; d < V / 2; d++) o[r][d] = fma2(make_float2(e[r], e[r]), make_float2(v[2 * d], v[2 * d + 1]), o[r][d]);
                }
            } else {
                const int nk = (int)min((uint32_t)ATT_BATCH, len - key0);
#pragma unroll 1
                for (int kk = 0; kk < nk; kk++) {
                    float v[V];
                    load_values<V>(v, Vs + kk * HD + lane * V);
#pragma unroll
                    for (int r = 0; r < R; r++) {
                        const float e = pw[kk * 4 + r];
                        if (e != 0.0f) {  // (what a row may not see never enters its sums, an infinity neither)
#pragma unroll
                            for (int d = 0; d < V / 2; d++) o[r][d] = fma2(make_float2(e, e), make_float2(v[2 * d], v[2 * d + 1]), o[r][d]);
                        }
                    }
                }
            }
            next_slot();
        }
        // the warps' sums, in their rings (no copy is in flight here, unless one gave up)
        l += shfl_x(l, 8);
        l += shfl_x(l, 16);
        if (lane < 8) {
            wm[my_row * ATT_WARPS + warp] = m;
            wl[my_row * ATT_WARPS + warp] = l;
        }
#pragma unroll
        for (int r = 0; r < R; r++) {
            float* dst = (float*)ring + r * HD + lane * V;
            if constexpr (V == 4) *(float4*)dst = make_float4(o[r][0].x, o[r][0].y, o[r][1].x, o[r][1].y);
            else *(float2*)dst = o[r][0];
        }
        if (part == c) cluster_wait();
        __syncthreads();
        // two threads per four outputs, four warps' sums each; then to the CTA whose share they are
        if (tid < 2 * L::F4) {
            const uint32_t item = tid >> 1, r = item / (HD / 4);
            const float4 m0 = *(const float4*)(wm + r * ATT_WARPS), m1 = *(const float4*)(wm + r * ATT_WARPS + 4);
            const float M = fmaxf(fmaxf(fmaxf(m0.x, m0.y), fmaxf(m0.z, m0.w)), fmaxf(fmaxf(m1.x, m1.y), fmaxf(m1.z, m1.w)));
            const float4 mm = (tid & 1) ? m1 : m0;
            const float w[4] = {weight_of(mm.x, M), weight_of(mm.y, M), weight_of(mm.z, M), weight_of(mm.w, M)};
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
            float den = 0.0f;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int wi = 4 * (tid & 1) + k;
                const float4 b = ((const float4*)(smem + wi * L::RING))[item];
                a.x = fmaf(w[k], b.x, a.x);
                a.y = fmaf(w[k], b.y, a.y);
                a.z = fmaf(w[k], b.z, a.z);
                a.w = fmaf(w[k], b.w, a.w);
                den = fmaf(w[k], wl[r * ATT_WARPS + wi], den);
            }
            a.x += shfl_x(a.x, 1);
            a.y += shfl_x(a.y, 1);
            a.z += shfl_x(a.z, 1);
            a.w += shfl_x(a.w, 1);
            den += shfl_x(den, 1);
            const uint32_t to = item >> share_log, slot = (item & (share - 1)) * ATT_PARTS + part;
            if (tid & 1) {
                peer_store(peer_addr(xm + slot, to), M, peer_addr(all_in, to));
                peer_store(peer_addr(xl + slot, to), den, peer_addr(all_in, to));
            } else {
                peer_store(peer_addr(xo + slot, to), a, peer_addr(all_in, to));
            }
        }
        if (part + C < ATT_PARTS) {
            __syncthreads();  // the rings are free again
            it = first_of(part + C);
            if (lane == 0) {
                fence_proxy_async();
                while (ok && in_flight < S && it < t_end) issue();
            }
        }
    }
    if (!ok && lane == 0) {
        // A copy did not arrive in time: record it, and give the copies in flight one more bounded wait each so that nothing lands in shared
        // memory that has been handed on. (The barriers have been kept: the other warps and CTAs wait there.)
        atomicExch(status, 1u);
        for (; in_flight > 0; in_flight--) {
            bar_wait(&bars[s], phase);
            if (++s == S) {
                s = 0;
                phase ^= 1;
            }
        }
    }
    __syncwarp();
    auto store = [&](uint32_t item, float4 a, float den) {
        const uint32_t r = row0 + item / (HD / 4);
        const float inv = 1.0f / den;
        if (r < all)
            *(float4*)(out + (r >> g_log) * at.act_stride + (size_t)((kvh << g_log) + (r & g_mask)) * HD + item % (HD / 4) * 4) = make_float4(a.x * inv, a.y * inv, a.z * inv, a.w * inv);
    };
    // Every CTA waits for all that is meant for it, so none ends before its peers have stored.
    if (!bar_wait<true>(all_in, 0)) atomicExch(status, 1u);
    // sixteen lanes per four outputs, one for each part's sums
    const uint32_t unit = kvh * sh.groups + group, active = SHARED ? *active_s : 1;
    if (tid < (int)(share * ATT_PARTS + 31) / 32 * 32) {  // (whole warps; the last half of one may read past its share, and stores nothing)
        float4 a = xo[tid];
        float M = xm[tid], den = xl[tid];
        const float m = M;
#pragma unroll
        for (int k = 1; k < ATT_PARTS; k *= 2) M = fmaxf(M, shfl_x(M, k));
        const float w = weight_of(m, M);
        a = make_float4(w * a.x, w * a.y, w * a.z, w * a.w);
        den *= w;
#pragma unroll
        for (int k = 1; k < ATT_PARTS; k *= 2) {
            a.x += shfl_x(a.x, k);
            a.y += shfl_x(a.y, k);
            a.z += shfl_x(a.z, k);
            a.w += shfl_x(a.w, k);
            den += shfl_x(den, k);
        }
        const uint32_t item = (c << share_log) + tid / ATT_PARTS;
        if (tid % ATT_PARTS == 0 && tid < (int)share * ATT_PARTS) {
            if (active == 1) {
                store(item, a, den);
            } else {
                float4* const to = sh.part + (((size_t)unit << sh.log) + my_share) * (2 * L::F4) + 2 * item;
                to[0] = a;
                to[1] = make_float4(M, den, 0.0f, 0.0f);
            }
        }
    }
    if constexpr (!SHARED) return;
    if (active == 1) return;
    // The last of the shares' CTAs that have these outputs adds them, a lane for each share.
    __shared__ uint32_t others;
    __threadfence();
    __syncthreads();
    if (tid == 0) others = atomicAdd(sh.counts + unit * ATT_PARTS + c, 1u);
    __syncthreads();
    if (others != active - 1) return;
    __threadfence();
    if (tid == 0) sh.counts[unit * ATT_PARTS + c] = 0;  // (for the next launch)
    if (tid < (int)(share * ATT_PARTS + 31) / 32 * 32) {
        const uint32_t item = (c << share_log) + min((uint32_t)tid / ATT_PARTS, share - 1), k = tid % ATT_PARTS;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), ml = make_float4(-INFINITY, 0.f, 0.f, 0.f);
        if (k <= shares_mask && ((k - span0) & shares_mask) < active) {
            const float4* const from = sh.part + (((size_t)unit << sh.log) + k) * (2 * L::F4) + 2 * item;
            a = __ldcg(from);
            ml = __ldcg(from + 1);
        }
        float M = ml.x;
#pragma unroll
        for (int o = 1; o < ATT_MOST_SHARES; o *= 2) M = fmaxf(M, shfl_x(M, o));
        const float w = weight_of(ml.x, M);
        a = make_float4(w * a.x, w * a.y, w * a.z, w * a.w);
        float den = ml.y * w;
#pragma unroll
        for (int o = 1; o < ATT_MOST_SHARES; o *= 2) {
            a.x += shfl_x(a.x, o);
            a.y += shfl_x(a.y, o);
            a.z += shfl_x(a.z, o);
            a.w += shfl_x(a.w, o);
            den += shfl_x(den, o);
        }
        if (k == 0 && tid < (int)share * ATT_PARTS) store(item, a, den);
    }
}

// How many clusters share a KV head's keys: by heads and the caches' size alone, since a token's sums have to be the same in steps of one and of several
// tokens. More of them only where that puts more CTAs to work on one token, and
// - while the clusters of a step of four tokens still run at once (one for each head and share, some 36 of eight CTAs fit the chip), from 3072 keys
//   a share on, where the exchange through memory (2 us) is made up for; 1536 where one token's clusters already have eight CTAs. f32 caches of 128
//   dimensions, 12300 keys, one and four tokens, us a launch without and with: 4 heads of 1 KV head 17.6 / 19.1 and 9.7 / 17.9, 16 of 4 19.3 / 46.2
//   and 16.5 / 31.4, 16 of 16 of 64 dimensions, 4100 keys, 18.6 / 18.0 and 12.9 / 14.0;
// - or else from 16384 keys on, where one to three tokens gain more than four lose (two waves of clusters). 32 heads of 8 KV heads, one, two, three
//   and four tokens: f32, 24600 keys 42 / 86 / 88 / 88 and 35 / 63 / 84 / 111, 32000 keys 58 / 112 / 111 / 112 and 47 / 69 / 101 / 135, of 64
//   dimensions 42 / 82 / 82 / 82 and 29 / 54 / 77 / 102; f16, 24600 keys, one and four 45.6 / 91.0 and 33.6 / 109.4. (12300 keys 28.0 / 48.8, f16
//   28.1 / 49.7 without.)
uint32_t attend_shares(uint32_t nh, uint32_t nkv, uint32_t max_len) {
    const uint32_t units = nkv * ((nh / nkv + ATT_MOST_ROWS - 1) / ATT_MOST_ROWS);  // clusters of one token
    auto ctas = [&](uint32_t s) { return units * s * (units * s > 14 ? 8 : 16); };
    uint32_t shares = 1;
    for (uint32_t s = 2; s <= ATT_MOST_SHARES && nh * s <= 32 && max_len >= (units > 14 ? 1536 : 3072) * s; s *= 2)
        if (ctas(s) > ctas(shares)) shares = s;
    for (uint32_t s = 2; shares == 1 && s <= ATT_MOST_SHARES && units * s <= 32 && max_len >= 16384; s *= 2)
        if (ctas(s) > ctas(1)) shares = s;
    return shares;
}

template <int HD, int R, typename T>
cudaError_t attend_t(const float* q, void* kc, void* vc, float* out, const uint32_t* sp, const DecAttn& p, uint32_t* status, cudaStream_t st, bool pdl,
                     const FusedRope& fr, const AttnTokens& at, const AttScratch& scratch) {
    constexpr size_t smem = AttShared<HD, R, T>::BYTES;
    auto kern = attend_kernel<HD, R, T, false>;
    const unsigned G = p.nh / p.nkv, groups = (G * (unsigned)std::max(1, at.n) + R - 1) / R, shares = attend_shares(p.nh, p.nkv, p.max_len);
    const unsigned C = p.nkv * groups * shares > 14 ? 8 : 16;
    AttShares sh{};
    while ((1u << sh.log) < shares) sh.log++;
    sh.groups = groups;
    sh.groups_inv = (65536 + groups - 1) / groups;  // (at most 8 groups x 16 shares)
    if (shares > 1) {
        if (!scratch.part || !scratch.counts) return cudaErrorInvalidValue;
        sh.counts = scratch.counts;
        sh.part = (float4*)scratch.part;
        kern = attend_kernel<HD, R, T, true>;  // (code of its own: what the shares ask costs the others 2 %)
    }
    int g_log = 0;
    while ((1u << g_log) < G) g_log++;
    if (cudaError_t e = ensure_dynamic_smem((const void*)kern, smem, 0); e != cudaSuccess) return e;
    // (clusters of more than eight CTAs have to be asked for)
    if (cudaError_t e = cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1); e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C, p.nkv, groups * shares);
    cfg.blockDim = dim3(ATT_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kern, q, (T*)kc, (T*)vc, out, sp, p, status, fr, at, g_log, sh);
}

template <int HD, typename T>
cudaError_t attend_r(const float* q, void* kc, void* vc, float* out, const uint32_t* sp, const DecAttn& p, uint32_t* status, cudaStream_t st, bool pdl,
                     const FusedRope& fr, const AttnTokens& at, const AttScratch& scratch) {
    const uint32_t rows = p.nh / p.nkv * (uint32_t)std::max(1, at.n);
    if (rows <= 1) return attend_t<HD, 1, T>(q, kc, vc, out, sp, p, status, st, pdl, fr, at, scratch);
    if (rows <= 2) return attend_t<HD, 2, T>(q, kc, vc, out, sp, p, status, st, pdl, fr, at, scratch);
    return attend_t<HD, ATT_MOST_ROWS, T>(q, kc, vc, out, sp, p, status, st, pdl, fr, at, scratch);
}

}  // namespace

bool attend_supports(uint32_t nh, uint32_t nkv, uint32_t hd) {
    if (nkv == 0 || nh % nkv) return false;
    const uint32_t g = nh / nkv;
    return (hd == 64 || hd == 128) && (g == 1 || g == 2 || g == 4 || g == 8);
}

static size_t attend_units(uint32_t nh, uint32_t nkv, uint32_t tokens) { return nkv * (((size_t)(nh / nkv) * tokens + ATT_MOST_ROWS - 1) / ATT_MOST_ROWS); }
size_t attend_part_floats(uint32_t nh, uint32_t nkv, uint32_t hd, uint32_t max_len, uint32_t tokens) {
    const size_t shares = attend_shares(nh, nkv, max_len);
    return shares > 1 ? attend_units(nh, nkv, tokens) * shares * (ATT_MOST_ROWS * hd / 4) * 8 : 0;
}
size_t attend_count_words(uint32_t nh, uint32_t nkv, uint32_t max_len, uint32_t tokens) {
    return attend_shares(nh, nkv, max_len) > 1 ? attend_units(nh, nkv, tokens) * ATT_PARTS : 0;
}

cudaError_t launch_attend(const float* q, void* kc, void* vc, int kv_f16, float* out, const uint32_t* sp, const DecAttn& p, uint32_t* status,
                          const AttScratch& scratch, cudaStream_t st, bool pdl, const FusedRope* frp, const AttnTokens* atp) {
    if (!attend_supports(p.nh, p.nkv, p.hd)) return cudaErrorInvalidValue;
    AttnTokens at{};
    if (atp) at = *atp;
    if (at.n > ATT_STEP_TOKENS) return cudaErrorInvalidValue;
    FusedRope fr{};
    if (frp) {
        fr = *frp;
        if (fr.r.nh != p.nh || fr.r.nkv != p.nkv || fr.r.hd != p.hd || 2 * fr.r.half_rot > p.hd || fr.r.v_norm || fr.r.v_from_k)
            return cudaErrorInvalidValue;
    }
    if (p.hd == 64)
        return kv_f16 ? attend_r<64, __half>(q, kc, vc, out, sp, p, status, st, pdl, fr, at, scratch) : attend_r<64, float>(q, kc, vc, out, sp, p, status, st, pdl, fr, at, scratch);
    return kv_f16 ? attend_r<128, __half>(q, kc, vc, out, sp, p, status, st, pdl, fr, at, scratch) : attend_r<128, float>(q, kc, vc, out, sp, p, status, st, pdl, fr, at, scratch);
}

}  // namespace b2
