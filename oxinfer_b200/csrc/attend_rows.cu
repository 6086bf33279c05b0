// Causal attention of a prefill step's query tokens over the cache on the fifth-generation tensor cores (tcgen05): S = Q K^T and O += P V with f16
// operands and f32 sums, softmax running in f32. The reference's prefill attention is its f32 CPU kernel (attention_ext,
// src/model.rs:2214-2309) or attention_cached on the device; this one rounds q, k, v and the probabilities to f16, which the parity bound of the prefill
// plan covers. An f32 cache is first copied to f16.
//
// The rows of a KV head are its query heads' tokens, row r being head r % G of token r / G, so that a tile of 128 rows ends within 128 / G tokens
// whatever G is. A CTA takes two tiles (256 rows) and key tiles of 128:
//   warps 0..3, 4..7 : softmax of a row tile, a thread a row: scores out of tensor memory, their largest, exponentials, probabilities as f16 back
//                      into tensor memory in the scores' place. Where a row of the warp has a new largest score, the sums in O are brought to it. (Only
//                      where it has grown by 2^8: 3 % faster, but the largest probability is then no longer exactly 1: up to 17 % more error for
//                      peaked rows.) Then the epilogue.
//   warps 8, 9       : issue the instructions of a row tile each: while one tile's probabilities are made, the other tile's products run. (An
//                      instruction's two descriptors take a thread about 90 cycles to set up, the tensor cores 64 to work through.)
//   warp 10          : copies keys and values (128-byte swizzled tiles of 64 dimensions, two slots each; rows behind the last are zeros).
// Tensor memory: two tiles of scores (128 columns each) and two of sums (head dimension each): all 512 columns, one CTA an SM.
// Few rows over many keys: Z CTAs of a cluster take a share of the key tiles each, and add their sums through shared memory.
// 64 keys that no row of a tile sees (half of the tile at the end of the causal triangle, windows) are left out of its products: 32 / 8 heads, 2048
// tokens with RoPE 120.6 -> 113.4 us, and what stands in them reaches nobody. Launches whose CTAs all run at once are dependent ones.
//
// What bounds it: 128 x 128 scores of a head of 128 take the tensor cores 1024 cycles and the exponential unit as many.
// f32 caches, 32 query and 8 KV heads of 128, launches of 2048 tokens 98 us before 64 keys were left out (mma.sync, 64 x 64 tiles a warp group: 202).
// With the RoPE launch and the copy of the cache to f16, us a layer now: 2048 tokens 121, behind 4000 keys 288, 300 tokens behind 1000 keys 38, 64
// behind 4000 36, 128 tokens alone 17.2 (23.4 without dependent launches), 16 alone 12.9 (19.0); f16 caches 113, 268, 34, 29, 15.7, 11.
// Error against 64 bits: as the form on mma.sync
// (ratio 0.978 .. 1.009 over 96 shapes and two score ranges). A launch of few tokens over few keys is a chain of 7 us: the queries' and the
// first keys' loads, one tile, the rows out.
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "gemm_wt.h"
#include "pdl.cuh"
#include "tcgen05.cuh"

namespace b2 {

namespace {

constexpr int AR_THREADS = 384, AR_TILE = 128;  // rows of a tile, and keys
constexpr uint32_t AR_TMEM_COLS = 512;

struct __align__(16) ArShared {
    float m[2 * AR_TILE], l[2 * AR_TILE];  // the rows' largest scores (in powers of two) and denominators
    uint64_t k_full[2], k_empty[2], v_full[2], v_empty[2], q_full, s_full[2], p_full[2][2], o_full;  // p_full: [row tile][half of the keys]
    uint32_t tmem_base;
    volatile uint32_t abort_flag;
};
struct ArArgs {
    const float* q;
    float* out;
    size_t stride;
    uint32_t rows, G, g_inv, pos0, window;  // rows: tokens x G; g_inv: ceil(2^32 / G), 0 for one head
    float c;                         // scores in powers of two; q_sign: its sign
    float q_sign;
    int Z;
    GemmStatus* status;
};

__device__ __forceinline__ void ar_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, "
        "%22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
          "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]),
          "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]),
          "=r"(v[31])
        : "r"(taddr));
}
__device__ __forceinline__ void ar_st32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, "
        "%21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]),
        "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]),
        "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
__device__ __forceinline__ void ar_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void ar_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void ar_mma_ts(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
        "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ float ar_max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// Two at a time, each rounded as the single instruction rounds it.
__device__ __forceinline__ float2 ar_fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\tfma.rn.f32x2 a, a, b, c;\n\tmov.b64 {%0, %1}, a;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}
__device__ __forceinline__ float2 ar_add2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 a, b;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tadd.rn.f32x2 a, a, b;\n\tmov.b64 {%0, %1}, a;\n\t}" : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float ar_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ uint32_t ar_pack(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *(const uint32_t*)&h;
}
// Values as the B operand, [64 dimensions][key rows of 128 bytes] a swizzled tile: the instruction's N runs along a row, its K from row to row.
__device__ __forceinline__ uint64_t ar_v_desc(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFF);
    d |= (uint64_t)((AR_TILE * 128) >> 4) << 16;  // from 64 dimensions to the next
    d |= (uint64_t)(1024 >> 4) << 32;             // from eight keys to the next
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
__device__ __forceinline__ float4 ar_peer_f4(const void* p, uint32_t cta) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(cluster_addr(p, cta)) : "memory");
    return v;
}
__device__ __forceinline__ float ar_peer_f(const void* p, uint32_t cta) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(cluster_addr(p, cta)) : "memory");
    return v;
}

// The first key that a query at position qp sees.
__device__ __forceinline__ uint32_t ar_first_key(const ArArgs& a, uint32_t qp) { return a.window != 0 && qp + 1 > a.window ? qp + 1 - a.window : 0; }
// Row r's token (r G < 2^32).
__device__ __forceinline__ uint32_t ar_token(const ArArgs& a, uint32_t r) { return a.g_inv ? __umulhi(r, a.g_inv) : r; }

template <int HD>
__host__ __device__ constexpr size_t attend_rows_smem() {  // queries of two tiles, two slots of keys and of values; over them the sums (f32)
    const size_t tiles = (size_t)6 * AR_TILE * HD * 2;
    return (tiles < TMEM_512_SMEM ? TMEM_512_SMEM : tiles) + 1024;
}

static_assert(attend_rows_smem<64>() >= TMEM_512_SMEM && attend_rows_smem<128>() >= TMEM_512_SMEM);

// Grid (Z x row blocks, KV heads), Z CTAs along x a cluster.
template <int HD>
__global__ void __launch_bounds__(AR_THREADS, 1)
attend_rows_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ ArArgs a) {
    constexpr uint32_t TILE_BYTES = AR_TILE * HD * 2, HALVES = HD / 64, HALF_BYTES = AR_TILE * 128;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* const smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* const q_s = smem;                    // [tile][half][128 rows][128 bytes]
    uint8_t* const k_s = smem + 2 * TILE_BYTES;   // [slot]..
    uint8_t* const v_s = smem + 4 * TILE_BYTES;
    __shared__ ArShared shared;
    ArShared* sh = &shared;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t z = blockIdx.x % a.Z, kvh = blockIdx.y;
    const uint32_t r_block = (gridDim.x - 1 - blockIdx.x) / a.Z * (2 * AR_TILE);  // the blocks with the most keys first
    const uint32_t r_end = min(r_block + 2 * AR_TILE, a.rows);
    const int tiles = r_block + AR_TILE < r_end ? 2 : 1;
    const uint32_t first_qp = a.pos0 + ar_token(a, r_block), last_qp = a.pos0 + ar_token(a, r_end - 1);
    const uint32_t lo = ar_first_key(a, first_qp);
    const uint32_t all_0 = lo / AR_TILE, all_n = last_qp / AR_TILE + 1 - all_0, share = (all_n + a.Z - 1) / a.Z;
    const uint32_t t_first = all_0 + z * share;
    const int n = (int)min(share, all_0 + all_n > t_first ? all_0 + all_n - t_first : 0u);  // this CTA's key tiles

    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; s++) {
            mbar_init(&sh->k_full[s], 1);
            mbar_init(&sh->k_empty[s], tiles);
            mbar_init(&sh->v_full[s], 1);
            mbar_init(&sh->v_empty[s], tiles);
            mbar_init(&sh->s_full[s], 1);
            mbar_init(&sh->p_full[s][0], 4);
            mbar_init(&sh->p_full[s][1], 4);
        }
        mbar_init(&sh->q_full, 8);
        mbar_init(&sh->o_full, 2);
        sh->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 8) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh->tmem_base)), "r"(AR_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh->tmem_base;
    pdl_wait();  // (queries, keys and values come from the kernel ahead)

    // A launch of 384 threads has 168 registers a thread: the softmax warps take 232 (a row's 128 scores among them), the others keep 40.
    if (warp >= 8) {
      asm volatile("setmaxnreg.dec.sync.aligned.u32 40;" ::: "memory");
      if (warp == 10) {
        // ---------------- keys and values ----------------
        int k_issued = 0, v_issued = 0;
        for (int i = 0; i < n; i++) {
            const int s = i & 1, row = (int)((t_first + i) * AR_TILE);
            const uint32_t back = (uint32_t)(((i >> 1) - 1) & 1);
            auto copy = [&](uint64_t* full, uint64_t* empty, uint8_t* dst, const CUtensorMap* map, uint32_t where) {
                if (i >= 2 && !__all_sync(0xffffffffu, mbar_wait(empty, back, sh, a.status, where, (uint32_t)i))) return false;
                if (elect_one()) {
                    mbar_arrive_expect_tx(full, TILE_BYTES);
#pragma unroll
                    for (int h = 0; h < (int)HALVES; h++) tma_load_3d(dst + s * TILE_BYTES + h * HALF_BYTES, map, full, 64 * h, row, (int)kvh);
                }
                __syncwarp();
                return true;
            };
            if (!copy(&sh->k_full[s], &sh->k_empty[s], k_s, &tmap_k, 61)) break;  // (the keys' slot is free before the values')
            k_issued = i + 1;
            if (!copy(&sh->v_full[s], &sh->v_empty[s], v_s, &tmap_v, 62)) break;
            v_issued = i + 1;
        }
        if (sh->abort_flag) {  // copies in flight land before the shared memory goes away
            for (int i = max(0, k_issued - 2); i < k_issued; i++) mbar_wait(&sh->k_full[i & 1], (uint32_t)((i >> 1) & 1), sh, a.status, 63, (uint32_t)i, false);
            for (int i = max(0, v_issued - 2); i < v_issued; i++) mbar_wait(&sh->v_full[i & 1], (uint32_t)((i >> 1) & 1), sh, a.status, 64, (uint32_t)i, false);
        }
      } else if (warp < 10) {
        // ---------------- instructions ----------------
        constexpr uint32_t idesc_qk = (1u << 4) | ((AR_TILE >> 3) << 17) | ((AR_TILE >> 4) << 24);
        constexpr uint32_t idesc_pv = (1u << 4) | (1u << 16) | ((HD >> 3) << 17) | ((AR_TILE >> 4) << 24);  // (B with N along its rows)
        const int w = warp - 8;
        const uint64_t qd = smem_desc_sw128(smem_u32(q_s) + w * TILE_BYTES), kd = smem_desc_sw128(smem_u32(k_s)), vd = ar_v_desc(smem_u32(v_s));
        const uint32_t s_at = tmem + w * AR_TILE, o_at = tmem + 2 * AR_TILE + w * HD;
        auto scores = [&](int s) {
            if (elect_one()) {
                const uint64_t k = kd + (s * TILE_BYTES >> 4);
#pragma unroll
                for (int kk = 0; kk < HD / 16; kk++) {
                    const uint32_t at = (uint32_t)(kk >> 2) * (HALF_BYTES >> 4) + 2 * (kk & 3);
                    mma_f16(s_at, qd + at, k + at, idesc_qk, kk > 0);
                }
                mma_commit(&sh->s_full[w]);
                mma_commit(&sh->k_empty[s]);
            }
            __syncwarp();
        };
        bool ok = n > 0 && w < tiles;
        auto wait = [&](uint64_t* bar, uint32_t phase, uint32_t where, int i) {
            ok = ok && __all_sync(0xffffffffu, mbar_wait(bar, phase, sh, a.status, where, (uint32_t)i));
            tc_fence_after();
            return ok;
        };
        // 64 keys that no row of the tile sees are left out: their probabilities are zeros, but a value that is not finite would still reach the sums
        const uint32_t tile_0 = min(r_block + w * AR_TILE, a.rows - 1), see_to = a.pos0 + ar_token(a, min(tile_0 + AR_TILE - 1, a.rows - 1));
        const uint32_t see_from = ar_first_key(a, a.pos0 + ar_token(a, tile_0));
        uint32_t started = 0;
        if (ok && wait(&sh->q_full, 0, 65, 0) && wait(&sh->k_full[0], 0, 66, 0)) scores(0);
        for (int i = 0; i < n && ok; i++) {
            const int s = i & 1, s1 = s ^ 1;
            if (!wait(&sh->v_full[s], (uint32_t)((i >> 1) & 1), 67, i)) break;
            if (i + 1 < n && !wait(&sh->k_full[s1], (uint32_t)(((i + 1) >> 1) & 1), 68, i)) break;
#pragma unroll
            for (int h = 0; h < 2; h++) {  // (the first half's products run under the second half's exponentials)
                if (!wait(&sh->p_full[w][h], (uint32_t)(i & 1), 69, i)) break;
                const uint32_t j = (t_first + i) * AR_TILE + 64 * h;
                const bool seen = j <= see_to && j + 63 >= see_from;
                if (elect_one()) {
                    const uint64_t v = vd + (s * TILE_BYTES >> 4) + 512 * h;
                    if (seen) {
#pragma unroll
                        for (int kk = 0; kk < AR_TILE / 32; kk++) ar_mma_ts(o_at, s_at + 32 * h + 8 * kk, v + 128 * kk, idesc_pv, started | kk);
                    }
                    if (h) mma_commit(&sh->v_empty[s]);
                }
                started |= seen;
                __syncwarp();
            }
            if (ok && i + 1 < n) scores(s1);
        }
        // (a share without keys: its sums, zeros, take the queries' place, which other warps may still be writing)
        if (n == 0) mbar_wait(&sh->q_full, 0, sh, a.status, 65, 0);
        if (elect_one()) mma_commit(&sh->o_full);
        __syncwarp();
        if (n > 0 && w < tiles && !ok) mbar_wait(&sh->o_full, 0, sh, a.status, 70, 0, false);
      }
      if (a.Z > 1) {  // (the softmax warps' two below)
          __syncwarp();
          cluster_sync_all();
          cluster_sync_all();
      }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 232;" ::: "memory");
        // ---------------- softmax ----------------
        const int w = warp >> 2;
        const bool live = w < tiles;
        {  // the tile's queries as f16: a warp's 32 rows, a row's values over the lanes
            constexpr int PER = HD / 4, ROWS = 32 / PER;  // lanes a row, rows a turn
            const uint32_t d4 = (uint32_t)(lane % PER), half = d4 >> 4, chunk = (d4 & 15) >> 1, in = (d4 & 1) * 8;
            // sixteen loads in flight (one by one behind the stores they took 11000 cycles)
            constexpr int FLIGHT = 16;
#pragma unroll
            for (int i0 = 0; i0 < 32; i0 += FLIGHT * ROWS) {
                float4 v[FLIGHT];
#pragma unroll
                for (int i = 0; i < FLIGHT; i++) {
                    const uint32_t r = min(r_block + w * AR_TILE + (warp & 3) * 32 + i0 + i * ROWS + lane / PER, a.rows - 1), tok = ar_token(a, r);
                    v[i] = *(const float4*)(a.q + tok * a.stride + (size_t)(kvh * a.G + (r - tok * a.G)) * HD + 4 * d4);
                }
#pragma unroll
                for (int i = 0; i < FLIGHT; i++) {
                    const uint32_t row = (uint32_t)((warp & 3) * 32 + i0 + i * ROWS + lane / PER);
                    *(uint2*)(q_s + w * TILE_BYTES + half * HALF_BYTES + row * 128 + ((chunk ^ (row & 7)) << 4) + in) =
                        make_uint2(ar_pack(v[i].x * a.q_sign, v[i].y * a.q_sign), ar_pack(v[i].z * a.q_sign, v[i].w * a.q_sign));
                }
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh->q_full);
        }
        const uint32_t row = (uint32_t)((warp & 3) * 32 + lane), r = min(r_block + w * AR_TILE + row, a.rows - 1), qp = a.pos0 + ar_token(a, r);
        const uint32_t tile_qp = a.pos0 + ar_token(a, min(r_block + w * AR_TILE, a.rows - 1));                          // the tile's first position
        const uint32_t tile_end = a.pos0 + ar_token(a, min(r_block + w * AR_TILE + AR_TILE - 1, a.rows - 1));           // and its last
        const uint32_t my_lo = ar_first_key(a, qp);
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16, s_at = tmem + lane_base + w * AR_TILE, o_at = tmem + lane_base + 2 * AR_TILE + w * HD;
        float m = -INFINITY, l = 0.0f;
        bool ok = true;
        for (int i = 0; i < n && live; i++) {
            ok = __all_sync(0xffffffffu, mbar_wait(&sh->s_full[w], (uint32_t)(i & 1), sh, a.status, 71, (uint32_t)i));
            if (!ok) break;
            tc_fence_after();
            uint32_t v[4][32];
#pragma unroll
            for (int h = 0; h < 4; h++) ar_ld32(s_at + 32 * h, v[h]);
            ar_ld_wait();
            const uint32_t j0 = (t_first + i) * AR_TILE;
            if (j0 + AR_TILE - 1 > tile_qp || (a.window != 0 && j0 + a.window <= tile_end)) {  // some row does not see some key
                const uint32_t hi = qp >= j0 ? min(qp - j0 + 1, (uint32_t)AR_TILE) : 0u, from = my_lo > j0 ? my_lo - j0 : 0u;  // keys from .. hi - 1 of the tile
                auto below = [](uint32_t n, int h) { return n >= 32u * h + 32 ? 0xffffffffu : n <= 32u * h ? 0u : (1u << (n - 32 * h)) - 1; };  // a bit per key below n
#pragma unroll
                for (int h = 0; h < 4; h++) {
                    const uint32_t seen = below(hi, h) & ~below(from, h);
#pragma unroll
                    for (int e = 0; e < 32; e++)
                        if (!(seen & (1u << e))) v[h][e] = 0xff800000u;
                }
            }
            float mx[4];
#pragma unroll
            for (int h = 0; h < 4; h++) {
                mx[h] = fmaxf(__uint_as_float(v[h][0]), __uint_as_float(v[h][1]));
#pragma unroll
                for (int e = 2; e < 32; e += 2) mx[h] = ar_max3(mx[h], __uint_as_float(v[h][e]), __uint_as_float(v[h][e + 1]));
            }
            const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * a.c;
            if (i == 0) {
                m = top;
            } else if (__any_sync(0xffffffffu, top > m)) {
                const float mn = fmaxf(m, top), f = m == -INFINITY ? 0.0f : ar_exp2(m - mn);
                m = mn;
                l *= f;
#pragma unroll
                for (int h = 0; h < HD / 32; h++) {
                    uint32_t o[32];
                    ar_ld32(o_at + 32 * h, o);
                    ar_ld_wait();
#pragma unroll
                    for (int e = 0; e < 32; e++) o[e] = __float_as_uint(__uint_as_float(o[e]) * f);
                    ar_st32(o_at + 32 * h, o);
                }
            }
            const float base = m == -INFINITY ? 0.0f : -m;
            float2 part[2] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
#pragma unroll
            for (int h = 0; h < 2; h++) {
                uint32_t pk[32];
#pragma unroll
                for (int e = 0; e < 32; e++) {
                    const uint32_t* at = &v[2 * h + (e >> 4)][2 * (e & 15)];
                    float2 x = ar_fma2(make_float2(__uint_as_float(at[0]), __uint_as_float(at[1])), make_float2(a.c, a.c), make_float2(base, base));
                    x = make_float2(ar_exp2(x.x), ar_exp2(x.y));
                    part[e & 1] = ar_add2(part[e & 1], x);
                    pk[e] = ar_pack(x.x, x.y);
                }
                ar_st32(s_at + 32 * h, pk);
                ar_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh->p_full[w][h]);
            }
            l += (part[0].x + part[0].y) + (part[1].x + part[1].y);
        }
        // ---------------- the sums, into shared memory over the tiles ----------------
        ok = __all_sync(0xffffffffu, mbar_wait(&sh->o_full, 0, sh, a.status, 72, 0) && !sh->abort_flag);
        if (ok && live) {
            tc_fence_after();
            float4* const dst = (float4*)(smem + (size_t)(w * AR_TILE + row) * HD * 4);
            // (the tile's rows may see none of this CTA's keys: there are no sums then)
            const bool none = n == 0 || tile_end < t_first * AR_TILE || ar_first_key(a, tile_qp) >= (t_first + n) * AR_TILE;
#pragma unroll
            for (int h = 0; h < HD / 32; h++) {
                uint32_t o[32];
                ar_ld32(o_at + 32 * h, o);
                ar_ld_wait();
#pragma unroll
                for (int e = 0; e < 8; e++)
                    dst[(8 * h + e) ^ (row & 7)] = none ? make_float4(0.f, 0.f, 0.f, 0.f)
                                                        : make_float4(__uint_as_float(o[4 * e]), __uint_as_float(o[4 * e + 1]), __uint_as_float(o[4 * e + 2]), __uint_as_float(o[4 * e + 3]));
            }
            sh->m[w * AR_TILE + row] = m;
            sh->l[w * AR_TILE + row] = a.Z > 1 ? l : l > 0.0f ? 1.0f / l : 0.0f;
        }
        __syncwarp();
        if (a.Z > 1) cluster_sync_all();
        else asm volatile("bar.sync 1, 256;" ::: "memory");
        // ---------------- the rows out: CTA z every Z-th run of 32 / PER rows ----------------
        if (!sh->abort_flag) {
            constexpr int PER = HD / 4, ROWS = 32 / PER;
            const uint32_t f = (uint32_t)(lane % PER);
            const uint32_t count = r_end - r_block, step = a.Z * 8 * ROWS;
            // (short loops: unrolled, their code runs at the rate of its instruction fetches, 10000 cycles)
            auto put = [&](uint32_t row, float4 o, float inv) {
                const uint32_t r = r_block + row, tok = ar_token(a, r);
                if (row < count)
                    *(float4*)(a.out + tok * a.stride + (size_t)(kvh * a.G + (r - tok * a.G)) * HD + 4 * f) = make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv);
            };
            auto at_row = [&](uint32_t row) { return (const float4*)(smem + (size_t)row * HD * 4) + (f ^ (row & 7)); };
            if (a.Z == 1) {
#pragma unroll 2
                for (uint32_t at = warp * ROWS + lane / PER; at < count + lane / PER; at += step) {
                    const uint32_t row = min(at, count - 1);
                    put(at, *at_row(row), sh->l[row]);
                }
            } else {
                for (uint32_t at = (z * 8 + warp) * ROWS; at < count; at += step) {
                    const uint32_t row = min(at + lane / PER, count - 1);
                    float m[8], l[8];
                    float4 b[8];
#pragma unroll
                    for (int k = 0; k < 8; k++) {  // (Z is 2, 4 or 8)
                        if (k >= a.Z) break;
                        m[k] = ar_peer_f(&sh->m[row], k);
                        l[k] = ar_peer_f(&sh->l[row], k);
                        b[k] = ar_peer_f4(at_row(row), k);
                    }
                    float M = m[0];
#pragma unroll
                    for (int k = 1; k < 8; k++)
                        if (k < a.Z) M = fmaxf(M, m[k]);
                    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
                    float den = 0.0f;
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        if (k >= a.Z) break;
                        const float wgt = M == -INFINITY ? 0.0f : ar_exp2(m[k] - M);
                        o = make_float4(fmaf(wgt, b[k].x, o.x), fmaf(wgt, b[k].y, o.y), fmaf(wgt, b[k].z, o.z), fmaf(wgt, b[k].w, o.w));
                        den = fmaf(wgt, l[k], den);
                    }
                    put(at + lane / PER, o, den > 0.0f ? 1.0f / den : 0.0f);
                }
            }
        }
        if (a.Z > 1) {  // no CTA leaves while another reads its sums
            __syncwarp();
            cluster_sync_all();
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 8) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(AR_TMEM_COLS) : "memory");
    }
}

// f32 cache rows [0, len) of every KV head -> an f16 copy with the same layout ([nkv][max_len][hd]); keys and values along z.
__global__ void __launch_bounds__(256) kv_rows_to_f16_kernel(const float* __restrict__ k, const float* __restrict__ v, __half* __restrict__ k16, __half* __restrict__ v16,
                                                             uint32_t max_len, uint32_t len, uint32_t hd4) {
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;  // a group of 4 values of the head's first `len` rows
    if (i >= len * hd4) return;
    const size_t at = ((size_t)blockIdx.y * max_len * hd4 + i) * 4;
    const float4 x = *(const float4*)((blockIdx.z ? v : k) + at);
    *(uint2*)((blockIdx.z ? v16 : k16) + at) = make_uint2(ar_pack(x.x, x.y), ar_pack(x.z, x.w));
}

template <int HD>
cudaError_t attend_rows_t(const CUtensorMap& k, const CUtensorMap& v, const ArArgs& a, uint32_t nkv, int sm_count, cudaStream_t st) {
    constexpr size_t smem = attend_rows_smem<HD>();
    auto kern = attend_rows_kernel<HD>;
    if (cudaError_t e = ensure_dynamic_smem((const void*)kern, smem, 0); e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((a.rows + 2 * AR_TILE - 1) / (2 * AR_TILE) * a.Z, nkv);
    cfg.blockDim = dim3(AR_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)a.Z;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    // Dependent where the CTAs run at once: the start (tensor memory, barriers, maps) under the kernel ahead. (f16 caches, 32 query and 8 KV heads
    // of 128, RoPE and attention
    // of 8 / 128 / 600 tokens: 14.9 / 19.4 / 36.5 us, dependent 10.9 / 17.2 / 33.9, on mma.sync 12.9 / 21.3 / 56; of 2048, 256 CTAs: 120 and 123.)
    cfg.numAttrs = cfg.gridDim.x * nkv <= (unsigned)sm_count ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kern, k, v, a);
}

// The cache's f16 rows [nkv][len of max_len][hd] by tiles of 128 rows x 64 dimensions; rows from len on read as zeros.
bool kv_map(CUtensorMap* m, const __half* base, uint32_t nkv, uint32_t len, uint32_t max_len, uint32_t hd) {
    TensorMapEncodeFn enc = tensor_map_encode();
    if (!enc) return false;
    cuuint64_t dims[3] = {hd, len, nkv};
    cuuint64_t strides[2] = {(cuuint64_t)hd * 2, (cuuint64_t)max_len * hd * 2};
    cuuint32_t box[3] = {64, AR_TILE, 1}, estr[3] = {1, 1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, (void*)base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

bool attend_rows_supports(uint32_t nh, uint32_t nkv, uint32_t hd) { return nkv != 0 && nh % nkv == 0 && (hd == 64 || hd == 128); }

size_t attend_rows_scratch_bytes(uint32_t nkv, uint32_t max_len, uint32_t hd, int kv_f16) {
    return kv_f16 ? 0 : (size_t)2 * nkv * max_len * hd * 2;
}

cudaError_t launch_attend_rows(const float* q, float* out, size_t stride, uint32_t tokens, const void* kc, const void* vc, int kv_f16, void* scratch,
                               uint32_t len, const DecAttn& p, GemmStatus* status, int sm_count, cudaStream_t st) {
    if (!attend_rows_supports(p.nh, p.nkv, p.hd) || tokens == 0 || stride % 4 || ((uintptr_t)q & 15) || ((uintptr_t)out & 15) || len > p.max_len || len < tokens || p.nkv > 65535)
        return cudaErrorInvalidValue;
    const __half *kh = (const __half*)kc, *vh = (const __half*)vc;
    if (!kv_f16) {  // an f16 copy of the rows the step reads (the kernel's operands are f16 either way)
        if (!scratch) return cudaErrorInvalidValue;
        __half* k16 = (__half*)scratch;
        __half* v16 = k16 + (size_t)p.nkv * p.max_len * p.hd;
        if (cudaError_t e = launch_k(kv_rows_to_f16_kernel, dim3((len * (p.hd / 4) + 255) / 256, p.nkv, 2), dim3(256), 0, st, true, (const float*)kc, (const float*)vc, k16, v16,
                                     p.max_len, len, p.hd / 4);
            e != cudaSuccess)
            return e;
        kh = k16;
        vh = v16;
    }
    CUtensorMap km, vm;
    if (!kv_map(&km, kh, p.nkv, len, p.max_len, p.hd) || !kv_map(&vm, vh, p.nkv, len, p.max_len, p.hd)) return cudaErrorInvalidValue;
    ArArgs a{};
    a.q = q;
    a.out = out;
    a.stride = stride;
    a.G = p.nh / p.nkv;
    a.g_inv = a.G == 1 ? 0u : (uint32_t)(((1ull << 32) + a.G - 1) / a.G);
    a.rows = tokens * a.G;
    a.pos0 = len - tokens;
    a.window = p.window >= p.max_len ? 0 : p.window;  // (none then, and a key's position plus the window does not wrap)
    a.q_sign = p.scale < 0.0f ? -1.0f : 1.0f;
    a.c = std::max(p.scale * a.q_sign, 1e-30f) * 1.44269504f;  // (a factor of zero would make a masked key's score NaN)
    a.status = status;
    // Shares of the keys while two fit the chip beside each other and have two tiles each
    const uint32_t ctas = (a.rows + 2 * AR_TILE - 1) / (2 * AR_TILE) * p.nkv, tiles = (len + AR_TILE - 1) / AR_TILE;
    a.Z = 1;
    while (a.Z < 8 && 2 * a.Z * ctas <= (uint32_t)sm_count && 4 * (uint32_t)a.Z <= tiles) a.Z *= 2;
    return p.hd == 64 ? attend_rows_t<64>(km, vm, a, p.nkv, sm_count, st) : attend_rows_t<128>(km, vm, a, p.nkv, sm_count, st);
}

}  // namespace b2
