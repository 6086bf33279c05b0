// Decode plan: resolves a b2_graph to device pointers, decides where each product's activation split is made (by
// the product itself, with the RMS norm in front of it, or by a kernel of its own), captures the op list into CUDA
// graphs, and runs steps.
// What the reference does per token with ~11 cuLaunchKernel calls per layer from the host
// (src/cuda_decode.rs:1466-1658) is one cudaGraphLaunch here.
#include "plan.h"

#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <algorithm>
#include <map>
#include <memory>
#include <tuple>

namespace b2 {

namespace {

constexpr uint32_t OP_SPLIT = 100;  // internal: the record of a vector (launch_split)
constexpr int ATT_THREADS_HOST = 256;  // threads of an attention unit (a thread per head dimension makes the token's key row)
static bool overlaps_f(const float* a, size_t na, const float* b, size_t nb) { return a && b && na && nb && a < b + nb && b < a + na; }
std::string fmt(const char* f, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, f);
    vsnprintf(buf, sizeof buf, f, ap);
    va_end(ap);
    return buf;
}

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

#define PLAN_CUDA(call, what)                                                                  \
    do {                                                                                       \
        cudaError_t e_ = (call);                                                               \
        if (e_ != cudaSuccess) {                                                               \
            err = fmt("[b200qmm: plan: %s: %s]", what, cudaGetErrorString(e_));                \
            return e_ == cudaErrorMemoryAllocation ? B2_ERR_NOMEM : B2_ERR_CUDA;               \
        }                                                                                      \
    } while (0)

// Bytes of one row in each of the (up to four) device planes of a format; 0 = plane unused.
void row_bytes(const WeightDev& w, size_t (&rb)[4]) {
    const size_t K = w.n_in;
    rb[0] = rb[1] = rb[2] = rb[3] = 0;
    switch (w.fmt) {
        case B2_FMT_MLX4:
        case B2_FMT_Q4_K: rb[0] = (K / 256) * 144; break;
        case B2_FMT_Q6_K:
            rb[0] = K / 2;
            rb[1] = K / 4;
            rb[2] = K / 16;
            rb[3] = (K / 256) * 2;
            break;
        case B2_FMT_Q8_0:
            rb[0] = K;
            rb[1] = (K / 32) * 2;
            break;
        case B2_FMT_F8E4M3: rb[0] = K; break;  // (its block scales: fuse_rows)
    }
}
// Whether a matrix's rows may be a part of a concatenation: FP8 parts have to be whole rows of scale blocks.
bool fusable(const WeightDev& w) {
    return w.fmt != B2_FMT_F8E4M3 || w.p1 == nullptr || (w.n_out % w.bs_rows == 0 && w.bs_row0 % w.bs_rows == 0);
}

// One matrix whose rows are the rows of `parts` in order (same format and n_in): device copies, owned by the plan.
cudaError_t fuse_rows(const std::vector<const WeightDev*>& parts, WeightDev* out, std::vector<void*>& owned) {
    *out = *parts[0];
    size_t rb[4], total = 0;
    row_bytes(*parts[0], rb);
    for (const WeightDev* w : parts) total += w->n_out;
    out->n_out = total;
    const uint8_t* WeightDev::*planes[4] = {&WeightDev::p0, &WeightDev::p1, &WeightDev::p2, &WeightDev::p3};
    for (int pl = 0; pl < 4; pl++) {
        if (!rb[pl]) continue;
        uint8_t* d = nullptr;
        cudaError_t e = cudaMalloc((void**)&d, total * rb[pl]);
        if (e != cudaSuccess) return e;
        owned.push_back(d);
        size_t at = 0;
        for (const WeightDev* w : parts) {
            e = cudaMemcpy(d + at, w->*planes[pl], w->n_out * rb[pl], cudaMemcpyDeviceToDevice);
            if (e != cudaSuccess) return e;
            at += w->n_out * rb[pl];
        }
        out->*planes[pl] = d;
    }
    if (parts[0]->fmt == B2_FMT_F8E4M3 && parts[0]->p1) {
        const size_t row = parts[0]->bs_ncb * 4;
        uint8_t* d = nullptr;
        cudaError_t e = cudaMalloc((void**)&d, total / parts[0]->bs_rows * row);
        if (e != cudaSuccess) return e;
        owned.push_back(d);
        size_t at = 0;
        for (const WeightDev* w : parts) {
            const size_t bytes = w->n_out / w->bs_rows * row;
            e = cudaMemcpy(d + at, w->p1 + w->bs_row0 / w->bs_rows * row, bytes, cudaMemcpyDeviceToDevice);
            if (e != cudaSuccess) return e;
            at += bytes;
        }
        out->p1 = d;
        out->bs_row0 = 0;
    }
    // (a copy within the device does not wait for itself, and products fetch weights before they wait for the work ahead)
    return cudaStreamSynchronize(cudaStreamLegacy);
}

}  // namespace

DecodePlanImpl::~DecodePlanImpl() {
    for (void* p : fused_) cudaFree(p);
    if (step_exec_) cudaGraphExecDestroy(step_exec_);
    for (cudaGraphExec_t e : multi_exec_)
        if (e) cudaGraphExecDestroy(e);
    if (gen_exec_) cudaGraphExecDestroy(gen_exec_);
    if (ev0_) cudaEventDestroy(ev0_);
    if (ev1_) cudaEventDestroy(ev1_);
    if (cap_stream_) cudaStreamDestroy(cap_stream_);
    for (auto& k : kv_) {
        if (k.k) cudaFree(k.k);
        if (k.v) cudaFree(k.v);
    }
    for (void* m : peer_maps_) cudaIpcCloseMemHandle(m);
    for (auto& kv : gemm_plans_)
        for (GemmPlan* gp : kv.second) gemm_tc_plan_destroy(gp);
    void* frees[] = {kv16_, x16_, unscale_, tmp_a_, tmp_b_, gemm_status_, xflags_, bufs_, records_, consts_, att_scratch_.part, words_, rope_table_, argmax_val_, argmax_idx_, token_, out_tokens_, stage_};
    for (void* p : frees)
        if (p) cudaFree(p);
}

bool DecodePlanImpl::uses_weight(uint64_t h) const {
    for (uint64_t w : weight_handles_)
        if (w == h) return true;
    return h != 0 && h == gen_embed_;
}

int DecodePlanImpl::create(const b2_graph* g, const std::function<const WeightDev*(uint64_t)>& resolve, int sm_count, bool fast, int tokens,
                           bool prefill, DecodePlanImpl** out, std::string& err) {
    if (!g || !g->bufs || !g->ops || g->n_bufs == 0 || g->n_ops == 0 || !out) {
        err = "[b200qmm: decode_plan: empty graph]";
        return B2_ERR_ARG;
    }
    if (g->max_len == 0 || g->n_rope > 8 || (tokens > 0 && g->max_len < (uint32_t)tokens)) {
        err = "[b200qmm: decode_plan: max_len must be positive (and hold a whole step) and at most 8 RoPE tables are taken]";
        return B2_ERR_ARG;
    }
    if (tokens < 1 || tokens > (prefill ? 8192 : 4)) {
        err = prefill ? "[b200qmm: decode_plan: a prefill plan takes steps of 1 to 8192 tokens]" : "[b200qmm: decode_plan: a plan takes steps of 1 to 4 tokens]";
        return tokens >= 1 ? B2_DECLINED : B2_ERR_ARG;
    }
    if (prefill && g->n_logits) {
        err = "[b200qmm: decode_plan: a prefill plan ends at the hidden states (a graph without logits)]";
        return B2_DECLINED;
    }
    std::unique_ptr<DecodePlanImpl> p(new DecodePlanImpl());
    p->sm_count_ = sm_count;
    p->fast_ = fast;
    p->tokens_ = tokens;
    const size_t T = (size_t)tokens;
    if (const char* e = getenv("B2_PLAN_PDL")) p->pdl_ = atoi(e) != 0;
    if (const char* e = getenv("B2_PLAN_FUSE")) p->fuse_ = atoi(e) != 0;
    if (const char* e = getenv("B2_PLAN_DEFER_NORM")) p->defer_norm_ = atoi(e) != 0;
    int self_level = 2;  // which products split their vectors themselves: 0 none, 1 those behind a norm, 2 all
    if (const char* e = getenv("B2_PLAN_EPILOGUE")) self_level = atoi(e);
    if (const char* e = getenv("B2_PLAN_FUSE_ROPE")) p->fuse_rope_ = atoi(e) != 0;
    if (prefill) {  // the one-token kernels' fusions do not apply: the products are GEMMs
        p->prefill_ = true;
        p->defer_norm_ = p->fuse_rope_ = false;
        const char* e = getenv("B2_PREFILL_ATTEND");
        p->loop_attend_ = e && strcmp(e, "loop") == 0;
    }
    p->max_len_ = g->max_len;
    p->kv_f16_ = g->kv_f16 ? 1 : 0;

    // ---- activation buffers: one allocation, each buffer 256-byte aligned --------------------------
    size_t total = 0;
    std::vector<size_t> off(g->n_bufs);
    for (uint32_t i = 0; i < g->n_bufs; i++) {
        off[i] = total;
        total += align_up((size_t)g->bufs[i], 64);
    }
    total = std::max<size_t>(total, 64);
    p->block_floats_ = total;
    PLAN_CUDA(cudaMalloc((void**)&p->bufs_, T * total * sizeof(float)), "cudaMalloc(buffers)");
    PLAN_CUDA(cudaMemset(p->bufs_, 0, T * total * sizeof(float)), "cudaMemset(buffers)");
    for (uint32_t i = 0; i < g->n_bufs; i++) {
        p->buf_ptr_.push_back(p->bufs_ + off[i]);
        p->buf_len_.push_back((size_t)g->bufs[i]);
    }
    bool bad_view = false;
    auto view = [&](b2_view v, size_t n) -> float* {
        if (v.buf >= g->n_bufs || (size_t)v.off + n > p->buf_len_[v.buf]) {
            bad_view = true;
            return nullptr;
        }
        return p->buf_ptr_[v.buf] + v.off;
    };

    // ---- RoPE table layout ------------------------------------------------------------------------
    std::vector<uint32_t> cs_off(g->n_rope + 1, 0);
    for (uint32_t i = 0; i < g->n_rope; i++) cs_off[i + 1] = cs_off[i] + 2 * g->rope_halves[i];
    p->cs_stride_ = cs_off[g->n_rope];
    p->cs_off_ = cs_off;

    // ---- KV caches --------------------------------------------------------------------------------
    const size_t esz = p->kv_f16_ ? 2 : 4;
    size_t max_row = 0;
    for (uint32_t i = 0; i < g->n_kv; i++) {
        Kv k;
        k.nkv = g->kv_nkv[i];
        k.hd = g->kv_hd[i];
        size_t bytes = (size_t)k.nkv * g->max_len * k.hd * esz;
        PLAN_CUDA(cudaMalloc(&k.k, bytes), "cudaMalloc(K cache)");
        p->kv_.push_back(k);  // pushed before V so that a failure below still frees K
        PLAN_CUDA(cudaMalloc(&p->kv_.back().v, bytes), "cudaMalloc(V cache)");
        PLAN_CUDA(cudaMemset(p->kv_.back().k, 0, bytes), "cudaMemset(K cache)");
        PLAN_CUDA(cudaMemset(p->kv_.back().v, 0, bytes), "cudaMemset(V cache)");
        max_row = std::max(max_row, (size_t)k.nkv * k.hd);
    }

    // ---- norm weights: one device block -----------------------------------------------------------
    size_t n_consts = 0;
    for (uint32_t i = 0; i < g->n_ops; i++) {
        const b2_op& o = g->ops[i];
        if (o.kind == B2_OP_NORM && o.p0) n_consts += align_up(o.n, 64);
        if (o.kind == B2_OP_QK_ROPE) n_consts += (o.p0 ? align_up(o.hd, 64) : 0) + (o.p1 ? align_up(o.hd, 64) : 0);
    }
    PLAN_CUDA(cudaMalloc((void**)&p->consts_, std::max<size_t>(n_consts, 64) * sizeof(float)), "cudaMalloc(norm weights)");
    size_t consts_at = 0;
    auto put_const = [&](const float* host, size_t n, const float** dev) -> cudaError_t {
        float* d = p->consts_ + consts_at;
        consts_at += align_up(n, 64);
        *dev = d;
        return cudaMemcpy(d, host, n * sizeof(float), cudaMemcpyHostToDevice);
    };

    // ---- ops -------------------------------------------------------------------------------------
    // Records of vectors. key = (buffer, offset, length, form); `valid` = the region that holds the record of the current contents.
    using Key = std::tuple<uint32_t, uint32_t, uint32_t, bool>;
    std::map<Key, size_t> valid;
    std::vector<std::pair<size_t, bool>> regions;  // length and form
    auto touch = [&](uint32_t buf) {  // a write into `buf`: records of its vectors are stale
        for (auto it = valid.begin(); it != valid.end();) it = std::get<0>(it->first) == buf ? valid.erase(it) : std::next(it);
    };

    for (uint32_t i = 0; i < g->n_ops; i++) {
        const b2_op& o = g->ops[i];
        Op op;
        op.kind = o.kind;
        switch (o.kind) {
            case B2_OP_NORM: {
                if (o.n == 0 || o.rows == 0) {
                    err = "[b200qmm: decode_plan: norm of nothing]";
                    return B2_ERR_ARG;
                }
                size_t xs = o.x_stride ? o.x_stride : o.n, os = o.out_stride ? o.out_stride : o.n;
                op.x = view(o.x, (size_t)(o.rows - 1) * xs + o.n);
                op.y = view(o.y, (size_t)(o.rows - 1) * os + o.n);
                op.norm = DecNorm{o.n, (uint32_t)xs, (uint32_t)os, o.add ? 1u : 0u, o.pre == 0.0f ? 1.0f : o.pre, o.eps};
                op.rows = o.rows;
                if (o.p0) PLAN_CUDA(put_const(o.p0, o.n, &op.p0), "cudaMemcpy(norm weights)");
                touch(o.y.buf);
                break;
            }
            case B2_OP_LINEAR: {
                const WeightDev* w = resolve(o.w);
                if (!w) {
                    err = "[b200qmm: decode_plan: unknown weight handle]";
                    return B2_ERR_ARG;
                }
                if (w->n_out != o.n_out || w->n_in != o.n_in) {
                    err = fmt("[b200qmm: decode_plan: linear %u x %u does not match its weight %zu x %zu]", o.n_out, o.n_in, w->n_out, w->n_in);
                    return B2_ERR_ARG;
                }
                if (!prefill && !gemv_supports(*w)) {
                    err = "[b200qmm: decode_plan: a weight's shape is outside the matrix-vector kernels]";
                    return B2_DECLINED;
                }
                if (prefill && (!gemm_tc_supports(*w, (size_t)tokens) || o.mode == B2_MODE_ADD_GATED || o.n_out % 4)) {
                    err = "[b200qmm: decode_plan: a prefill plan takes products with a tensor-core kernel (Q4_K, MLX-4, Q6_K, Q8_0, FP8), rows in multiples of 4, "
                          "and no gated mode]";
                    return B2_DECLINED;
                }
                op.w = *w;
                p->weight_handles_.push_back(o.w);
                op.mode = (int)o.mode;
                if (o.mode > B2_MODE_ADD_GATED) {
                    err = "[b200qmm: decode_plan: bad linear mode]";
                    return B2_ERR_ARG;
                }
                op.pair = o.mode == B2_MODE_SILU_PAIR || o.mode == B2_MODE_GELU_PAIR;
                if (op.pair) {
                    const WeightDev* u = resolve(o.w2);
                    if (!u) {
                        err = "[b200qmm: decode_plan: a pair needs its second matrix]";
                        return B2_ERR_ARG;
                    }
                    if (u->fmt != w->fmt || u->n_in != w->n_in || u->n_out != w->n_out) {
                        err = "[b200qmm: decode_plan: the pair's matrices differ in shape or format]";
                        return B2_DECLINED;
                    }
                    op.w2 = *u;
                    p->weight_handles_.push_back(o.w2);
                }
                op.x = view(o.x, o.n_in);
                op.y = view(o.y, o.n_out);
                if (o.mode == B2_MODE_ADD_GATED) op.z = view(o.z, 1);
                // Products of the same vector that store into consecutive ranges (q, k, v) run as one launch over
                // a row-wise concatenation of their matrices (a device copy the plan owns).
                if (p->fuse_ && o.mode == B2_MODE_STORE && fusable(*w)) {
                    std::vector<const WeightDev*> parts{w};
                    uint32_t end = o.y.off + o.n_out, j = i + 1;
                    for (; j < g->n_ops; j++) {
                        const b2_op& n = g->ops[j];
                        if (n.kind != B2_OP_LINEAR || n.mode != B2_MODE_STORE || n.x.buf != o.x.buf || n.x.off != o.x.off || n.n_in != o.n_in ||
                            n.y.buf != o.y.buf || n.y.off != end || n.y.buf == n.x.buf)
                            break;
                        const WeightDev* nw = resolve(n.w);
                        if (!nw || nw->fmt != w->fmt || nw->n_in != w->n_in || nw->n_out != n.n_out || nw->group != w->group || !fusable(*nw) ||
                            nw->bs_rows != w->bs_rows || nw->bs_cols != w->bs_cols || nw->bs_ncb != w->bs_ncb || !nw->p1 != !w->p1)
                            break;
                        parts.push_back(nw);
                        p->weight_handles_.push_back(n.w);
                        end += n.n_out;
                    }
                    if (parts.size() > 1) {
                        PLAN_CUDA(fuse_rows(parts, &op.w, p->fused_), "fusing matrices of one vector");
                        op.y = view(o.y, end - o.y.off);
                        i = j - 1;  // the fused ops are done
                    }
                }
                if (!prefill && gemv_mma_supports(op.w)) {
                    const bool halves = gemv_mma_halves(op.w);
                    auto [v, fresh] = valid.try_emplace(Key{o.x.buf, o.x.off, o.n_in, halves}, regions.size());
                    if (fresh) {
                        Op sp;
                        sp.kind = OP_SPLIT;
                        sp.x = sp.sx = op.x;
                        sp.n = o.n_in;
                        sp.halves = halves;
                        sp.region = (int)regions.size();
                        regions.push_back({o.n_in, halves});
                        p->ops_.push_back(sp);
                    }
                    op.region = (int)v->second;
                    op.sx = op.x;
                    op.halves = halves;
                }
                if (o.y.buf == o.x.buf && !(o.y.off + o.n_out <= o.x.off || o.x.off + o.n_in <= o.y.off)) {
                    err = "[b200qmm: decode_plan: a linear op writes over its own input]";
                    return B2_ERR_ARG;
                }
                touch(o.y.buf);
                break;
            }
            case B2_OP_QK_ROPE: {
                if (o.kv >= g->n_kv || o.rope >= g->n_rope || g->kv_nkv[o.kv] != o.nkv || g->kv_hd[o.kv] != o.hd || o.hd > 256 || o.hd % 32 ||
                    g->rope_halves[o.rope] != o.half_rot || 2 * o.half_rot > o.hd) {
                    err = "[b200qmm: decode_plan: qk_rope does not match its KV cache or RoPE table]";
                    return B2_ERR_ARG;
                }
                size_t q_stride = o.q_stride ? o.q_stride : o.hd;
                size_t need = std::max({(size_t)(o.nh - 1) * q_stride + o.hd, (size_t)o.k_off + (size_t)o.nkv * o.hd,
                                        o.v_from_k ? (size_t)0 : (size_t)o.v_off + (size_t)o.nkv * o.hd});
                op.x = view(o.x, need);
                op.y = view(o.y, (size_t)o.nh * o.hd);
                op.kv = o.kv;
                op.rope = DecRope{o.nh, o.nkv, o.hd, o.half_rot, (uint32_t)q_stride, o.k_off, o.v_off, o.interleaved, o.v_norm, o.v_from_k,
                                  g->max_len, p->cs_stride_, cs_off[o.rope], o.eps};
                if (o.p0) PLAN_CUDA(put_const(o.p0, o.hd, &op.p0), "cudaMemcpy(q norm)");
                if (o.p1) PLAN_CUDA(put_const(o.p1, o.hd, &op.p1), "cudaMemcpy(k norm)");
                touch(o.y.buf);
                break;
            }
            case B2_OP_ATTEND: {
                if (o.kv >= g->n_kv || g->kv_nkv[o.kv] != o.nkv || g->kv_hd[o.kv] != o.hd) {
                    err = "[b200qmm: decode_plan: attend does not match its KV cache]";
                    return B2_ERR_ARG;
                }
                if (prefill && !attend_rows_supports(o.nh, o.nkv, o.hd)) {
                    err = "[b200qmm: decode_plan: prefill attention takes head dimensions 64 and 128]";
                    return B2_DECLINED;
                }
                if ((!prefill || p->loop_attend_) && !attend_supports(o.nh, o.nkv, o.hd)) {
                    err = fmt("[b200qmm: decode_plan: attention with %u heads over %u KV heads of %u is outside the kernel (head dim 64 / 128, "
                              "1 / 2 / 4 / 8 heads per KV head)]", o.nh, o.nkv, o.hd);
                    return B2_DECLINED;
                }
                op.x = view(o.x, (size_t)o.nh * o.hd);
                op.y = view(o.y, (size_t)o.nh * o.hd);
                op.kv = o.kv;
                op.attn = DecAttn{o.nh, o.nkv, o.hd, g->max_len, o.window, o.scale};
                touch(o.y.buf);
                break;
            }
            case B2_OP_GLU: {
                op.x = view(o.x, o.n);
                op.z = view(o.z, o.n);
                op.y = view(o.y, o.n);
                op.n = o.n;
                op.gelu = o.gelu ? 1 : 0;
                touch(o.y.buf);
                break;
            }
            case B2_OP_EXCHANGE: {
                if (tokens > 1) {
                    err = "[b200qmm: decode_plan: a tensor-parallel graph runs one token per step]";
                    return B2_DECLINED;
                }
                if (o.n == 0 || o.n % 32) {
                    err = "[b200qmm: decode_plan: an exchanged vector must be a positive multiple of 32 values]";
                    return B2_ERR_ARG;
                }
                op.x = view(o.x, o.n);
                op.n = o.n;
                if (op.x) op.off = (size_t)(op.x - p->bufs_);
                p->has_exchange_ = true;
                touch(o.x.buf);
                break;
            }
            default:
                err = fmt("[b200qmm: decode_plan: op kind %u is not taken by this backend]", o.kind);
                return B2_DECLINED;
        }
        if (bad_view) {
            err = fmt("[b200qmm: decode_plan: op %u reaches outside its buffer]", i);
            return B2_ERR_ARG;
        }
        p->ops_.push_back(op);
    }
    p->n_input_ = g->n_input;
    p->n_hidden_ = g->n_hidden;
    p->n_logits_ = g->n_logits;
    p->input_ = view(g->input, g->n_input);
    p->hidden_ = view(g->hidden, g->n_hidden);
    if (g->n_logits) p->logits_ = view(g->logits, g->n_logits);
    if (bad_view) {
        err = "[b200qmm: decode_plan: input / hidden / logits reach outside their buffers]";
        return B2_ERR_ARG;
    }

    // What an op reads and writes, as far as the passes below need it (they treat attention and RoPE as touching their whole views).
    auto reads = [&](const Op& o, const float* v, size_t n) {
        switch (o.kind) {
            case B2_OP_LINEAR:
                return (o.region < 0 && overlaps_f(v, n, o.x, o.w.n_in)) || (o.mode == B2_MODE_ADD_GATED && overlaps_f(v, n, o.z, 1)) ||
                       ((o.mode == B2_MODE_ADD || o.mode == B2_MODE_ADD_GATED) && overlaps_f(v, n, o.y, o.w.n_out));
            case OP_SPLIT: return overlaps_f(v, n, o.sx, o.n);
            case B2_OP_NORM:
                return overlaps_f(v, n, o.x, (size_t)(o.rows - 1) * o.norm.x_stride + o.norm.n) ||
                       (o.norm.add && overlaps_f(v, n, o.y, (size_t)(o.rows - 1) * o.norm.out_stride + o.norm.n));
            case B2_OP_EXCHANGE: return overlaps_f(v, n, o.x, o.n);
            case B2_OP_GLU: return overlaps_f(v, n, o.x, o.n) || overlaps_f(v, n, o.z, o.n);
            default: return overlaps_f(v, n, o.x, n) || overlaps_f(v, n, o.y, n) || overlaps_f(o.x, 1, v, n);
        }
    };
    auto writes = [&](const Op& o, const float* v, size_t n) {
        switch (o.kind) {
            case B2_OP_LINEAR: return overlaps_f(v, n, o.y, o.w.n_out);
            case OP_SPLIT: return false;
            case B2_OP_NORM: return overlaps_f(v, n, o.y, (size_t)(o.rows - 1) * o.norm.out_stride + o.norm.n);
            case B2_OP_EXCHANGE: return overlaps_f(v, n, o.x, o.n);
            case B2_OP_GLU: return overlaps_f(v, n, o.y, o.n);
            case B2_OP_ATTEND: return overlaps_f(v, n, o.y, (size_t)o.attn.nh * o.attn.hd);
            default: return overlaps_f(v, n, o.y, (size_t)o.rope.nh * o.rope.hd);
        }
    };
    // whether an op writes all of v
    auto covers = [&](const Op& o, const float* v, size_t n) {
        const float* y = o.kind == B2_OP_EXCHANGE ? nullptr : o.y;
        const size_t len = o.kind == B2_OP_LINEAR ? o.w.n_out : o.kind == B2_OP_NORM ? (o.rows == 1 ? o.norm.n : 0) : o.kind == B2_OP_GLU ? o.n : 0;
        return y && y <= v && v + n <= y + len;
    };
    // Whether anything from op b on reads v before it is written anew, a step following on a step, up to op a.
    auto read_later = [&](size_t b, size_t a, const float* v, size_t n) {
        for (size_t c = b; c != a; c = c + 1 < p->ops_.size() ? c + 1 : 0) {
            const Op& o = p->ops_[c];
            const size_t rope = o.kind == B2_OP_QK_ROPE ? std::max({(size_t)(o.rope.nh - 1) * o.rope.q_stride + o.rope.hd, (size_t)o.rope.k_off + (size_t)o.rope.nkv * o.rope.hd,
                                                                    (size_t)o.rope.v_off + (size_t)o.rope.nkv * o.rope.hd})
                                                        : 0;
            const bool reading = o.kind == B2_OP_QK_ROPE  ? overlaps_f(v, n, o.x, rope)
                                 : o.kind == B2_OP_ATTEND ? overlaps_f(v, n, o.x, (size_t)o.attn.nh * o.attn.hd)
                                                          : reads(o, v, n);
            if (reading) return true;
            if (covers(o, v, n)) return false;
        }
        return false;
    };
    // ---- norms whose output only splits read become part of the split: x times the weights is split, and the products multiply their
    // results by the factor (nothing has to wait for the whole row first, and the norm is not launched) ----
    if (p->defer_norm_) {
        for (size_t a = 0; a < p->ops_.size(); a++) {
            const Op nrm = p->ops_[a];
            if (nrm.kind != B2_OP_NORM || nrm.rows != 1 || nrm.norm.add || nrm.norm.n % 4) continue;
            const float* y = nrm.y;
            const size_t n = nrm.norm.n;
            if (overlaps_f(y, n, p->hidden_, p->n_hidden_) || overlaps_f(y, n, p->logits_, p->n_logits_) || overlaps_f(y, n, p->input_, p->n_input_)) continue;
            bool ok = true, stale = false;
            std::vector<size_t> users;
            for (size_t b = a + 1; b < p->ops_.size() && ok; b++) {
                const Op& o = p->ops_[b];
                if (o.kind == OP_SPLIT && o.sx == y && o.n == n && !o.normed && !stale) users.push_back(b);
                else if (reads(o, y, n)) ok = false;
                if (covers(o, y, n)) break;
                if (writes(o, y, n)) ok = false;  // a part of it: what the rest holds would have to be known
                stale = stale || writes(o, nrm.x, n);  // a split behind this point would read another x
            }
            if (!ok || users.empty()) continue;
            for (size_t b : users) {
                Op& s = p->ops_[b];
                s.sx = nrm.x;
                s.nw = nrm.p0;
                s.npre = nrm.norm.pre;
                s.neps = nrm.norm.eps;
                s.normed = 1;
            }
            p->ops_.erase(p->ops_.begin() + (ptrdiff_t)a);
            a--;
        }
    }
    // ---- products that split their vector themselves: every product of the record must find the vector unchanged, and none may
    // write over it (its CTAs read the vector at different times) ----
    for (size_t a = 0; a < p->ops_.size(); a++) {
        Op& s = p->ops_[a];
        if (s.kind != OP_SPLIT) continue;
        bool ok = self_level >= (s.normed ? 1 : 2);
        std::vector<size_t> users;
        bool stale = false;
        for (size_t b = a + 1; b < p->ops_.size(); b++) {
            Op& o = p->ops_[b];
            const bool user = o.kind == B2_OP_LINEAR && o.region == s.region;
            if (user) {
                users.push_back(b);
                if (stale || writes(o, s.sx, s.n)) ok = false;
            }
            stale = stale || writes(o, s.sx, s.n);
        }
        s.self = ok;
        s.parts = ok;
        for (size_t b : users) s.parts = s.parts && gemv_tc_supports(p->ops_[b].w);
        for (size_t b : users) {
            Op& o = p->ops_[b];
            o.parts = s.parts;
            o.sx = s.sx;
            o.nw = s.nw;
            o.npre = s.npre;
            o.neps = s.neps;
            o.normed = s.normed;
            o.self = s.self;
        }
    }
    // ---- records ---------------------------------------------------------------------------------
    size_t rec_total = 0;
    std::vector<size_t> region_at;
    for (auto& [n, halves] : regions) {
        region_at.push_back(rec_total);
        rec_total += align_up(split_bytes_of(n, halves), 256);
    }
    rec_total = std::max<size_t>(rec_total, 256);
    p->rec_block_ = rec_total;
    PLAN_CUDA(cudaMalloc((void**)&p->records_, T * rec_total), "cudaMalloc(records)");
    for (Op& o : p->ops_)
        if (o.region >= 0) o.rec_at = region_at[(size_t)o.region];

    // ---- RoPE inside the attention kernel ----------------------------------------------------------------------
    // A QK_ROPE op without per-head norms whose rotated queries only the ATTEND op right behind it reads: the attention
    // kernel rotates the queries as it stages them and the unit that holds the newest keys appends the token's key and
    // value (FusedRope); one launch fewer per layer.
    if (p->fuse_rope_) {
        std::vector<Op> kept;
        kept.reserve(p->ops_.size());
        for (size_t b = 0; b < p->ops_.size(); b++) {
            Op& at = p->ops_[b];
            Op* rp = kept.empty() ? nullptr : &kept.back();
            if (at.kind == B2_OP_ATTEND && rp && rp->kind == B2_OP_QK_ROPE && !rp->p0 && !rp->p1 && !rp->rope.v_norm && !rp->rope.v_from_k &&
                rp->kv == at.kv && rp->y == at.x && rp->rope.nh == at.attn.nh && rp->rope.nkv == at.attn.nkv && rp->rope.hd == at.attn.hd &&
                rp->rope.hd <= (uint32_t)ATT_THREADS_HOST) {
                // nobody else may read the rotated queries: they are not written any more
                bool other_reader = overlaps_f(rp->y, (size_t)rp->rope.nh * rp->rope.hd, p->hidden_, p->n_hidden_) ||
                                    overlaps_f(rp->y, (size_t)rp->rope.nh * rp->rope.hd, p->logits_, p->n_logits_);
                for (size_t c = 0; c < p->ops_.size() && !other_reader; c++) {
                    if (c == b || &p->ops_[c] == &at) continue;
                    const Op& o = p->ops_[c];
                    if (o.kind == B2_OP_QK_ROPE) continue;  // writes it
                    const float* q0 = rp->y;
                    const size_t qn = (size_t)rp->rope.nh * rp->rope.hd;
                    const size_t xn = o.kind == B2_OP_LINEAR ? o.w.n_in : o.kind == B2_OP_ATTEND ? (size_t)o.attn.nh * o.attn.hd
                                      : o.kind == B2_OP_NORM ? (size_t)(o.rows - 1) * o.norm.x_stride + o.norm.n : o.n;
                    if (o.kind == B2_OP_ATTEND && o.x == q0) continue;  // another layer's attention over its own fused queries
                    if (overlaps_f(q0, qn, o.x, xn) || overlaps_f(q0, qn, o.z, o.n ? o.n : 1) || overlaps_f(q0, qn, o.sx, xn)) other_reader = true;
                }
                if (!other_reader) {
                    at.fr = FusedRope{rp->x, nullptr, rp->rope};  // the table's address is known at launch
                    kept.back() = at;
                    continue;
                }
            }
            kept.push_back(at);
        }
        p->ops_ = std::move(kept);
    }

    // ---- scratch ------------------------------------------------------------------------------------
    size_t part_floats = 0, count_words = 0;
    for (const Op& o : p->ops_) {
        if (o.kind != B2_OP_ATTEND || (prefill && !p->loop_attend_)) continue;
        const uint32_t tokens = prefill ? 1 : (uint32_t)T;
        part_floats = std::max(part_floats, attend_part_floats(o.attn.nh, o.attn.nkv, o.attn.hd, o.attn.max_len, tokens));
        count_words = std::max(count_words, attend_count_words(o.attn.nh, o.attn.nkv, o.attn.max_len, tokens));
    }
    if (part_floats) PLAN_CUDA(cudaMalloc((void**)&p->att_scratch_.part, part_floats * sizeof(float)), "cudaMalloc(attention shares)");
    const size_t n_words = 8 + 4 * T + count_words;
    PLAN_CUDA(cudaMalloc((void**)&p->words_, n_words * 4), "cudaMalloc(step words)");
    PLAN_CUDA(cudaMemset(p->words_, 0, n_words * 4), "cudaMemset(step words)");
    if (p->has_exchange_) {
        PLAN_CUDA(cudaMalloc((void**)&p->xflags_, 32 * 4), "cudaMalloc(exchange flags)");
        PLAN_CUDA(cudaMemset(p->xflags_, 0, 32 * 4), "cudaMemset(exchange flags)");
    }
    p->sp_ = p->words_;
    p->status_ = p->words_ + 4;
    p->argmax_counter_ = p->words_ + 5;
    p->sp_multi_ = p->words_ + 8;
    p->att_scratch_.counts = p->words_ + 8 + 4 * T;
    size_t table = (size_t)std::max<uint32_t>(p->cs_stride_, 1) * g->max_len;
    PLAN_CUDA(cudaMalloc((void**)&p->rope_table_, table * sizeof(float)), "cudaMalloc(rope table)");
    PLAN_CUDA(cudaMemset(p->rope_table_, 0, table * sizeof(float)), "cudaMemset(rope table)");
    const size_t n_partials = std::max(128, sm_count);  // one per CTA of the argmax kernel
    PLAN_CUDA(cudaMalloc((void**)&p->argmax_val_, n_partials * sizeof(float)), "cudaMalloc(argmax)");
    PLAN_CUDA(cudaMalloc((void**)&p->argmax_idx_, n_partials * sizeof(int)), "cudaMalloc(argmax)");
    PLAN_CUDA(cudaMalloc((void**)&p->token_, sizeof(int)), "cudaMalloc(token)");
    PLAN_CUDA(cudaMalloc((void**)&p->out_tokens_, (size_t)g->max_len * sizeof(int)), "cudaMalloc(tokens)");
    p->stage_floats_ = std::max<size_t>(max_row, 1) * 256;
    PLAN_CUDA(cudaMalloc((void**)&p->stage_, 2 * p->stage_floats_ * sizeof(float)), "cudaMalloc(KV staging)");
    PLAN_CUDA(cudaStreamCreateWithFlags(&p->cap_stream_, cudaStreamNonBlocking), "cudaStreamCreate");
    PLAN_CUDA(cudaEventCreate(&p->ev0_), "cudaEventCreate");
    PLAN_CUDA(cudaEventCreate(&p->ev1_), "cudaEventCreate");

    if (prefill) {
        for (size_t a = 0; a + 1 < p->ops_.size(); a++) {
            Op& o = p->ops_[a];
            if (!(o.kind == B2_OP_NORM && o.rows == 1 && !o.norm.add) && !(o.kind == B2_OP_LINEAR && o.pair)) continue;
            const size_t n = o.kind == B2_OP_NORM ? o.norm.n : o.w.n_out;
            size_t b = a + 1;
            while (b < p->ops_.size() && p->ops_[b].kind == B2_OP_LINEAR && p->ops_[b].x == o.y && p->ops_[b].w.n_in == n && !writes(p->ops_[b], o.y, n))
                if (p->ops_[b++].pair) break;  // (its own result may take the f16 rows' place)
            o.x16_only = b > a + 1 && b < p->ops_.size() && !overlaps_f(o.y, n, p->hidden_, p->n_hidden_) && !overlaps_f(o.y, n, p->input_, p->n_input_) &&
                         !read_later(b, a, o.y, n);
        }
        size_t max_k = 64, max_n = 64;
        for (const Op& o : p->ops_)
            if (o.kind == B2_OP_LINEAR) {
                max_k = std::max(max_k, o.w.n_in);
                max_n = std::max(max_n, o.w.n_out);
            }
        PLAN_CUDA(cudaMalloc(&p->x16_, T * max_k * 2), "cudaMalloc(f16 activations)");
        PLAN_CUDA(cudaMalloc((void**)&p->unscale_, T * sizeof(float)), "cudaMalloc(row factors)");
        PLAN_CUDA(cudaMalloc((void**)&p->tmp_a_, T * max_n * sizeof(float)), "cudaMalloc(products)");
        PLAN_CUDA(cudaMalloc((void**)&p->tmp_b_, T * max_n * sizeof(float)), "cudaMalloc(products)");
        size_t kv16 = 0;
        for (const Kv& k : p->kv_) kv16 = std::max(kv16, attend_rows_scratch_bytes(k.nkv, g->max_len, k.hd, p->kv_f16_));
        if (kv16) PLAN_CUDA(cudaMalloc(&p->kv16_, kv16), "cudaMalloc(f16 cache rows)");
        PLAN_CUDA(cudaMalloc((void**)&p->gemm_status_, sizeof(GemmStatus)), "cudaMalloc(GEMM status)");
        PLAN_CUDA(cudaMemset(p->gemm_status_, 0, sizeof(GemmStatus)), "cudaMemset(GEMM status)");
        *out = p.release();  // nothing is captured: a step launches its kernels (a few per op, whatever the token count)
        return B2_OK;
    }
    // One eager pass (loads every kernel outside a capture, and surfaces launch errors with their op),
    // then the step graph.
    PLAN_CUDA(launch_set_step(p->sp_, 0, 0, 0, nullptr, 0, p->cap_stream_), "set_step");
    int rc = p->run_ops(p->cap_stream_, err, false, false);
    if (rc) return rc;
    PLAN_CUDA(cudaStreamSynchronize(p->cap_stream_), "first pass");
    rc = p->check_status(err);
    if (rc) return rc;
    rc = p->capture(p->cap_stream_, false, &p->step_exec_, err);
    if (rc) return rc;
    // Steps of several tokens: the same eager pass and a graph per token count.
    for (int nt = 2; nt <= tokens; nt++) {
        uint32_t words[16] = {};
        for (int tk = 0; tk < nt; tk++) words[4 * tk] = (uint32_t)tk;
        PLAN_CUDA(cudaMemcpyAsync(p->sp_multi_, words, 16 * nt, cudaMemcpyHostToDevice, p->cap_stream_), "cudaMemcpy(step words)");
        rc = p->run_ops_multi(p->cap_stream_, nt, err, false);
        if (rc) return rc;
        PLAN_CUDA(cudaStreamSynchronize(p->cap_stream_), "first pass (several tokens)");
        rc = p->check_status(err);
        if (rc) return rc;
        rc = p->capture(p->cap_stream_, false, &p->multi_exec_[nt], err, nt);
        if (rc) return rc;
    }
    *out = p.release();
    return B2_OK;
}

GemvIn DecodePlanImpl::product_in(const Op& o, bool self) const {
    GemvIn in;
    if (self) {
        in.x = o.sx;
        in.x_stride = block_floats_;
        in.norm_w = o.nw;
        in.pre = o.npre;
    } else {
        in.rec = records_ + o.rec_at;
        in.rec_stride = rec_block_;
    }
    in.norm = o.normed;
    in.eps = o.neps;
    in.fast = fast_;
    in.status = status_;
    return in;
}

// `chained`: every launch but the first (`first_chained`: the first too) carries the programmatic-dependent-launch
// attribute, so each kernel starts (and fetches its first weights) while the one before it drains.
int DecodePlanImpl::run_ops(cudaStream_t st, std::string& err, bool chained, bool first_chained) {
    launches_ = 0;
    for (size_t i = 0; i < ops_.size(); i++) {
        const Op& o = ops_[i];
        if (o.kind == OP_SPLIT && o.self) continue;
        const bool pdl = chained && (launches_ > 0 || first_chained);
        launches_++;
        cudaError_t e = cudaSuccess;
        switch (o.kind) {
            case B2_OP_NORM: e = launch_norm(o.x, o.y, o.p0, o.norm, o.rows, st, pdl); break;
            case OP_SPLIT: e = launch_split(o.sx, 0, o.nw, o.npre, o.n, 1, records_ + o.rec_at, 0, o.halves, fast_, st, pdl); break;
            case B2_OP_LINEAR:
                e = o.region >= 0 ? launch_gemv_mma(o.w, o.pair ? &o.w2 : nullptr, product_in(o, o.self), 1, o.y, 0, o.mode, o.z, 0, sm_count_, st, pdl)
                                  : launch_gemv_f8_float(o.w, o.pair ? &o.w2 : nullptr, o.x, o.y, o.mode, o.z, sm_count_, st, pdl);
                break;
            case B2_OP_QK_ROPE:
                e = launch_qk_rope(o.x, o.y, kv_[o.kv].k, kv_[o.kv].v, kv_f16_, o.p0, o.p1, rope_table_, sp_, o.rope, st, pdl);
                break;
            case B2_OP_ATTEND:
                if (o.fr.qkv) {
                    FusedRope fr = o.fr;
                    fr.cs_table = rope_table_;
                    e = launch_attend(o.x, kv_[o.kv].k, kv_[o.kv].v, kv_f16_, o.y, sp_, o.attn, status_, att_scratch_, st, pdl, &fr);
                } else {
                    e = launch_attend(o.x, kv_[o.kv].k, kv_[o.kv].v, kv_f16_, o.y, sp_, o.attn, status_, att_scratch_, st, pdl);
                }
                break;
            case B2_OP_GLU: e = launch_glu(o.x, o.z, o.y, o.n, o.gelu, st, pdl); break;
            case B2_OP_EXCHANGE:
                if (attached_) e = launch_exchange(peers_, o.off, o.n, xflags_, status_, st, pdl, o.meet_first);  // the first pass of a lone rank has nobody to meet
                break;
            default: e = cudaErrorInvalidValue;
        }
        if (e != cudaSuccess) {
            err = fmt("[b200qmm: plan: op %zu (kind %u): %s]", i, o.kind, cudaGetErrorString(e));
            return B2_ERR_CUDA;
        }
    }
    return B2_OK;
}

// The ops for nt tokens at once, op by op: a product reads its weights once for all tokens (each token's sums are its one-token sums),
// every other op runs once per token on that token's blocks (activations, records, step words) or has the token as a grid dimension.
int DecodePlanImpl::run_ops_multi(cudaStream_t st, int nt, std::string& err, bool chained) {
    auto A = [&](const float* p, int tk) -> float* { return p ? const_cast<float*>(p) + (size_t)tk * block_floats_ : nullptr; };
    bool first = true;
    uint64_t count = 0;
    auto pdl = [&]() {
        const bool v = chained && !first;
        first = false;
        count++;
        return v;
    };
    // A vector's record is made in a launch of its own where the products' CTAs would split all of it, more than `self_blocks` blocks of 256
    // values per warp.
    constexpr size_t self_blocks = 2;
    auto self = [&](const Op& o, size_t n) { return o.parts || (o.self && split_blocks_of(n) * (size_t)nt <= 16 * self_blocks); };
    for (size_t i = 0; i < ops_.size(); i++) {
        const Op& o = ops_[i];
        cudaError_t e = cudaSuccess;
        switch (o.kind) {
            case B2_OP_NORM:
                if (o.rows == 1) {  // all tokens in one launch: a CTA per row either way
                    DecNorm n = o.norm;
                    n.x_stride = n.out_stride = (uint32_t)block_floats_;
                    e = launch_norm(o.x, o.y, o.p0, n, (uint32_t)nt, st, pdl());
                    break;
                }
                for (int tk = 0; tk < nt && e == cudaSuccess; tk++) e = launch_norm(A(o.x, tk), A(o.y, tk), o.p0, o.norm, o.rows, st, pdl());
                break;
            case OP_SPLIT:
                if (!self(o, o.n)) e = launch_split(o.sx, block_floats_, o.nw, o.npre, o.n, nt, records_ + o.rec_at, rec_block_, o.halves, fast_, st, pdl());
                break;
            case B2_OP_LINEAR:
                if (o.region >= 0) {
                    e = launch_gemv_mma(o.w, o.pair ? &o.w2 : nullptr, product_in(o, self(o, o.w.n_in)), nt, o.y, block_floats_, o.mode, o.z, block_floats_, sm_count_,
                                        st, pdl());
                    break;
                }
                for (int tk = 0; tk < nt && e == cudaSuccess; tk++)
                    e = launch_gemv_f8_float(o.w, o.pair ? &o.w2 : nullptr, A(o.x, tk), A(o.y, tk), o.mode, A(o.z, tk), sm_count_, st, pdl());
                break;
            case B2_OP_QK_ROPE:  // all tokens in one launch (the one-token arithmetic per head)
                e = launch_qk_rope_rows(o.x, o.y, block_floats_, (uint32_t)nt, kv_[o.kv].k, kv_[o.kv].v, kv_f16_, o.p0, o.p1, rope_table_, sp_multi_, o.rope,
                                        st);
                first = false;
                count++;
                break;
            case B2_OP_ATTEND: {
                // One launch attends for all tokens, and rotates and appends where the one-token plan's does. Otherwise it is an
                // ordinary launch: all tokens' rows of the caches come from the launch just ahead of it.
                const AttnTokens at{nt, block_floats_};
                FusedRope fr = o.fr;
                fr.cs_table = rope_table_;
                const bool dependent = pdl();
                e = launch_attend(o.x, kv_[o.kv].k, kv_[o.kv].v, kv_f16_, o.y, sp_multi_, o.attn, status_, att_scratch_, st, dependent && o.fr.qkv, o.fr.qkv ? &fr : nullptr,
                                  &at);
                break;
            }
            case B2_OP_GLU:
                for (int tk = 0; tk < nt && e == cudaSuccess; tk++) e = launch_glu(A(o.x, tk), A(o.z, tk), A(o.y, tk), o.n, o.gelu, st, pdl());
                break;
            default: e = cudaErrorInvalidValue;
        }
        if (e != cudaSuccess) {
            err = fmt("[b200qmm: plan: op %zu (kind %u) for %d tokens: %s]", i, o.kind, nt, cudaGetErrorString(e));
            return B2_ERR_CUDA;
        }
    }
    multi_launches_[nt] = count;
    return B2_OK;
}

// Captures [embedding lookup,] ops [, argmax + advance] on `st` (not the legacy stream) into an executable graph.
int DecodePlanImpl::capture(cudaStream_t st, bool with_head, cudaGraphExec_t* out, std::string& err, int nt) {
    PLAN_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal), "cudaStreamBeginCapture");
    int rc = B2_OK;
    cudaError_t e = cudaSuccess;
    if (with_head) e = launch_dequantize(gen_embed_dev_, 0, 1, input_, st, token_);
    if (e == cudaSuccess) rc = nt > 1 ? run_ops_multi(st, nt, err, pdl_) : run_ops(st, err, pdl_, with_head);
    if (e == cudaSuccess && rc == B2_OK && with_head)
        e = launch_argmax(logits_, n_logits_, argmax_val_, argmax_idx_, argmax_counter_, token_, out_tokens_, sp_, st, pdl_);
    cudaGraph_t graph = nullptr;
    cudaError_t e2 = cudaStreamEndCapture(st, &graph);
    if (rc) {
        if (graph) cudaGraphDestroy(graph);
        return rc;
    }
    if (e != cudaSuccess || e2 != cudaSuccess) {
        if (graph) cudaGraphDestroy(graph);
        err = fmt("[b200qmm: plan: capture: %s]", cudaGetErrorString(e != cudaSuccess ? e : e2));
        return B2_ERR_CUDA;
    }
    e = cudaGraphInstantiate(out, graph, 0);
    cudaGraphDestroy(graph);
    PLAN_CUDA(e, "cudaGraphInstantiate");
    return B2_OK;
}

int DecodePlanImpl::inject_timeout(std::string& err) {
    const uint32_t s = 2;
    PLAN_CUDA(cudaMemcpy(status_, &s, 4, cudaMemcpyHostToDevice), "cudaMemcpy(status)");
    return B2_OK;
}

int DecodePlanImpl::check_status(std::string& err) {
    uint32_t s = 0;
    PLAN_CUDA(cudaMemcpy(&s, status_, 4, cudaMemcpyDeviceToHost), "cudaMemcpy(status)");
    if (s) {
        cudaMemset(status_, 0, 4);
        err = s == 4 ? "[b200qmm: plan: a peer did not arrive at an exchange within the time limit]"
              : s == 2 ? "[b200qmm: plan: a product's wait ran into the time limit]"
                     : "[b200qmm: plan: an attention kernel's wait on its copy ran into the time limit]";
        return B2_ERR_TIMEOUT;
    }
    return B2_OK;
}

int DecodePlanImpl::step(cudaStream_t st, size_t pos, const float* x, const float* rope_cs, float* hidden, float* logits, std::string& err) {
    if (prefill_) return step_multi(st, pos, 1, x, rope_cs, hidden, logits, err);
    if (!x || (cs_stride_ && !rope_cs) || !hidden) {
        err = "[b200qmm: plan step: x, rope_cs and hidden are required]";
        return B2_ERR_ARG;
    }
    if (pos >= max_len_) {
        err = fmt("[b200qmm: plan step: position %zu is past the %u the caches hold]", pos, max_len_);
        return B2_ERR_ARG;
    }
    if (logits && !n_logits_) {
        err = "[b200qmm: plan step: the graph has no logits]";
        return B2_ERR_ARG;
    }
    if (has_exchange_ && !attached_) {
        err = "[b200qmm: plan step: a tensor-parallel plan needs its peers first (b2_plan_attach_peers)]";
        return B2_ERR_ARG;
    }
    PLAN_CUDA(launch_set_step(sp_, (uint32_t)pos, (uint32_t)pos, 0, nullptr, 0, st), "set_step");
    PLAN_CUDA(cudaMemcpyAsync(input_, x, n_input_ * sizeof(float), cudaMemcpyHostToDevice, st), "cudaMemcpy(x)");
    if (cs_stride_) PLAN_CUDA(cudaMemcpyAsync(rope_table_, rope_cs, cs_stride_ * sizeof(float), cudaMemcpyHostToDevice, st), "cudaMemcpy(rope)");
    PLAN_CUDA(cudaGraphLaunch(step_exec_, st), "cudaGraphLaunch");
    PLAN_CUDA(cudaMemcpyAsync(hidden, hidden_, n_hidden_ * sizeof(float), cudaMemcpyDeviceToHost, st), "cudaMemcpy(hidden)");
    if (logits) PLAN_CUDA(cudaMemcpyAsync(logits, logits_, n_logits_ * sizeof(float), cudaMemcpyDeviceToHost, st), "cudaMemcpy(logits)");
    PLAN_CUDA(cudaStreamSynchronize(st), "step");
    return check_status(err);
}

int DecodePlanImpl::step_multi(cudaStream_t st, size_t pos, size_t t, const float* x, const float* rope_cs, float* hidden, float* logits,
                               std::string& err) {
    if (prefill_) {
        if (logits) {
            err = "[b200qmm: plan step: a prefill plan has no logits]";
            return B2_ERR_ARG;
        }
        return step_prefill(st, pos, t, x, rope_cs, hidden, err);
    }
    if (t == 0 || t > (size_t)tokens_) {
        err = fmt("[b200qmm: plan step: %zu tokens in a step of a plan made for %d]", t, tokens_);
        return B2_ERR_ARG;
    }
    if (t == 1) return step(st, pos, x, rope_cs, hidden, logits, err);  // one row per table: the one-token layout
    if (!x || (cs_stride_ && !rope_cs) || !hidden) {
        err = "[b200qmm: plan step: x, rope_cs and hidden are required]";
        return B2_ERR_ARG;
    }
    if (pos + t > max_len_) {
        err = fmt("[b200qmm: plan step: positions %zu .. %zu are past the %u the caches hold]", pos, pos + t - 1, max_len_);
        return B2_ERR_ARG;
    }
    if (logits && !n_logits_) {
        err = "[b200qmm: plan step: the graph has no logits]";
        return B2_ERR_ARG;
    }
    uint32_t words[16] = {};
    for (size_t tk = 0; tk < t; tk++) {
        words[4 * tk] = (uint32_t)(pos + tk);  // the token's position
        words[4 * tk + 1] = (uint32_t)pos;     // the position of row 0 of the RoPE table
    }
    PLAN_CUDA(cudaMemcpyAsync(sp_multi_, words, 16 * t, cudaMemcpyHostToDevice, st), "cudaMemcpy(step words)");
    PLAN_CUDA(cudaMemcpy2DAsync(input_, block_floats_ * 4, x, (size_t)n_input_ * 4, (size_t)n_input_ * 4, t, cudaMemcpyHostToDevice, st),
              "cudaMemcpy(x)");
    for (size_t i = 0; i + 1 < cs_off_.size(); i++) {  // table i: t rows of cos | sin, behind the rows of the tables ahead of it
        const size_t row = (size_t)(cs_off_[i + 1] - cs_off_[i]) * 4;
        if (row == 0) continue;
        PLAN_CUDA(cudaMemcpy2DAsync(rope_table_ + cs_off_[i], (size_t)cs_stride_ * 4, rope_cs + t * cs_off_[i], row, row, t, cudaMemcpyHostToDevice, st),
                  "cudaMemcpy(rope)");
    }
    PLAN_CUDA(cudaGraphLaunch(multi_exec_[t], st), "cudaGraphLaunch");
    PLAN_CUDA(cudaMemcpy2DAsync(hidden, (size_t)n_hidden_ * 4, hidden_, block_floats_ * 4, (size_t)n_hidden_ * 4, t, cudaMemcpyDeviceToHost, st),
              "cudaMemcpy(hidden)");
    if (logits)
        PLAN_CUDA(cudaMemcpy2DAsync(logits, (size_t)n_logits_ * 4, logits_, block_floats_ * 4, (size_t)n_logits_ * 4, t, cudaMemcpyDeviceToHost, st),
                  "cudaMemcpy(logits)");
    PLAN_CUDA(cudaStreamSynchronize(st), "step");
    return check_status(err);
}

// A prefill step's kernels for t token rows. A product = the rows to f16 (each multiplied by a power of two, taken out again
// by the GEMM's epilogue), then the tensor-core GEMM: straight into the activation rows where it stores, into a scratch
// matrix where it adds to the rows (a row-wise add follows) or is one of a gate / up pair (the activation kernel follows).
int DecodePlanImpl::run_prefill(cudaStream_t st, size_t pos, size_t t, std::string& err) {
    std::vector<GemmPlan*>& plans = gemm_plans_[t];
    const bool build = plans.empty();
    size_t slot = 0;
    uint64_t count = 0;
    const size_t ld = block_floats_;
    const uint32_t rows = (uint32_t)t;
    const float* x16_src = nullptr;  // the vector whose f16 rows the scratch holds
    size_t x16_k = 0;
    const float* addend = nullptr;  // rows that the norm behind a product still has to add to its own
    auto gemm = [&](const WeightDev& w, float* y, size_t y_ld) -> cudaError_t {
        GemmPlan* gp = nullptr;
        if (build) {
            char msg[256] = {0};
            GemmPeerY py;
            py.ld = y_ld;
            cudaError_t e = gemm_tc_plan_create(w, x16_, t, y, B2_F32, &gp, msg, sizeof msg, 0, 0, 1, y_ld != w.n_out ? &py : nullptr);
            if (e != cudaSuccess) {
                err = fmt("[b200qmm: prefill: %s]", msg);
                return e;
            }
            plans.push_back(gp);
        } else {
            gp = plans[slot];
        }
        slot++;
        count++;
        return launch_gemm_tc(gp, w, t, y, B2_F32, gemm_status_, sm_count_, st, unscale_);
    };
    int rc = B2_OK;
    for (size_t i = 0; i < ops_.size() && rc == B2_OK; i++) {
        const Op& o = ops_[i];
        cudaError_t e = cudaSuccess;
        switch (o.kind) {
            case B2_OP_NORM:
                if (o.rows == 1 && norm_rows_supports(o.norm.n, o.x, o.y, o.p0, ld, ld)) {
                    // a product right behind it that reads exactly this vector gets its f16 rows from the norm kernel
                    const Op* nx = i + 1 < ops_.size() ? &ops_[i + 1] : nullptr;
                    const bool feeds = nx && nx->kind == B2_OP_LINEAR && nx->x == o.y && nx->w.n_in == o.norm.n && o.norm.n % 8 == 0;
                    e = launch_norm_rows(o.x, ld, feeds && o.x16_only ? nullptr : o.y, ld, o.p0, o.norm, rows, feeds ? x16_ : nullptr, unscale_, addend, st);
                    addend = nullptr;
                    count++;
                    if (feeds) {
                        x16_src = o.y;
                        x16_k = o.norm.n;
                        break;  // (the overlap check below would forget the rows just made)
                    }
                } else if (o.rows == 1) {
                    DecNorm n = o.norm;
                    n.x_stride = n.out_stride = (uint32_t)ld;
                    e = launch_norm(o.x, o.y, o.p0, n, rows, st, false);
                    count++;
                } else {
                    for (size_t tk = 0; tk < t && e == cudaSuccess; tk++, count++)
                        e = launch_norm(o.x + tk * ld, o.y + tk * ld, o.p0, o.norm, o.rows, st, false);
                }
                if (overlaps_f(o.y, (size_t)(o.rows - 1) * o.norm.out_stride + o.norm.n, x16_src, x16_k)) x16_src = nullptr;
                break;
            case B2_OP_LINEAR: {
                const size_t K = o.w.n_in, n_out = o.w.n_out;
                if (!(x16_src == o.x && x16_k == K)) {
                    e = launch_to_f16(o.x, B2_F32, t, K, x16_, unscale_, st, 0, ld);
                    count++;
                    x16_src = o.x;
                    x16_k = K;
                }
                if (e != cudaSuccess) break;
                if (o.pair) {
                    e = gemm(o.w, tmp_a_, n_out);
                    if (e == cudaSuccess) e = gemm(o.w2, tmp_b_, n_out);
                    // a product right behind the pair that reads exactly its output gets its f16 rows from the activation kernel
                    // (both GEMMs above have read the scratch rows by then: the kernel is an ordinary launch behind them)
                    const Op* nx = i + 1 < ops_.size() ? &ops_[i + 1] : nullptr;
                    const bool feeds = nx && nx->kind == B2_OP_LINEAR && nx->x == o.y && nx->w.n_in == n_out && glu_rows_f16_supports((uint32_t)n_out);
                    if (e == cudaSuccess)
                        e = launch_glu_rows(tmp_a_, n_out, tmp_b_, n_out, feeds && o.x16_only ? nullptr : o.y, ld, (uint32_t)n_out, rows, o.mode == B2_MODE_GELU_PAIR, st,
                                            feeds ? x16_ : nullptr, unscale_);
                    count++;
                    if (feeds && e == cudaSuccess) {
                        x16_src = o.y;
                        x16_k = n_out;
                        break;  // (the overlap check below would forget the rows just made)
                    }
                } else if (o.mode == B2_MODE_STORE && ((uintptr_t)o.y & 15) == 0) {
                    e = gemm(o.w, o.y, ld);
                } else {
                    // (a product that adds goes through the scratch matrix: its dense rows let the GEMM pick its widest tiles, which
                    // the strided destination's copy-engine stores cannot take; measured 63 + 13 us against 95 us at 4096 x 4096)
                    e = gemm(o.w, tmp_a_, n_out);
                    // (a norm right behind it that reads exactly these rows makes the sum on its way)
                    const Op* nx = i + 1 < ops_.size() ? &ops_[i + 1] : nullptr;
                    if (o.mode == B2_MODE_ADD && nx && nx->kind == B2_OP_NORM && nx->rows == 1 && nx->x == o.y && nx->norm.n == n_out &&
                        norm_rows_supports(nx->norm.n, nx->x, nx->y, nx->p0, ld, ld)) {
                        addend = tmp_a_;
                    } else if (e == cudaSuccess) {
                        e = launch_rows_op(o.y, ld, tmp_a_, n_out, (uint32_t)n_out, rows, o.mode == B2_MODE_ADD, st);
                        count++;
                    }
                }
                if (overlaps_f(o.y, n_out, x16_src, x16_k)) x16_src = nullptr;
                break;
            }
            case B2_OP_QK_ROPE:
                e = launch_qk_rope_rows(o.x, o.y, ld, rows, kv_[o.kv].k, kv_[o.kv].v, kv_f16_, o.p0, o.p1, rope_table_, sp_, o.rope, st);
                count++;
                if (overlaps_f(o.y, (size_t)o.rope.nh * o.rope.hd, x16_src, x16_k)) x16_src = nullptr;
                break;
            case B2_OP_ATTEND:
                if (loop_attend_) {
                    for (size_t tk = 0; tk < t && e == cudaSuccess; tk++, count++)
                        e = launch_attend(o.x + tk * ld, kv_[o.kv].k, kv_[o.kv].v, kv_f16_, o.y + tk * ld, sp_multi_ + 4 * tk, o.attn, status_, att_scratch_, st);
                } else {
                    e = launch_attend_rows(o.x, o.y, ld, rows, kv_[o.kv].k, kv_[o.kv].v, kv_f16_, kv16_, (uint32_t)(pos + t), o.attn, gemm_status_, sm_count_, st);
                    count += kv_f16_ ? 1 : 2;
                }
                if (overlaps_f(o.y, (size_t)o.attn.nh * o.attn.hd, x16_src, x16_k)) x16_src = nullptr;
                break;
            case B2_OP_GLU:
                if (o.n % 4 == 0 && (((uintptr_t)o.x | (uintptr_t)o.y | (uintptr_t)o.z) & 15) == 0) {
                    e = launch_glu_rows(o.x, ld, o.z, ld, o.y, ld, o.n, rows, o.gelu, st);
                    count++;
                } else {
                    for (size_t tk = 0; tk < t && e == cudaSuccess; tk++, count++)
                        e = launch_glu(o.x + tk * ld, o.z + tk * ld, o.y + tk * ld, o.n, o.gelu, st, false);
                }
                if (overlaps_f(o.y, o.n, x16_src, x16_k)) x16_src = nullptr;
                break;
            default: e = cudaErrorInvalidValue;
        }
        if (e != cudaSuccess) {
            if (err.empty()) err = fmt("[b200qmm: prefill: op %zu (kind %u) for %zu tokens: %s]", i, o.kind, t, cudaGetErrorString(e));
            rc = B2_ERR_CUDA;
        }
    }
    if (rc != B2_OK && build) {  // a half-made list must not be found again
        for (GemmPlan* gp : plans) gemm_tc_plan_destroy(gp);
        gemm_plans_.erase(t);
    }
    prefill_launches_ = count;
    return rc;
}

int DecodePlanImpl::step_prefill(cudaStream_t st, size_t pos, size_t t, const float* x, const float* rope_cs, float* hidden, std::string& err) {
    if (!x || (cs_stride_ && !rope_cs) || !hidden) {
        err = "[b200qmm: plan step: x, rope_cs and hidden are required]";
        return B2_ERR_ARG;
    }
    if (t == 0 || t > (size_t)tokens_ || pos + t > max_len_) {
        err = fmt("[b200qmm: plan step: %zu tokens from position %zu: the plan takes %d per step and its caches hold %u positions]", t, pos, tokens_,
                  max_len_);
        return B2_ERR_ARG;
    }
    err.clear();
    PLAN_CUDA(launch_set_step(sp_, (uint32_t)pos, (uint32_t)pos, 0, nullptr, 0, st), "set_step");
    if (loop_attend_) {
        std::vector<uint32_t> words(4 * t, 0u);
        for (size_t tk = 0; tk < t; tk++) {
            words[4 * tk] = (uint32_t)(pos + tk);
            words[4 * tk + 1] = (uint32_t)pos;
        }
        PLAN_CUDA(cudaMemcpyAsync(sp_multi_, words.data(), 16 * t, cudaMemcpyHostToDevice, st), "cudaMemcpy(step words)");
        PLAN_CUDA(cudaStreamSynchronize(st), "step words");
    }
    PLAN_CUDA(cudaMemcpy2DAsync(input_, block_floats_ * 4, x, (size_t)n_input_ * 4, (size_t)n_input_ * 4, t, cudaMemcpyHostToDevice, st),
              "cudaMemcpy(x)");
    for (size_t i = 0; i + 1 < cs_off_.size(); i++) {
        const size_t row = (size_t)(cs_off_[i + 1] - cs_off_[i]) * 4;
        if (row == 0) continue;
        PLAN_CUDA(cudaMemcpy2DAsync(rope_table_ + cs_off_[i], (size_t)cs_stride_ * 4, rope_cs + t * cs_off_[i], row, row, t, cudaMemcpyHostToDevice, st),
                  "cudaMemcpy(rope)");
    }
    PLAN_CUDA(cudaEventRecord(ev0_, st), "cudaEventRecord");
    int rc = run_prefill(st, pos, t, err);
    if (rc) {
        cudaStreamSynchronize(st);
        return rc;
    }
    PLAN_CUDA(cudaEventRecord(ev1_, st), "cudaEventRecord");
    PLAN_CUDA(cudaMemcpy2DAsync(hidden, (size_t)n_hidden_ * 4, hidden_, block_floats_ * 4, (size_t)n_hidden_ * 4, t, cudaMemcpyDeviceToHost, st),
              "cudaMemcpy(hidden)");
    PLAN_CUDA(cudaStreamSynchronize(st), "step");
    PLAN_CUDA(cudaEventElapsedTime(&last_ms_, ev0_, ev1_), "cudaEventElapsedTime");
    GemmStatus gs{};
    PLAN_CUDA(cudaMemcpy(&gs, gemm_status_, sizeof gs, cudaMemcpyDeviceToHost), "cudaMemcpy(GEMM status)");
    if (gs.code) {
        cudaMemset(gemm_status_, 0, sizeof gs);
        err = fmt("[b200qmm: prefill: a GEMM's bounded wait %u gave up in CTA %u]", gs.where, gs.cta);
        return B2_ERR_TIMEOUT;
    }
    return check_status(err);
}

int DecodePlanImpl::kv_write(cudaStream_t st, uint32_t kv, size_t pos0, size_t n, const float* k, const float* v, std::string& err) {
    if (kv >= kv_.size() || !k || !v || pos0 + n > max_len_) {
        err = "[b200qmm: plan kv_write: bad cache index, pointers or range]";
        return B2_ERR_ARG;
    }
    const Kv& c = kv_[kv];
    const size_t row = (size_t)c.nkv * c.hd, chunk = stage_floats_ / row;
    for (size_t at = 0; at < n; at += chunk) {
        size_t m = std::min(chunk, n - at);
        PLAN_CUDA(cudaMemcpyAsync(stage_, k + at * row, m * row * 4, cudaMemcpyHostToDevice, st), "cudaMemcpy(K rows)");
        PLAN_CUDA(cudaMemcpyAsync(stage_ + stage_floats_, v + at * row, m * row * 4, cudaMemcpyHostToDevice, st), "cudaMemcpy(V rows)");
        PLAN_CUDA(launch_kv_rows(stage_, c.k, kv_f16_, true, c.nkv, c.hd, max_len_, (uint32_t)(pos0 + at), (uint32_t)m, st), "kv_rows");
        PLAN_CUDA(launch_kv_rows(stage_ + stage_floats_, c.v, kv_f16_, true, c.nkv, c.hd, max_len_, (uint32_t)(pos0 + at), (uint32_t)m, st),
                  "kv_rows");
        PLAN_CUDA(cudaStreamSynchronize(st), "kv_write");  // the host rows may be pageable: the staging buffer is reused next round
    }
    return B2_OK;
}

int DecodePlanImpl::kv_read(cudaStream_t st, uint32_t kv, size_t pos0, size_t n, float* k, float* v, std::string& err) {
    if (kv >= kv_.size() || !k || !v || pos0 + n > max_len_) {
        err = "[b200qmm: plan kv_read: bad cache index, pointers or range]";
        return B2_ERR_ARG;
    }
    const Kv& c = kv_[kv];
    const size_t row = (size_t)c.nkv * c.hd, chunk = stage_floats_ / row;
    for (size_t at = 0; at < n; at += chunk) {
        size_t m = std::min(chunk, n - at);
        PLAN_CUDA(launch_kv_rows(stage_, c.k, kv_f16_, false, c.nkv, c.hd, max_len_, (uint32_t)(pos0 + at), (uint32_t)m, st), "kv_rows");
        PLAN_CUDA(launch_kv_rows(stage_ + stage_floats_, c.v, kv_f16_, false, c.nkv, c.hd, max_len_, (uint32_t)(pos0 + at), (uint32_t)m, st),
                  "kv_rows");
        PLAN_CUDA(cudaMemcpyAsync(k + at * row, stage_, m * row * 4, cudaMemcpyDeviceToHost, st), "cudaMemcpy(K rows)");
        PLAN_CUDA(cudaMemcpyAsync(v + at * row, stage_ + stage_floats_, m * row * 4, cudaMemcpyDeviceToHost, st), "cudaMemcpy(V rows)");
        PLAN_CUDA(cudaStreamSynchronize(st), "kv_read");
    }
    return B2_OK;
}

int DecodePlanImpl::generate(cudaStream_t st, uint64_t embed_handle, const WeightDev& embed, int32_t first_token, size_t pos0, size_t n_tokens,
                             const float* rope_cs_table, int32_t* out_tokens, float* elapsed_ms, std::string& err) {
    if (!n_logits_ || !logits_) {
        err = "[b200qmm: plan generate: the graph has no logits]";
        return B2_ERR_ARG;
    }
    if (!out_tokens || (cs_stride_ && !rope_cs_table) || n_tokens == 0 || pos0 + n_tokens > max_len_) {
        err = fmt("[b200qmm: plan generate: %zu tokens from position %zu do not fit the %u positions of the caches, or a pointer is missing]",
                  n_tokens, pos0, max_len_);
        return B2_ERR_ARG;
    }
    if (has_exchange_ && !attached_) {
        err = "[b200qmm: plan generate: a tensor-parallel plan needs its peers first (b2_plan_attach_peers)]";
        return B2_ERR_ARG;
    }
    if (embed.n_in != n_input_ || first_token < 0 || (size_t)first_token >= embed.n_out) {
        err = "[b200qmm: plan generate: the embedding matrix does not match the graph's input, or the token is outside it]";
        return B2_ERR_ARG;
    }
    if (!gen_exec_ || gen_embed_ != embed_handle || gen_embed_dev_.p0 != embed.p0) {
        if (gen_exec_) cudaGraphExecDestroy(gen_exec_);
        gen_exec_ = nullptr;
        gen_embed_ = embed_handle;
        gen_embed_dev_ = embed;
        // the two kernels the step graph does not have, once outside a capture
        PLAN_CUDA(launch_set_step(sp_, 0, 0, 0, token_, first_token, cap_stream_), "set_step");
        PLAN_CUDA(launch_dequantize(embed, 0, 1, input_, cap_stream_, token_), "embedding lookup");
        PLAN_CUDA(launch_argmax(logits_, n_logits_, argmax_val_, argmax_idx_, argmax_counter_, token_, out_tokens_, sp_, cap_stream_), "argmax");
        PLAN_CUDA(cudaStreamSynchronize(cap_stream_), "generate warm-up");
        int rc = capture(cap_stream_, true, &gen_exec_, err);
        if (rc) return rc;
    }
    PLAN_CUDA(launch_set_step(sp_, (uint32_t)pos0, (uint32_t)pos0, 0, token_, first_token, st), "set_step");
    if (cs_stride_)
        PLAN_CUDA(cudaMemcpyAsync(rope_table_, rope_cs_table, n_tokens * cs_stride_ * sizeof(float), cudaMemcpyHostToDevice, st), "cudaMemcpy(rope)");
    PLAN_CUDA(cudaEventRecord(ev0_, st), "cudaEventRecord");
    for (size_t i = 0; i < n_tokens; i++) PLAN_CUDA(cudaGraphLaunch(gen_exec_, st), "cudaGraphLaunch");
    PLAN_CUDA(cudaEventRecord(ev1_, st), "cudaEventRecord");
    PLAN_CUDA(cudaMemcpyAsync(out_tokens, out_tokens_, n_tokens * sizeof(int), cudaMemcpyDeviceToHost, st), "cudaMemcpy(tokens)");
    PLAN_CUDA(cudaStreamSynchronize(st), "generate");
    if (elapsed_ms) PLAN_CUDA(cudaEventElapsedTime(elapsed_ms, ev0_, ev1_), "cudaEventElapsedTime");
    return check_status(err);
}


// ---- tensor-parallel plans: peers ------------------------------------------------------------------------------------
int DecodePlanImpl::export_handle(void* out128, std::string& err) {
    if (!has_exchange_) {
        err = "[b200qmm: plan export: the graph has no exchange op]";
        return B2_ERR_ARG;
    }
    cudaIpcMemHandle_t h[2];
    static_assert(sizeof h == B2_PLAN_HANDLE_BYTES, "handle size");
    PLAN_CUDA(cudaIpcGetMemHandle(&h[0], bufs_), "cudaIpcGetMemHandle(buffers)");
    PLAN_CUDA(cudaIpcGetMemHandle(&h[1], xflags_), "cudaIpcGetMemHandle(flags)");
    memcpy(out128, h, sizeof h);
    return B2_OK;
}

int DecodePlanImpl::attach_peers(uint32_t rank, uint32_t world, const void* handles, std::string& err) {
    if (!has_exchange_ || attached_ || world < 2 || world > 8 || rank >= world || !handles) {
        err = "[b200qmm: plan attach: needs a graph with exchange ops, 2 to 8 ranks, and is done once]";
        return B2_ERR_ARG;
    }
    peers_.rank = rank;
    peers_.world = world;
    for (uint32_t p = 0; p < world; p++) {
        if (p == rank) {
            peers_.base[p] = bufs_;
            peers_.flags[p] = xflags_;
            continue;
        }
        cudaIpcMemHandle_t h[2];
        memcpy(h, (const char*)handles + (size_t)p * B2_PLAN_HANDLE_BYTES, sizeof h);
        void *b = nullptr, *f = nullptr;
        PLAN_CUDA(cudaIpcOpenMemHandle(&b, h[0], cudaIpcMemLazyEnablePeerAccess), "cudaIpcOpenMemHandle(buffers)");
        peer_maps_.push_back(b);
        PLAN_CUDA(cudaIpcOpenMemHandle(&f, h[1], cudaIpcMemLazyEnablePeerAccess), "cudaIpcOpenMemHandle(flags)");
        peer_maps_.push_back(f);
        peers_.base[p] = (float*)b;
        peers_.flags[p] = (uint32_t*)f;
    }
    attached_ = true;
    // Which exchanges need the meeting before the writes: those with a kernel, since the previous exchange, that reads
    // the vector outside this rank's own part (the first exchange of the list always meets: its predecessors are the
    // previous step's kernels).
    {
        auto reads_outside = [&](const float* a, size_t na, const Op& ex) {
            if (!a || na == 0) return false;
            const float* v = ex.x;
            const size_t part = ex.n / world;
            const float* own = v + (size_t)rank * part;
            if (!(a < v + ex.n && v < a + na)) return false;  // does not touch the vector
            return !(a >= own && a + na <= own + part);        // touches it outside the own part
        };
        bool first = true;
        for (size_t i = 0; i < ops_.size(); i++) {
            if (ops_[i].kind != B2_OP_EXCHANGE) continue;
            Op& ex = ops_[i];
            bool need = first;
            first = false;
            for (size_t b = i; b-- > 0 && !need;) {
                const Op& o = ops_[b];
                if (o.kind == B2_OP_EXCHANGE) break;
                switch (o.kind) {
                    case B2_OP_LINEAR:
                        if (o.self || o.region < 0) need = reads_outside(o.region < 0 ? o.x : o.sx, o.w.n_in, ex);
                        if (o.mode != B2_MODE_STORE && !o.pair) need = need || reads_outside(o.y, o.w.n_out, ex);
                        need = need || reads_outside(o.z, 1, ex);
                        break;
                    case B2_OP_NORM: need = reads_outside(o.x, (size_t)(o.rows - 1) * o.norm.x_stride + o.norm.n, ex); break;
                    case OP_SPLIT: need = !o.self && reads_outside(o.sx, o.n, ex); break;
                    case B2_OP_GLU: need = reads_outside(o.x, o.n, ex) || reads_outside(o.z, o.n, ex); break;
                    case B2_OP_QK_ROPE: need = reads_outside(o.x, (size_t)o.rope.v_off + (size_t)o.rope.nkv * o.rope.hd + (size_t)o.rope.nh * o.rope.q_stride, ex); break;
                    case B2_OP_ATTEND: need = reads_outside(o.x, (size_t)o.attn.nh * o.attn.hd, ex); break;
                    default: need = true;
                }
            }
            ex.meet_first = need;
        }
    }
    // the step graph captured at creation has no exchange nodes: capture it again
    if (step_exec_) cudaGraphExecDestroy(step_exec_);
    step_exec_ = nullptr;
    return capture(cap_stream_, false, &step_exec_, err);
}

}  // namespace b2
