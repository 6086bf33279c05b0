"""What this framework's speed is measured on: one pass of each of its public entry points at the sizes that its users run.

``listed()`` holds the fixed cases, ``draw(rng)`` gives more of the same ranges. Everything a program holds before the call (uploaded
weights, plans with their caches, input arrays) is made by ``prepare``; ``run`` makes the call. Weights and inputs are random and follow
from the seed: zero-mean weights in the on-disk layouts of the formats, activations N(0, 1).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from oxinfer_b200 import decode as D
from oxinfer_b200._lib import FMT_F8E4M3, FMT_Q4_K, FMT_Q6_K, FMT_Q8_0, MODE_SILU_PAIR, MODE_STORE
from oxinfer_b200.backend import Backend, Gguf, Job, MlxQ4, RowsJob
from oxinfer_b200.synth import OTHER_BLOCKS, OTHER_NAMES

DEV = "cuda"
DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
OTHER_IDS = {name: kind for kind, name in OTHER_NAMES.items()}
# bytes per weight as stored
WIDTH = {"mlx4": 0.5625, "q4_k": 144 / 256, "q6_k": 210 / 256, "q8_0": 34 / 32, "f8": 1.0}
WIDTH.update({name: OTHER_BLOCKS[kind][1] / OTHER_BLOCKS[kind][0] for kind, name in OTHER_NAMES.items()})

# Decoder shapes: hidden size, query heads, key / value heads, head dimension, feed-forward width, vocabulary.
SHAPES = {
    "h4096": (4096, 32, 8, 128, 14336, 128256),   # the benchmark's 8-billion-parameter shape
    "h3072": (3072, 24, 12, 128, 8192, 32064),
    "h2048": (2048, 32, 8, 64, 8192, 32064),
    "h1536": (1536, 12, 12, 128, 4096, 32000),
    "h1024": (1024, 16, 2, 64, 2816, 32000),
}


def listed() -> list:
    return [
        # One token of batch-1 decode through a single MLX 4-bit projection, vectors on the device: the smallest call there is.
        {"name": "matvec_mlx4_4096x4096", "path": "matvec", "fmt": "mlx4", "n_out": 4096, "n_in": 4096, "pair": False},
        # The same at a feed-forward width for a format that runs on the generic block kernel.
        {"name": "matvec_q5_k_14336x4096", "path": "matvec", "fmt": "q5_k", "n_out": 14336, "n_in": 4096, "pair": False},
        # The trait's own decode call: the q / k / v products of one token from host memory to host memory, one call.
        {"name": "rows_q4_k_qkv_t1", "path": "boundary", "fmt": "q4_k", "n_in": 4096, "jobs": "4096,1024,1024", "t": 1},
        # A handful of tokens (speculative verification, a few sequences decoding together) through an 8-bit matrix.
        {"name": "matmul_q8_0_t6", "path": "matmul", "fmt": "q8_0", "t": 6, "n_out": 4096, "n_in": 14336, "x": "f32", "y": "f32", "fp8": False},
        # A short ragged prompt through a Q6_K matrix.
        {"name": "matmul_q6_k_t37", "path": "matmul", "fmt": "q6_k", "t": 37, "n_out": 14336, "n_in": 4096, "x": "f32", "y": "f32", "fp8": False},
        # The headline prefill product.
        {"name": "matmul_q4_k_t512", "path": "matmul", "fmt": "q4_k", "t": 512, "n_out": 14336, "n_in": 4096, "x": "bf16", "y": "f32", "fp8": False},
        # A large dense projection with FP8 weights and FP8 activations: the largest case.
        {"name": "matmul_f8_t8192_fp8act", "path": "matmul", "fmt": "f8", "t": 8192, "n_out": 28672, "n_in": 12288, "x": "bf16", "y": "bf16", "fp8": True},
        # The routed experts of one layer at a small serving batch and at a prefill batch.
        {"name": "moe_t64", "path": "moe", "fmt": "mlx4", "t": 64, "experts": 128, "k": 8, "h": 2048, "inter": 768},
        {"name": "moe_t4096", "path": "moe", "fmt": "mlx4", "t": 4096, "experts": 128, "k": 8, "h": 2048, "inter": 768},
        # A whole decode token of the 8B-shaped decoder, host vectors in and out, 2048 tokens of context.
        {"name": "decode_h4096_ctx2048", "path": "decode", "shape": "h4096", "layers": 32, "weights": "q4_k", "ctx": 2048, "kv_f16": False},
        # Four drafted tokens verified in one step of a multi-token plan.
        {"name": "verify4_h4096_ctx2048", "path": "verify", "shape": "h4096", "layers": 16, "weights": "q4_k", "ctx": 2048, "t": 4, "kv_f16": False},
        # A 2048-token prompt through the prefill plan of half of that decoder.
        {"name": "prefill2048_h4096", "path": "prefill", "shape": "h4096", "layers": 16, "weights": "q4_k", "ctx": 0, "t": 2048, "kv_f16": False},
    ]


def _log(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    path = rng.choice(["matvec", "boundary", "matmul", "matmul", "moe", "decode", "verify", "prefill"])
    main = ["mlx4", "q4_k", "q6_k", "q8_0", "f8"]
    if path == "matvec":
        fmt = rng.choice(main + main + sorted(OTHER_IDS))
        return {"path": path, "fmt": fmt, "n_out": _log(rng, 512, 32064), "n_in": 256 * _log(rng, 4, 56), "pair": rng.random() < 0.25}
    if path == "boundary":
        jobs = [4 * _log(rng, 64, 3584) for _ in range(rng.randint(1, 3))]
        return {"path": path, "fmt": rng.choice(main), "n_in": 256 * _log(rng, 4, 48), "jobs": ",".join(map(str, jobs)), "t": _log(rng, 1, 512)}
    if path == "matmul":
        fmt, t, n_out, n_in = rng.choice(main), _log(rng, 2, 8192), _log(rng, 512, 28672), 256 * _log(rng, 4, 56)
        while 2.0 * t * n_out * n_in > 4e12:
            t //= 2
        # up to eight tokens a program keeps f32 rows (exact products); longer batches come in any of the three types
        few = t <= 8
        return {"path": path, "fmt": fmt, "t": t, "n_out": n_out, "n_in": n_in, "x": "f32" if few else rng.choice(["f32", "bf16", "f16"]),
                "y": "f32" if few else rng.choice(["f32", "bf16"]), "fp8": fmt == "f8" and not few and rng.random() < 0.6}
    if path == "moe":
        experts = rng.choice([8, 16, 32, 64, 128])
        return {"path": path, "fmt": rng.choice(["mlx4", "q4_k"]), "t": _log(rng, 1, 4096), "experts": experts, "k": rng.choice([2, 4, 6, 8]),
                "h": 256 * _log(rng, 4, 12), "inter": 256 * _log(rng, 2, 8)}
    case = {"path": path, "shape": rng.choice(sorted(SHAPES)), "layers": rng.randint(2, 12), "weights": rng.choice(["q4_k", "q4_k", "mixed", "mlx4", "f8"]),
            "ctx": _log(rng, 8, 8192), "kv_f16": rng.random() < 0.4}
    if path == "verify":
        case["t"] = rng.randint(2, 4)
    if path == "prefill":
        case["ctx"] = rng.choice([0, _log(rng, 8, 4096)])
        case["t"] = _log(rng, 16, 2048)
    return case


# ---- weights --------------------------------------------------------------------------------------------------------------------
def _bytes(g, *shape) -> torch.Tensor:
    return torch.randint(0, 256, shape, dtype=torch.uint8, device=DEV, generator=g)


def _uniform(g, shape, lo, hi) -> torch.Tensor:
    return torch.rand(shape, device=DEV, generator=g) * (hi - lo) + lo


def _put_f16(blocks: torch.Tensor, at: int, v: torch.Tensor) -> None:
    blocks[:, at : at + 2] = v.half().reshape(-1, 1).view(torch.uint8)


def _weight(fmt: str, n_out: int, n_in: int, g):
    """One matrix in its on-disk layout, standard deviation about 1 / sqrt(n_in)."""
    sigma = n_in ** -0.5
    if fmt == "mlx4":
        w = _bytes(g, n_out, n_in // 2).cpu().numpy().view(np.uint32)
        s = (_uniform(g, (n_out, n_in // 64), 0.4, 1.6) * (sigma / 4.6)).bfloat16()
        b = (-8.0 * s.float() + 0.08 * sigma * torch.randn(s.shape, device=DEV, generator=g)).bfloat16()
        return MlxQ4(w, s.view(torch.int16).cpu().numpy().view(np.uint16), b.view(torch.int16).cpu().numpy().view(np.uint16))
    if fmt == "f8":
        q = torch.randn((n_out, n_in), device=DEV, generator=g).mul_(30.0).clamp_(-448.0, 448.0).to(torch.float8_e4m3fn)
        scales = _uniform(g, (-(-n_out // 128), n_in // 128), 0.5, 1.5) * (sigma / 30.0)
        return Gguf(FMT_F8E4M3, q.view(torch.uint8).cpu().numpy().reshape(-1), scales.cpu().numpy(), 128, 128)
    if fmt == "q4_k":  # w = d (sc q - 7.5 m) with 6-bit sc, m: mean 0, std 258 d
        nb = n_out * (n_in // 256)
        blk = _bytes(g, nb, 144)
        d = _uniform(g, (nb,), 0.9, 1.1) * (sigma / 258.0)
        _put_f16(blk, 0, d)
        _put_f16(blk, 2, 7.5 * d)
        return Gguf(FMT_Q4_K, blk.cpu().numpy().reshape(-1))
    if fmt == "q6_k":  # w = d sc (q - 32) with sc in -32 .. 31
        nb = n_out * (n_in // 256)
        blk = _bytes(g, nb, 210)
        blk[:, 192:208] = (blk[:, 192:208] & 63) + 224  # as signed bytes -32 .. 31
        _put_f16(blk, 208, _uniform(g, (nb,), 0.9, 1.1) * (sigma / 342.0))
        return Gguf(FMT_Q6_K, blk.cpu().numpy().reshape(-1))
    if fmt == "q8_0":
        nb = n_out * (n_in // 32)
        blk = _bytes(g, nb, 34)
        _put_f16(blk, 0, _uniform(g, (nb,), 0.9, 1.1) * (sigma / 73.9))
        return Gguf(FMT_Q8_0, blk.cpu().numpy().reshape(-1))
    kind = OTHER_IDS[fmt]
    size, width, fields = OTHER_BLOCKS[kind]
    nb = n_out * (n_in // size)
    blk = _bytes(g, nb, width)
    for at, magnitude, signed in fields:
        v = magnitude * torch.randn((nb,), device=DEV, generator=g)
        _put_f16(blk, at, v if signed else v.abs())
    if fmt == "mxfp4":  # an exponent byte instead of an f16 scale
        blk[:, 0] = torch.randint(118, 125, (nb,), device=DEV, generator=g).to(torch.uint8)
    return Gguf(kind, blk.cpu().numpy().reshape(-1))


class State:
    """What a program holds between calls. A plan goes before the weights it reads."""

    plan = None

    def __del__(self):
        if self.plan is not None:
            self.plan.close()


_backends: dict = {}


def _backend(fp8: bool = False) -> Backend:
    """One context per setting for the whole process, on torch's stream, as a program with torch tensors binds it."""
    if fp8 not in _backends:
        be = Backend(0)
        be.set_stream(torch.cuda.current_stream().cuda_stream)
        be.set_fp8_activations(fp8)
        _backends[fp8] = be
    return _backends[fp8]


def _upload(be, fmt, n_out, n_in, g):
    dev = be.upload(_weight(fmt, n_out, n_in, g), n_out, n_in)
    assert dev is not None, be.last_declined
    return dev


def _randn(g, *shape) -> torch.Tensor:
    return torch.randn(shape, device=DEV, generator=g)


def _model(s: State, case: dict, g) -> None:
    """A decoder's uploaded weights and its plan, the caches filled up to ``ctx``. Two layers' bytes serve all layers in turn (every
    layer has device memory of its own, so a step reads as much as with bytes of its own)."""
    h, nh, nkv, hd, inter, vocab = SHAPES[case["shape"]]
    n_layers, path, ctx, t = case["layers"], case["path"], case["ctx"], case.get("t", 1)
    cfg = D.LlamaConfig(n_layers, h, nh, nkv, hd, inter, vocab)
    fmt = {"mixed": "q4_k"}.get(case["weights"], case["weights"])
    sizes = {"q": (nh * hd, h), "k": (nkv * hd, h), "v": (nkv * hd, h), "o": (h, nh * hd), "gate": (inter, h), "up": (inter, h), "down": (h, inter)}
    # the mixed files keep v and down in Q6_K and o in Q8_0
    fmts = {k: ({"v": "q6_k", "down": "q6_k", "o": "q8_0"}.get(k, fmt) if case["weights"] == "mixed" else fmt) for k in sizes}
    sets = [{k: _weight(fmts[k], *sizes[k], g) for k in sizes} for _ in range(min(2, n_layers))]

    def norm():
        return (1.0 + 0.1 * _randn(g, h)).cpu().numpy()

    layers = []
    for i in range(n_layers):
        layer = {k: s.be.upload(sets[i % len(sets)][k], *sizes[k]) for k in sizes}
        layer.update(ln_pre=norm(), ln_post=norm())
        layers.append(layer)
    prefill = path == "prefill"
    s.head = None if prefill else _upload(s.be, "q6_k", vocab, h, g)
    s.layers = layers
    graph = D.llama_graph(cfg, layers, norm(), s.head, prefill=prefill)
    max_len = -(-(ctx + t + 64) // 64) * 64
    make = {"decode": lambda: D.decode_plan(s.be, graph, max_len, kv_f16=case["kv_f16"]),
            "verify": lambda: D.decode_plan_multi(s.be, graph, max_len, 4, kv_f16=case["kv_f16"]),
            "prefill": lambda: D.decode_plan_prefill(s.be, graph, max_len, t, kv_f16=case["kv_f16"])}[path]
    s.plan = make()
    assert s.plan is not None, s.be.last_declined
    if ctx:
        k, v = (_randn(g, ctx, nkv, hd).cpu().numpy() for _ in range(2))
        for i in range(n_layers):
            s.plan.kv_write(i, 0, k, v)
    inv = D.rope_inv_freq(hd, cfg.rope_theta)
    s.pos, s.cs = ctx, np.stack([D.rope_table(ctx + i, inv) for i in range(t)])
    s.x = _randn(g, t, h).cpu().numpy()
    if prefill:  # prompts travel through page-locked arrays
        s.pinned = [torch.from_numpy(s.x).pin_memory(), torch.empty((t, h), pin_memory=True)]
        s.x, s.hidden = s.pinned[0].numpy(), s.pinned[1].numpy()


def prepare(case: dict, seed: int):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    s = State()
    s.case, path = case, case["path"]
    s.be = _backend(case.get("fp8", False))
    if path == "matvec":
        n_out, n_in = case["n_out"], case["n_in"]
        s.w = _upload(s.be, case["fmt"], n_out, n_in, g)
        s.up = _upload(s.be, case["fmt"], n_out, n_in, g) if case["pair"] else None
        s.x, s.y = _randn(g, n_in), torch.zeros(n_out, device=DEV)
    elif path == "boundary":
        s.x = _randn(g, case["t"], case["n_in"]).cpu().numpy()
        sizes = [int(n) for n in case["jobs"].split(",")]
        ys = [np.zeros((case["t"], n), np.float32) for n in sizes]
        kind = RowsJob if case["t"] <= 4 else Job
        s.jobs = [kind(_upload(s.be, case["fmt"], n, case["n_in"], g), y) for n, y in zip(sizes, ys)]
    elif path == "matmul":
        s.w = _upload(s.be, case["fmt"], case["n_out"], case["n_in"], g)
        s.x = _randn(g, case["t"], case["n_in"]).to(DTYPES[case["x"]])
        s.y = torch.zeros((case["t"], case["n_out"]), device=DEV, dtype=DTYPES[case["y"]])
    elif path == "moe":
        e, h, inter = case["experts"], case["h"], case["inter"]
        gate_up = [_upload(s.be, case["fmt"], 2 * inter, h, g) for _ in range(e)]
        down = [_upload(s.be, case["fmt"], h, inter, g) for _ in range(e)]
        s.w = s.be.upload_moe(gate_up, down, h, inter)
        assert s.w is not None, s.be.last_declined
        # router logits N(0, 1) with a bias per expert: a skewed load
        p = torch.softmax(_randn(g, case["t"], e) + _randn(g, e), dim=1)
        w, ids = p.topk(case["k"], dim=1)
        s.ids, s.route_w = ids.int().cpu().numpy(), (w / w.sum(1, keepdim=True)).cpu().numpy()
        s.x, s.y = _randn(g, case["t"], h), torch.zeros((case["t"], h), device=DEV)
    else:
        _model(s, case, g)
    return s


def run(s):
    path = s.case["path"]
    if path == "matvec":
        done = s.be.matvec_dev(s.w, s.x, s.y, MODE_SILU_PAIR if s.up else MODE_STORE, s.up)
        out = s.y
    elif path == "boundary":
        done = s.be.matvec_rows(s.x, s.jobs) if s.case["t"] <= 4 else s.be.matmul(s.x, s.jobs)
        out = [j.y for j in s.jobs]
    elif path == "matmul":
        done = s.be.matmul_dev(s.w, s.x, s.y)
        out = s.y
    elif path == "moe":  # adds to the residual rows y
        done = s.be.moe_dev(s.x, s.ids, s.route_w, s.w, s.y)
        out = s.y
    elif path == "decode":
        return s.plan.step(s.pos, s.x[0], s.cs[0])
    elif path == "verify":
        return s.plan.step_multi(s.pos, s.x, s.cs)
    else:
        return s.plan.step_multi(s.pos, s.x, s.cs, want_logits=False, hidden_out=s.hidden)[0]
    assert done, s.be.last_declined
    return out


def work(case: dict) -> dict:
    path, width = case["path"], WIDTH.get(case.get("fmt"), 0.0)
    if path == "matvec":
        n, k, m = case["n_out"], case["n_in"], 2 if case["pair"] else 1
        return {"bytes": m * n * k * width + 4 * (n + k), "flops": 2.0 * m * n * k}
    if path == "boundary":
        n, k, t = sum(int(v) for v in case["jobs"].split(",")), case["n_in"], case["t"]
        return {"bytes": n * k * width + 4 * t * (n + k), "flops": 2.0 * t * n * k}
    if path == "matmul":
        n, k, t = case["n_out"], case["n_in"], case["t"]
        size = {"f32": 4, "bf16": 2, "f16": 2}
        return {"bytes": n * k * width + t * (k * size[case["x"]] + n * size[case["y"]]), "flops": 2.0 * t * n * k}
    if path == "moe":
        e, k, t, h, inter = case["experts"], case["k"], case["t"], case["h"], case["inter"]
        used = e * (1.0 - (1.0 - min(k, e) / e) ** t)  # experts that a batch reaches when the routes are even
        return {"bytes": used * 3 * inter * h * width + 12 * t * h, "flops": 6.0 * t * k * inter * h}
    h, nh, nkv, hd, inter, vocab = SHAPES[case["shape"]]
    attn, mlp = h * hd * 2 * (nh + nkv), 3 * h * inter
    if case["weights"] == "mixed":
        stored = WIDTH["q4_k"] * (h * hd * (nh + nkv) + 2 * h * inter) + WIDTH["q6_k"] * (h * hd * nkv + h * inter) + WIDTH["q8_0"] * h * hd * nh
    else:
        stored = WIDTH[case["weights"]] * (attn + mlp)
    t, ctx, size = case.get("t", 1), case["ctx"], 2 if case["kv_f16"] else 4
    head = 0 if path == "prefill" else h * vocab
    cache = 2 * nkv * hd * size * (ctx + t)
    scored = t * ctx + t * (t + 1) / 2
    return {"bytes": case["layers"] * (stored + cache) + head * WIDTH["q6_k"] + 4 * t * (2 * h + (vocab if head else 0)),
            "flops": case["layers"] * (2.0 * t * (attn + mlp) + 4.0 * nh * hd * scored) + 2.0 * t * head}


def tolerance(case: dict) -> dict:
    """Up to eight f32 rows are multiplied with f32-like products (21 bits of every activation, f32 sums); longer batches have f16
    operands with f32 sums, and a bf16 result its own rounding. Whole decoders repeat that through their layers."""
    path = case["path"]
    if path == "matmul":
        if case["y"] == "bf16":
            return {"rel": 4e-3}
        return {"rel": 2e-5} if case["fp8"] else {"rel": 1e-5 if case["t"] <= 8 else 1e-3}
    if path == "boundary":
        return {"rel": 1e-5 if case["t"] <= 8 else 1e-3}
    if path == "moe":
        return {"rel": 1e-5 if case["t"] * case["k"] <= 64 else 1e-3}
    return {"matvec": {"rel": 1e-5}, "decode": {"rel": 3e-5}, "verify": {"rel": 3e-5}, "prefill": {"rel": 5e-3}}[path]
