"""Sliding windows, and rows that are not finite, in the attentions (`dattn`, src/cuda_decode.cu:396-536; `attention_ext`, src/model.rs:2214-2309)
against 64 bits. The graphs hold nothing but RoPE and attention; the factors are cos 1 and sin 0, so a step's input is its queries, keys and values."""
import numpy as np
import pytest

from oxinfer_b200 import decode as D

from util import row_err

pytestmark = pytest.mark.gpu

SHAPES = [(4, 2, 64), (8, 1, 128), (4, 4, 64)]
NO_LIMIT = 2**32 - 1


def graph(nh, nkv, hd, window):
    g = D.Graph()
    nq, row = nh * hd, nkv * hd
    qkv, q, out = g.buf(nq + 2 * row), g.buf(nq), g.buf(nq)
    g.qk_rope(qkv, q, 0, nh, nkv, hd, hd // 2, nq, nq + row, False, 1e-6)
    g.attend(q, out, 0, nh, nkv, hd, hd ** -0.5, window=window)
    g.input, g.n_input, g.hidden, g.n_hidden = qkv, nq + 2 * row, out, nq
    g.kv, g.rope_halves = [(nkv, hd)], [hd // 2]
    return g


def inputs(nh, nkv, hd, pos, t, seed):
    rng = np.random.default_rng(seed)
    k, v = (rng.standard_normal((pos, nkv * hd)).astype(np.float32) for _ in range(2))
    x = rng.standard_normal((t, (nh + 2 * nkv) * hd)).astype(np.float32)
    cs = np.concatenate([np.ones((t, hd // 2)), np.zeros((t, hd // 2))], axis=1).astype(np.float32)
    return k, v, x, cs


def reference(nh, nkv, hd, window, k, v, x):
    pos, t = len(k), len(x)
    nq, row = nh * hd, nkv * hd
    keys = np.concatenate([k, x[:, nq:nq + row]]).reshape(-1, nkv, hd).astype(np.float64)
    vals = np.concatenate([v, x[:, nq + row:]]).reshape(-1, nkv, hd).astype(np.float64)
    out = np.zeros((t, nh, hd))
    for i in range(t):
        lo = max(0, pos + i + 1 - window) if window else 0
        q = x[i, :nq].reshape(nkv, nh // nkv, hd).astype(np.float64)
        s = np.einsum("kgd,jkd->kgj", q, keys[lo:pos + i + 1]) * hd ** -0.5
        p = np.exp(s - s.max(axis=-1, keepdims=True))
        out[i] = (np.einsum("kgj,jkd->kgd", p, vals[lo:pos + i + 1]) / p.sum(-1)[..., None]).reshape(nh, hd)
    return out.reshape(t, nq)


@pytest.mark.parametrize("nh,nkv,hd", SHAPES)
@pytest.mark.parametrize("window", [1, 3, 48, 64, 129, 1000, NO_LIMIT])
def test_steps_of_several_tokens_with_windows_at_the_edges_of_the_tiles(backend, nh, nkv, hd, window):
    one, many = D.decode_plan(backend, graph(nh, nkv, hd, window), 1400), D.decode_plan_multi(backend, graph(nh, nkv, hd, window), 1400, 4)
    # windows of a step's tokens that start in different tiles (64 keys) and batches (8), parts of sixteen tiles, positions inside the first window
    for pos in (0, 2, 62, 65, 126, 191, 1022, 1100):
        k, v, x, cs = inputs(nh, nkv, hd, pos, 4, 40 + pos)
        for p in (one, many):
            if pos:
                p.kv_write(0, 0, k, v)
        want = reference(nh, nkv, hd, window, k, v, x)
        h1 = np.stack([one.step(pos + i, x[i], cs[i], want_logits=False)[0] for i in range(4)])
        for t in (2, 3, 4):
            hm, _ = many.step_multi(pos, x[:t], cs[:t], want_logits=False)
            assert np.array_equal(hm, h1[:t]), (pos, t)
        # (f32 sums of at most 1104 terms, scores of a few units)
        assert row_err(h1, want) < 2e-6 * max(1, hd / 64), (pos, row_err(h1, want))
    one.close()
    many.close()


# four shares, four (two groups of rows a token), two of sixteen heads, four of eight heads (and eight CTAs a cluster)
@pytest.mark.parametrize("nh,nkv,hd,max_len", [(4, 2, 64, 12400), (8, 1, 128, 12400), (16, 16, 64, 3200), (8, 8, 64, 12400)])
@pytest.mark.parametrize("window", [0, 1500])
@pytest.mark.parametrize("kv_f16", [False, True], ids=["f32cache", "f16cache"])
def test_clusters_that_share_a_heads_keys(backend, nh, nkv, hd, max_len, window, kv_f16):
    """Long caches: every 1024 keys go to the next cluster. One of them, the next ones too, all; windows that leave the first ones without keys."""
    one, many = (D.decode_plan(backend, graph(nh, nkv, hd, window), max_len, kv_f16=kv_f16), D.decode_plan_multi(backend, graph(nh, nkv, hd, window), max_len, 4, kv_f16=kv_f16))
    for pos in (0, 5, 1021, 1024, 2046, 3071, 5120, 12390):
        if pos + 4 > max_len:
            continue
        k, v, x, cs = inputs(nh, nkv, hd, pos, 4, 80 + pos)
        if kv_f16:  # (values that f16 holds)
            k, v, x = (a.astype(np.float16).astype(np.float32) for a in (k, v, x))
        for p in (one, many):
            if pos:
                p.kv_write(0, 0, k, v)
        want = reference(nh, nkv, hd, window, k, v, x)
        h1 = np.stack([one.step(pos + i, x[i], cs[i], want_logits=False)[0] for i in range(4)])
        for t in (4, 3, 2, 4):
            hm, _ = many.step_multi(pos, x[:t], cs[:t], want_logits=False)
            assert np.array_equal(hm, h1[:t]), (pos, t)
        assert row_err(h1, want) < 2e-6 * max(1, hd / 64), (pos, row_err(h1, want))
    one.close()
    many.close()


@pytest.mark.parametrize("nh,nkv,hd", SHAPES)
@pytest.mark.parametrize("window", [1, 100, 700, NO_LIMIT])
def test_prefill_with_windows_and_shares_of_the_keys(backend, nh, nkv, hd, window):
    pre = D.decode_plan_prefill(backend, graph(nh, nkv, hd, window), 9100, 300)
    # whole tiles (128 keys) outside the window; two, four and eight shares, most of them empty where the window is short
    for pos, t in ((0, 130), (127, 2), (500, 12), (1100, 33), (2100, 5), (4096, 300), (9050, 7)):
        k, v, x, cs = inputs(nh, nkv, hd, pos, t, 60 + pos)
        if pos:
            pre.kv_write(0, 0, k, v)
        got, _ = pre.step_multi(pos, x, cs, want_logits=False)
        # (queries, keys, values and probabilities rounded to f16: the bound of a prefill step)
        assert row_err(got, reference(nh, nkv, hd, window, k, v, x)) < 2e-3, (pos, t)
    pre.close()


def test_a_share_without_keys_adds_nothing_whatever_the_queries_hold(backend):
    """Nine key tiles in four shares: the last has none. Its sums are zeros in the place of its copy of the queries."""
    nh, nkv, hd, pos, t = 8, 1, 128, 1100, 33
    pre = D.decode_plan_prefill(backend, graph(nh, nkv, hd, 0), 1200, 64)
    k, v, x, cs = inputs(nh, nkv, hd, pos, t, 70)
    pre.kv_write(0, 0, k, v)
    clean, _ = pre.step_multi(pos, x, cs, want_logits=False)
    for token, head in ((0, 0), (5, 3), (15, 7), (32, 0)):
        bad = x.copy()
        bad[token, head * hd:(head + 1) * hd] = np.nan
        for _ in range(20):
            got, _ = pre.step_multi(pos, bad, cs, want_logits=False)
            own = np.zeros((t, nh), bool)
            own[token, head] = True
            rows = np.isnan(got.reshape(t, nh, hd)).all(-1)
            assert np.array_equal(rows, own) and np.array_equal(got.reshape(t, nh, hd)[~own], clean.reshape(t, nh, hd)[~own])
    pre.close()


@pytest.mark.parametrize("nh,nkv,hd", [(4, 2, 64), (8, 1, 128)])
@pytest.mark.parametrize("window", [0, 70])
def test_values_of_later_and_of_forgotten_tokens_reach_nobody(backend, nh, nkv, hd, window):
    """An infinite value (or one that f16 does not hold) is in nobody's sums who does not see its 64 keys."""
    pre = D.decode_plan_prefill(backend, graph(nh, nkv, hd, window), 512, 300)
    k, v, x, cs = inputs(nh, nkv, hd, 0, 300, 90)
    clean, _ = pre.step_multi(0, x, cs, want_logits=False)
    for token, value in ((70, np.inf), (129, 1e6), (255, -np.inf), (299, np.nan)):
        bad = x.copy()
        bad[token, (nh + nkv) * hd:] = value
        got, _ = pre.step_multi(0, bad, cs, want_logits=False)
        first = token // 64 * 64
        assert np.array_equal(got[:first], clean[:first]), token
        assert not np.isfinite(got[token]).any()
        if window:  # 64 keys that end before the windows of a tile of rows (128 / G tokens) begin
            tile = 128 // (nh // nkv)
            behind = -(-(first + 63 + window) // tile) * tile
            assert np.array_equal(got[behind:], clean[behind:]), token
    pre.close()
