"""The decode attention (`dattn`, src/cuda_decode.cu:396-536) over the shapes of its clusters: one to four rows a cluster, several groups of
rows, clusters of sixteen and of eight CTAs, contexts at the edges of its tiles (64 keys) and parts (16 tiles)."""
import numpy as np
import pytest

from oracle import oracle as O

from test_plan_multi_gpu import fill, one_by_one, rope_rows, same_caches, two_plans
from util import row_err

pytestmark = pytest.mark.gpu

# query heads, KV heads, head dimension: one row a KV head, two, eight (two groups a token), sixteen KV heads (eight CTAs a cluster at any token count)
SHAPES = [(4, 4, 64), (4, 2, 128), (8, 1, 64), (16, 16, 64)]


@pytest.mark.parametrize("nh,nkv,hd", SHAPES)
@pytest.mark.parametrize("kv_f16", [False, True], ids=["f32cache", "f16cache"])
def test_rows_groups_and_parts(backend, nh, nkv, hd, kv_f16):
    cfg = dict(n_layers=1, h=256, nh=nh, nkv=nkv, hd=hd, inter=256, vocab=256)
    one, many, inv_freq, cpu, keep = two_plans(backend, cfg, seed=1300 + nh, max_len=1300, kv_f16=kv_f16, interleaved=nkv != 2, with_cpu=not kv_f16)
    rng = np.random.default_rng(79)
    for pos in (5, 63, 1021, 1024, 1087):
        for t in (2, 4):
            fill((one, many), cfg, pos, 600 + pos, cpu)
            xs = rng.standard_normal((t, cfg["h"])).astype(np.float32)
            h1, l1 = one_by_one(one, pos, xs, inv_freq)
            hm, lm = many.step_multi(pos, xs, rope_rows(pos, t, inv_freq))
            assert np.array_equal(hm, h1) and np.array_equal(lm, l1), (pos, t)
            same_caches(one, many, cfg, pos, t)
            if cpu is not None:
                for i in range(t):
                    hc, lc = cpu.step(pos + i, xs[i], O.rope_table(pos + i, inv_freq), exact=True)
                    # (f32 sums over at most 1091 keys: the bound of the whole decoder's steps)
                    assert row_err(h1[i][None], hc[None]) < 1e-4 and row_err(l1[i][None], lc[None]) < 1e-4, (pos, i)
    one.close()
    many.close()


def test_turned_by_a_launch_of_its_own_the_bits_are_the_same(backend, monkeypatch):
    cfg = dict(n_layers=2, h=256, nh=4, nkv=2, hd=64, inter=256, vocab=256)
    plans = []
    for fuse in ("1", "0"):
        monkeypatch.setenv("B2_PLAN_FUSE_ROPE", fuse)
        plans.append(two_plans(backend, cfg, seed=1400, max_len=256))
    rng = np.random.default_rng(80)
    inv_freq = plans[0][2]
    for pos in (0, 62, 126):
        xs = rng.standard_normal((4, cfg["h"])).astype(np.float32)
        got = []
        for one, many, _, _, _ in plans:
            if pos:
                fill((one, many), cfg, pos, 700 + pos)
            got += [one_by_one(one, pos, xs, inv_freq), many.step_multi(pos, xs, rope_rows(pos, 4, inv_freq))]
        for h, l in got[1:]:
            assert np.array_equal(h, got[0][0]) and np.array_equal(l, got[0][1]), pos


def test_what_a_later_token_brings_does_not_reach_an_earlier_one(backend):
    """An infinity in the last token's input makes its own results not finite and nobody else's."""
    cfg = dict(n_layers=1, h=256, nh=4, nkv=2, hd=64, inter=256, vocab=256)
    one, many, inv_freq, _, keep = two_plans(backend, cfg, seed=1500, max_len=256)
    rng = np.random.default_rng(81)
    xs = rng.standard_normal((4, cfg["h"])).astype(np.float32)
    fill((one, many), cfg, 60, 900)
    h1, l1 = one_by_one(one, 60, xs[:3], inv_freq)
    xs[3, 7] = np.inf
    hm, lm = many.step_multi(60, xs, rope_rows(60, 4, inv_freq))
    assert np.array_equal(hm[:3], h1) and np.array_equal(lm[:3], l1)
    assert not np.isfinite(hm[3]).all()
