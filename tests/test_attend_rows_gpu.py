"""The prefill attention (`attention_ext`, src/model.rs:2214-2309) around its tiles of 128 rows and keys, and where clusters share out the keys."""
import numpy as np
import pytest

from test_plan_prefill_gpu import cache_err, fill, one_by_one, plans, rope_rows
from util import row_err

pytestmark = pytest.mark.gpu

# query heads, KV heads, head dimension: tiles of 128 / G tokens, two row tiles a CTA
SHAPES = [(4, 2, 64), (8, 1, 128), (4, 4, 64)]


@pytest.mark.parametrize("nh,nkv,hd", SHAPES)
@pytest.mark.parametrize("kv_f16", [False, True], ids=["f32cache", "f16cache"])
def test_tiles_blocks_and_shares_of_the_keys(backend, nh, nkv, hd, kv_f16):
    cfg = dict(n_layers=1, h=256, nh=nh, nkv=nkv, hd=hd, inter=256, vocab=256)
    one, pre, inv_freq, _, keep = plans(backend, cfg, seed=1700 + nh, tokens=300, max_len=4400, kv_f16=kv_f16)
    rng = np.random.default_rng(96)
    # one tile of keys, its edges, two / four / eight shares of them (512, 1024 and 4096 keys at few rows), a last share without keys
    for pos, t in ((0, 3), (0, 127), (1, 128), (127, 2), (0, 257), (500, 12), (1100, 33), (1152, 1), (4090, 7), (4096, 300)):
        if pos:
            fill((one, pre), cfg, pos, 800 + pos)
        xs = rng.standard_normal((t, cfg["h"])).astype(np.float32)
        h1 = one_by_one(one, pos, xs, inv_freq)
        hp, _ = pre.step_multi(pos, xs, rope_rows(pos, t, inv_freq))
        # the bound of a prefill step a layer of depth: f16 operands of the products and the attention
        assert row_err(hp, h1.astype(np.float64)) < 2e-3, (pos, t, row_err(hp, h1.astype(np.float64)))
        assert cache_err(pre, one, cfg, pos, t) < 2e-3
    one.close()
    pre.close()
