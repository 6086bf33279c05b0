"""The small-batch products (one to eight tokens, gemv_mma.cu) where tiles, rounds and parts of K end unevenly.

Bound: an activation keeps 23 bits of the largest value of its block of 256 (2^-24 of it at most is lost per value) and a row's sums
are f32 sums in at most eight slices, each of K / 8 / 32 terms or fewer: 2e-6 of a row of N(0, 1) activations covers K = 14336.
"""
import numpy as np
import pytest
import torch

import oxinfer_b200 as ob
from oracle import oracle as O
from oxinfer_b200 import synth

from util import FORMATS, make_pair, row_err

pytestmark = pytest.mark.gpu


def products(backend, dev, x):
    xd = torch.from_numpy(x).cuda()
    y = torch.full((len(x), dev.n_out), 7.0, device="cuda")
    assert backend.matmul_dev(dev, xd, y)
    torch.cuda.synchronize()
    return y.cpu().numpy()


@pytest.mark.parametrize("fmt", FORMATS)
# fewer rows than half a tile, a ragged last tile, more tiles than CTAs; fewer units than slices, an odd number of blocks, parts of K
@pytest.mark.parametrize("shape", [(5, 256), (20, 768), (2501, 1280), (37, 14336)])
def test_rows_of_one_to_eight_tokens(backend, fmt, shape):
    n_out, n_in = shape
    ref, m = make_pair(fmt, n_out, n_in, 900 + n_out)
    dev = backend.upload(ref, n_out, n_in)
    x = (synth.activations(8, n_in, 901) * np.float32(1.2345)).astype(np.float32)
    one = np.concatenate([products(backend, dev, x[i : i + 1]) for i in range(8)])
    assert row_err(one, m.matmul_f64(x)) < 2e-6
    for t in (2, 4, 5, 8):
        assert np.array_equal(products(backend, dev, x[:t]), one[:t])


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("shape", [(20000, 4096), (9600, 14336)])
def test_many_tiles_whose_sums_wait_for_the_next_part_of_k(backend, fmt, shape):
    n_out, n_in = shape
    ref, _ = make_pair(fmt, n_out, n_in, 910)
    dev = backend.upload(ref, n_out, n_in)
    x = synth.activations(8, n_in, 911)
    one = np.concatenate([products(backend, dev, x[i : i + 1]) for i in range(8)])
    for t in (3, 8):
        assert np.array_equal(products(backend, dev, x[:t]), one[:t])


def test_more_rows_than_a_grid_dimension_has(backend):
    """65,537 rows under the exactness switch, whose products take any number of rows from the same split."""
    n_out, n_in, t = 24, 256, 65537
    ref, _ = make_pair("q6_k", n_out, n_in, 925)
    dev = backend.upload(ref, n_out, n_in)
    x = np.tile(synth.activations(64, n_in, 926), (1025, 1))[:t]
    backend.set_exact(True)
    try:
        y, few = products(backend, dev, x), products(backend, dev, x[:64])
    finally:
        backend.set_exact(False)
    assert np.array_equal(y, np.tile(few, (1025, 1))[:t])


def test_longest_rows(backend):
    ref, m = make_pair("q8_0", 24, 58368, 920)
    dev = backend.upload(ref, 24, 58368)
    x = synth.activations(8, 58368, 921)
    y = products(backend, dev, x)
    assert row_err(y, m.matmul_f64(x)) < 4e-6  # (four times the terms in a slice)
    assert np.array_equal(products(backend, dev, x[:1]), y[:1])
    ref, _ = make_pair("q8_0", 24, 58624, 922)  # longer ones are refused
    dev = backend.upload(ref, 24, 58624)
    assert not backend.matvec_rows(synth.activations(1, 58624, 923), [ob.RowsJob(dev, np.zeros((1, 24), np.float32))])


@pytest.mark.parametrize("fmt", FORMATS + ["q5_k"])
@pytest.mark.parametrize("shift", [0, 8])
def test_results_over_their_own_vector(backend, fmt, shift):
    """y on top of x, whole or from its ninth value on: the bits of a y apart. GEMMs on another stream hold most SMs when the product
    starts, so that its first CTAs have stored their rows before the others read x."""
    n = 6144
    ref = synth.make(fmt, n, n, 970) if fmt in FORMATS else other(O.Q5_K, n, n, 970)[0]
    dev = backend.upload(ref, n, n)
    x = synth.activations(3, n, 971)
    want = products(backend, dev, x)
    side, busy = torch.cuda.Stream(), ob.Backend(0)
    busy.set_stream(side.cuda_stream)
    gw = busy.upload(synth.q4_k(14336, 4096, 972), 14336, 4096)
    gx, gy = torch.zeros((512, 4096), device="cuda", dtype=torch.float16), torch.zeros((512, 14336), device="cuda")

    def beside(run):
        torch.cuda.synchronize()
        for _ in range(4):
            assert busy.matmul_dev(gw, gx, gy)
        assert run()
        torch.cuda.synchronize()

    xd = torch.from_numpy(x).cuda()
    buf = torch.zeros(n + shift, device="cuda")
    buf[:n] = xd[0]
    beside(lambda: backend.matvec_dev(dev, buf[:n], buf[shift:]))
    assert np.array_equal(buf[shift:].cpu().numpy(), want[0])
    if shift == 0:  # a residual add in place, and several rows
        buf[:] = xd[0]
        beside(lambda: backend.matvec_dev(dev, buf, buf, ob.MODE_ADD))
        assert np.array_equal(buf.cpu().numpy(), x[0] + want[0])
        rows = xd.clone()
        beside(lambda: backend.matmul_dev(dev, rows, rows))
        assert np.array_equal(rows.cpu().numpy(), want)
    busy.close()


@pytest.mark.parametrize("fmt", FORMATS)
def test_values_that_are_not_finite_and_vectors_off_16_bytes(backend, fmt):
    n_out, n_in = 40, 1024
    ref, _ = make_pair(fmt, n_out, n_in, 930)
    dev = backend.upload(ref, n_out, n_in)
    x = synth.activations(2, n_in, 931)
    want = products(backend, dev, x)
    buf = torch.zeros(1 + n_in, device="cuda")
    buf[1:] = torch.from_numpy(x[0]).cuda()
    y = torch.zeros(n_out, device="cuda")
    assert backend.matvec_dev(dev, buf[1:], y)
    torch.cuda.synchronize()
    assert np.array_equal(y.cpu().numpy(), want[0])
    for bad in (np.inf, np.nan):
        x[1, 300] = bad
        y = products(backend, dev, x)
        assert not np.isfinite(y[1]).any()
        assert np.array_equal(y[0], want[0])


@pytest.mark.parametrize("fmt", ["mlx4", "q4_k", "q6_k", "q8_0"])
def test_fast_digits_of_the_largest_values_of_a_block(backend, fmt):
    """Under b2_set_fast_planes a value is rounded to 18 bits, at most 7.6e-6 of its block's largest. 8355680 .. 8355711 units of the split
    would round to a number that three signed digits cannot hold."""
    n_out, n_in = 40, 2048
    ref, m = make_pair(fmt, n_out, n_in, 960)
    dev = backend.upload(ref, n_out, n_in)
    x = 0.25 * synth.activations(3, n_in, 961)
    tops = np.array([8355679, 8355680, 8355696, 8355710, 8355711, 8355647, 8355648, 8355672], np.float64)
    blocks = x.reshape(3, 8, 256)
    blocks[:, np.arange(8), 17 * np.arange(8)] = np.stack([tops, -tops, tops[::-1]]) * 2.0**-22
    x = (blocks * 2.0 ** np.array([0, 5, -9, 3, 0, -20, 11, 1])[None, :, None]).reshape(3, n_in).astype(np.float32)
    w = np.abs(m.dequantize_rows().astype(np.float64))
    lost = 7.6e-6 * np.abs(x.reshape(3, 8, 256)).max(axis=2).astype(np.float64)
    bound = np.einsum("tb,nb->tn", lost, w.reshape(n_out, 8, 256).sum(axis=2))
    want = m.matmul_f64(x)
    try:
        backend.set_fast_planes(True)
        y = products(backend, dev, x)
        one = np.concatenate([products(backend, dev, x[i : i + 1]) for i in range(3)])
    finally:
        backend.set_fast_planes(False)
    # (a thousandth of the bound for the f32 sums: 2e-6 of a row against 7.6e-6 of every block's largest, 2048 times)
    assert (np.abs(y - want) <= 1.001 * bound + 2e-6 * np.abs(want)).all()
    assert np.array_equal(y, one)


OTHERS = list(O.OTHER_KINDS) + [O.NVFP4]


def other(kind, n_out, n_in, seed):
    data, _ = O.random_blocks(kind, n_out * n_in // O.block_size(kind), seed)
    scale = np.array([[0.03 + 0.001 * (seed % 7)]], np.float32) if kind == O.NVFP4 else None
    dims = (n_out, n_in) if kind == O.NVFP4 else (0, 0)
    return ob.Gguf(kind, data, scale, *dims), O.Matrix.gguf(kind, data, n_out, n_in, scale, *dims)


@pytest.mark.parametrize("kind", OTHERS, ids=lambda k: O.KIND_NAMES[k])
# as above; 20,480 values do not fit beside the rings in every format, whose generic kernel takes them then
@pytest.mark.parametrize("shape", [(5, 256), (20, 768), (1201, 1280), (37, 14336), (19, 20480)])
def test_other_formats_of_one_to_four_tokens(backend, kind, shape):
    n_out, n_in = shape
    ref, m = other(kind, n_out, n_in, 940 + kind)
    dev = backend.upload(ref, n_out, n_in)
    w = m.dequantize_rows().astype(np.float64)
    x = (synth.activations(4, n_in, 941) * np.float32(1.2345)).astype(np.float32)
    one = np.concatenate([products(backend, dev, x[i : i + 1]) for i in range(4)])
    # (rows of up to 20,480 terms, summed in one slice by the generic kernel: sqrt(20480 / 32) f32 roundings per lane)
    assert row_err(one, x.astype(np.float64) @ w.T) < 4e-6
    for t in (2, 4):
        assert np.array_equal(products(backend, dev, x[:t]), one[:t])


@pytest.mark.parametrize("kind", OTHERS, ids=lambda k: O.KIND_NAMES[k])
def test_other_formats_as_a_pair_and_as_a_shard(backend, kind):
    n_out, n_in = 77, 768
    (g, gm), (u, um) = other(kind, n_out, n_in, 950), other(kind, n_out, n_in, 951)
    dg, du = backend.upload(g, n_out, n_in), backend.upload(u, n_out, n_in)
    x = synth.activations(3, n_in, 952)
    a, b = (x.astype(np.float64) @ m.dequantize_rows().astype(np.float64).T for m in (gm, um))
    x = (x / np.abs(a).max()).astype(np.float32)  # silu stays in range
    a, b = (x.astype(np.float64) @ m.dequantize_rows().astype(np.float64).T for m in (gm, um))
    y = np.zeros((3, n_out), np.float32)
    assert backend.matvec_rows(x, [ob.RowsJob(dg, y, du)])
    assert row_err(y, a / (1.0 + np.exp(-a)) * b) < 1e-5
    plain = products(backend, dg, x)
    assert np.array_equal(products(backend, backend.shard_rows(dg, 13, n_out), x), plain[:, 13:])


def f32_product(w, x):
    """W x as an f32 kernel adds it: 32 lanes take 16 values at a time, a sum from zero with a fused multiply-add each (the product of a
    weight of 4 and an activation of 24 bits is exact in f64), the lanes' sums in a tree."""
    n_out, n_in = w.shape
    steps = -(-n_in // 512)
    terms = np.zeros((n_out, steps * 512), np.float64)
    terms[:, :n_in] = w.astype(np.float64) * x.astype(np.float64)
    terms = terms.reshape(n_out, steps, 32, 16)
    acc = np.zeros((n_out, 32), np.float32)
    for s in range(steps):
        part = np.zeros((n_out, 32), np.float32)
        for j in range(16):
            part = (part + terms[:, s, :, j]).astype(np.float32)
        acc += part
    while acc.shape[1] > 1:
        acc = acc[:, : acc.shape[1] // 2] + acc[:, acc.shape[1] // 2 :]
    return acc[:, 0]


@pytest.mark.parametrize("n_in", [256, 1024, 2816, 14336])
@pytest.mark.parametrize("pair", [False, True])
def test_fp8_products_are_as_close_as_f32_ones(backend, n_in, pair):
    """The 2-norm of the error against f64 is no larger than an f32 product's."""
    n_out, tokens = 1024, 4
    refs = [make_pair("f8_e4m3", n_out, n_in, 980 + i) for i in range(2 if pair else 1)]
    devs, w = [backend.upload(r, n_out, n_in) for r, _ in refs], [m.dequantize_rows() for _, m in refs]
    x = synth.activations(tokens, n_in, 982)
    x /= np.abs(w[0] @ x.T).max()  # silu stays in range
    got, f32, want = [], [], []
    for v in x:
        y = torch.zeros(n_out, device="cuda")
        assert backend.matvec_dev(devs[0], torch.from_numpy(v).cuda(), y, ob.MODE_SILU_PAIR if pair else ob.MODE_STORE, devs[1] if pair else None)
        got.append(y.cpu().numpy())
        d = [f32_product(m, v) for m in w]
        f32.append(d[0] / (np.float32(1) + np.exp(-d[0])) * d[1] if pair else d[0])
        d = [m.astype(np.float64) @ v.astype(np.float64) for m in w]
        want.append(d[0] / (1.0 + np.exp(-d[0])) * d[1] if pair else d[0])
    error = lambda v: np.linalg.norm(np.stack(v) - np.stack(want))  # noqa: E731
    assert error(got) < error(f32)
