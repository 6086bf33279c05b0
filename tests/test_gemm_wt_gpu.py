"""Products of more than eight tokens and the routed experts' segments: weights in tensor memory, tokens on the instruction's N side."""
import os

import numpy as np
import pytest
import torch

import oxinfer_b200 as ob
from oxinfer_b200 import synth

from util import make_pair, oracle_matrix, row_err

pytestmark = pytest.mark.gpu


# token counts around the steps of 16 and the change of the accumulator's width at 64; row counts around the tiles of 128; one super-block,
# an odd number of them, the first K that is divided (2 parts), 4 parts and 8 unequal ones; short K whose larger batch runs with tokens on M (all
# formats, Q6_K, all but Q6_K)
@pytest.mark.parametrize("fmt", ["mlx4", "q4_k", "q6_k", "q8_0", "f8_e4m3"])
@pytest.mark.parametrize("shape", [(127, 256, 9), (128, 768, 16), (130, 2816, 17), (260, 3072, 64), (384, 6400, 65), (1001, 12544, 37), (257, 12288, 128),
                                   (130, 256, 100), (300, 1024, 128), (31000, 256, 113)])
def test_products_of_up_to_128_tokens(backend, fmt, shape):
    """f16 operands with f32 sums: 1e-3 of a row (tests/test_gemm_gpu.py). A row shard has the bits of its rows, and a token of a smaller
    batch the bits of the larger one's, f32 in place of the strided or bf16 results of the other entry points included."""
    n_out, n_in, t = shape
    ref, m = make_pair(fmt, n_out, n_in, 900 + t)
    dev = backend.upload(ref, n_out, n_in)
    x = synth.activations(t, n_in, 901)
    y = np.full((t, n_out), np.nan, np.float32)
    assert backend.matmul(x, [ob.Job(dev, y)])
    assert row_err(y, m.matmul_f64(x)) < 1e-3
    if n_out > 128:
        shard = backend.shard_rows(dev, 128, n_out)
        ys = np.zeros((t, n_out - 128), np.float32)
        assert backend.matmul(x, [ob.Job(shard, ys)])
        assert np.array_equal(ys, y[:, 128:])
    y9 = np.zeros((9, n_out), np.float32)
    assert backend.matmul(x[t - 9 :], [ob.Job(dev, y9)])
    assert np.array_equal(y9, y[t - 9 :])
    xd, yd = torch.from_numpy(x).cuda(), torch.zeros((t, n_out), device="cuda", dtype=torch.bfloat16)
    assert backend.matmul_dev(dev, xd, yd)
    torch.cuda.synchronize()
    backend.check_status()
    assert torch.equal(yd.cpu(), torch.from_numpy(y).bfloat16())


# one token and one unit of 32 past what the smaller kernel takes, one segment of 32 to 128 tokens a pair (longer ones and several a pair:
# test_several_segments_a_pair; the smallest shape runs with tokens on M), rows that end inside a pair's 256 and inside a CTA's 128, an odd number of super-blocks
@pytest.mark.parametrize("fmt", ["mlx4", "q4_k", "q6_k", "q8_0", "f8_e4m3"])
@pytest.mark.parametrize("shape", [(200, 256, 129), (333, 768, 161), (1000, 512, 257), (2100, 1280, 300), (512, 2048, 700)])
def test_products_of_more_tokens(backend, fmt, shape):
    """f16 operands with f32 sums: 1e-3 of a row (tests/test_gemm_gpu.py). A row shard, which may run in other segments or on the form with
    tokens on M, has the bits of its rows, and a bf16 result is the f32 one rounded."""
    n_out, n_in, t = shape
    ref, m = make_pair(fmt, n_out, n_in, 940 + t)
    dev = backend.upload(ref, n_out, n_in)
    x = synth.activations(t, n_in, 941)
    y = np.full((t, n_out), np.nan, np.float32)
    assert backend.matmul(x, [ob.Job(dev, y)])
    assert row_err(y, m.matmul_f64(x)) < 1e-3
    shard = backend.shard_rows(dev, 128, n_out)
    ys = np.zeros((t, n_out - 128), np.float32)
    assert backend.matmul(x, [ob.Job(shard, ys)])
    assert np.array_equal(ys, y[:, 128:])
    xd, yd = torch.from_numpy(x).cuda(), torch.zeros((t, n_out), device="cuda", dtype=torch.bfloat16)
    assert backend.matmul_dev(dev, xd, yd)
    torch.cuda.synchronize()
    backend.check_status()
    assert torch.equal(yd.cpu(), torch.from_numpy(y).bfloat16())


def with_tokens_on_m(backend, x, dev, n_out):
    """The same product on gemm_tc.cu's form (any B2_GEMM_SPLIT_K but 1; 0 divides nothing)."""
    y = np.full((len(x), n_out), np.nan, np.float32)
    os.environ["B2_GEMM_SPLIT_K"] = "0"
    try:
        assert backend.matmul(x, [ob.Job(dev, y)])
    finally:
        del os.environ["B2_GEMM_SPLIT_K"]
    return y


# several segments a pair whose 10 or 22 groups of 64 k are not whole fours: the sets of dequantizers and the 12 staging slots go on over them
@pytest.mark.parametrize("fmt", ["q8_0", "f8_e4m3"])
@pytest.mark.parametrize("shape", [(20000, 640, 300), (3000, 1408, 3108)])
def test_byte_rows_that_end_inside_a_round_of_the_sets(backend, fmt, shape):
    """The bits of the form with tokens on M, and 1e-3 of a row (tests/test_gemm_gpu.py) on a sample of the tokens."""
    n_out, n_in, t = shape
    ref, m = make_pair(fmt, n_out, n_in, 960 + t)
    dev = backend.upload(ref, n_out, n_in)
    x = synth.activations(t, n_in, 961)
    y = np.full((t, n_out), np.nan, np.float32)
    assert backend.matmul(x, [ob.Job(dev, y)])
    rows = np.arange(0, t, 97)
    assert row_err(y[rows], m.matmul_f64(x[rows])) < 1e-3
    assert np.array_equal(y, with_tokens_on_m(backend, x, dev, n_out))


# equal runs of three segments of 64 to 256 tokens; 12 token ranges (a panel of eight and the rest) by 14 row blocks, the last 20 of 168 segments in
# two parts each; rows that end inside a pair's 256
@pytest.mark.parametrize("fmt", ["mlx4", "q4_k", "q6_k", "q8_0", "f8_e4m3"])
@pytest.mark.parametrize("shape", [(3000, 1536, 3108), (3400, 768, 2850)])
def test_several_segments_a_pair(backend, fmt, shape):
    """The bits of the form with tokens on M, and 1e-3 of a row (tests/test_gemm_gpu.py) on a sample of the tokens."""
    n_out, n_in, t = shape
    ref, m = make_pair(fmt, n_out, n_in, 970 + t)
    dev = backend.upload(ref, n_out, n_in)
    x = synth.activations(t, n_in, 971)
    y = np.full((t, n_out), np.nan, np.float32)
    assert backend.matmul(x, [ob.Job(dev, y)])
    rows = np.arange(0, t, 97)
    assert row_err(y[rows], m.matmul_f64(x[rows])) < 1e-3
    assert np.array_equal(y, with_tokens_on_m(backend, x, dev, n_out))


# pairs per expert: none, one, a tile of 16 and one more, 128 and one more (two tiles of 80 and 49 rows), three tiles; 45 experts in 51 tiles
# (MLX-4: 44), so that a pair of CTAs takes two or three segments of the gate / up projection (204) and one or two of the down projection (102) in turn
COUNTS = [([1, 16, 0, 17, 128, 129, 300, 64], 256, 512), ([70], 2048, 768), ([29 * i % 150 for i in range(45)], 512, 512)]


def expert_rows(backend, fmt, counts, h, inter):
    """(result, f64 result) of the pairs of each expert that has some."""
    n = len(counts)
    refs = [(synth.make(fmt, 2 * inter, h, 920 + 2 * e), synth.make(fmt, h, inter, 921 + 2 * e)) for e in range(n)]
    moe = backend.upload_moe([backend.upload(g, 2 * inter, h) for g, _ in refs], [backend.upload(d, h, inter) for _, d in refs], h, inter)
    flat = np.random.default_rng(922).permutation(np.repeat(np.arange(n, dtype=np.int32), counts))
    x = synth.activations(len(flat), h, 923)
    y = torch.zeros((len(flat), h), device="cuda")
    assert backend.moe_dev(torch.from_numpy(x).cuda(), flat.reshape(-1, 1), np.ones((len(flat), 1), np.float32), moe, y)
    torch.cuda.synchronize()
    backend.check_status()
    for e, (g, d) in enumerate(refs):
        rows = np.flatnonzero(flat == e)
        if len(rows) == 0:
            continue
        gu = oracle_matrix(g, 2 * inter, h).matmul_f64(x[rows])
        a = gu[:, :inter] / (1.0 + np.exp(-gu[:, :inter])) * gu[:, inter:]
        yield y[torch.from_numpy(rows).cuda()].cpu().numpy(), a @ oracle_matrix(d, h, inter).dequantize_rows().astype(np.float64).T


@pytest.mark.parametrize("fmt", ["mlx4", "q4_k"])
@pytest.mark.parametrize("counts,h,inter", COUNTS)
def test_segments_of_every_length(backend, fmt, counts, h, inter):
    for got, want in expert_rows(backend, fmt, counts, h, inter):
        assert row_err(got, want) < 1e-3


@pytest.mark.parametrize("counts,h,inter", COUNTS)
def test_exact_segments_of_mlx4(backend, counts, h, inter):
    """Two-term activations on one-term weights run on gemm_wt.cu, tiles of up to 128 rows of an expert: the exact switch's 1e-4
    (tests/test_gemm_gpu.py), which one-term activations miss (2.8e-4 and more on these layers)."""
    backend.set_exact(True)
    try:
        for got, want in expert_rows(backend, "mlx4", counts, h, inter):
            assert row_err(got, want) < 1e-4
    finally:
        backend.set_exact(False)


def test_a_first_q6_k_product_inside_a_capture(backend):
    """A product with tokens on M allocates and copies nothing when its weights and buffers come up for the first time: it can be captured."""
    n_out, n_in, t = 300, 1024, 128
    devs = [backend.upload(make_pair("q6_k", n_out, n_in, 990 + i)[0], n_out, n_in) for i in range(2)]
    x = torch.from_numpy(synth.activations(t, n_in, 992)).cuda()
    y, want = torch.zeros((2, t, n_out), device="cuda"), torch.zeros((t, n_out), device="cuda")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    backend.set_stream(stream.cuda_stream)
    try:
        assert backend.matmul_dev(devs[0], x, y[0])  # (scratch for this batch)
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            assert backend.matmul_dev(devs[1], x, y[1])
        graph.replay()
        assert backend.matmul_dev(devs[1], x, want)
        torch.cuda.synchronize()
        backend.check_status()
    finally:
        backend.set_stream(0)
    assert torch.equal(y[1], want) and not torch.equal(y[0], want)
