"""4-bit and Q8_0 products of one to eight tokens on the tensor cores (`dmv_*`, `dmvk_*`, src/cuda_decode.cu:139-232) at the edges of their tiles (128 rows, 64 of
a pair), of the four parts of K and the sets' blocks, and over several rounds of the clusters."""
import numpy as np
import pytest

import oxinfer_b200 as ob
from oracle import oracle as O
from oxinfer_b200 import synth

from test_gemv_gpu import TIGHT, make_pair
from util import row_err

pytestmark = pytest.mark.gpu

# rows, K: parts without a block (one and two blocks), with unequal numbers, more blocks than sets; one row, tiles' edges, several tiles a cluster
SHAPES = [(1, 256), (129, 512), (65, 768), (127, 1280), (64, 1024), (300, 5120), (128, 16640), (5000, 1024), (9300, 2560)]


@pytest.mark.parametrize("fmt", ["q4_k", "mlx4", "q8_0"])
@pytest.mark.parametrize("n_out,n_in", SHAPES)
def test_tiles_parts_and_tokens(backend, fmt, n_out, n_in):
    ref, m = make_pair(fmt, n_out, n_in, 500 + n_in % 97)
    up, mu = make_pair(fmt, n_out, n_in, 900 + n_in % 89)
    dev, du = backend.upload(ref, n_out, n_in), backend.upload(up, n_out, n_in)
    x = synth.activations(8, n_in, 501)
    ones, pairs = np.zeros((8, n_out), np.float32), np.zeros((8, n_out), np.float32)
    for i in range(8):
        assert backend.matvec_rows(x[i:i + 1], [ob.RowsJob(dev, ones[i:i + 1])])
        assert backend.matvec_rows(x[i:i + 1], [ob.RowsJob(dev, pairs[i:i + 1], up=du)])
    assert row_err(ones, m.matmul_f64(x)) < TIGHT
    g, u = m.matmul_f64(x), mu.matmul_f64(x)
    # (the activation multiplies the errors of both products and rounds its exponential: the bound of the pair's other tests)
    assert row_err(pairs, g / (1.0 + np.exp(-g)) * u) < 1e-4
    for t in (2, 3, 4):
        y, yp = np.full((t, n_out), np.nan, np.float32), np.full((t, n_out), np.nan, np.float32)
        assert backend.matvec_rows(x[:t], [ob.RowsJob(dev, y), ob.RowsJob(dev, yp, up=du)])
        assert np.array_equal(y, ones[:t]) and np.array_equal(yp, pairs[:t]), t
    for t in (5, 8):  # from records, a launch per four rows (from the rows themselves: below)
        y = np.full((t, n_out), np.nan, np.float32)
        assert backend.matmul(x[:t], [ob.Job(dev, y)])
        assert np.array_equal(y, ones[:t]), t


@pytest.mark.parametrize("fmt", ["q4_k", "mlx4", "q8_0"])
def test_device_rows_and_row_shards_have_the_whole_matrix_bits(backend, fmt):
    torch = pytest.importorskip("torch")
    n_out, n_in = 700, 2560
    ref, m = make_pair(fmt, n_out, n_in, 611)
    dev = backend.upload(ref, n_out, n_in)
    x = synth.activations(7, n_in, 612)
    ones = np.zeros((7, n_out), np.float32)
    for i in range(7):
        assert backend.matvec_rows(x[i:i + 1], [ob.RowsJob(dev, ones[i:i + 1])])
    backend.set_stream(torch.cuda.current_stream().cuda_stream)
    try:
        xd = torch.from_numpy(x).cuda()
        for t in (2, 4, 5, 7):
            y = torch.full((t, n_out), float("nan"), device="cuda")
            assert backend.matmul_dev(dev, xd[:t].contiguous(), y)
            assert np.array_equal(y.cpu().numpy(), ones[:t]), t
        # results over the rows they are made of (the entry point then reads a copy)
        both = torch.zeros(4, max(n_in, n_out), device="cuda").reshape(-1)
        both[: 4 * n_in] = xd[:4].reshape(-1)
        xs, ys = both[: 4 * n_in].view(4, n_in), both[: 4 * n_out].view(4, n_out)
        assert backend.matmul_dev(dev, xs, ys)
        assert np.array_equal(ys.cpu().numpy(), ones[:4])
    finally:
        backend.set_stream(0)


@pytest.mark.parametrize("fmt", ["q4_k", "mlx4"])
@pytest.mark.parametrize("t", [1, 2, 3, 4])
def test_matrices_of_one_call_share_a_launch_and_keep_their_bits(backend, fmt, t):
    """Row counts at the edges of the tiles; more than four matrices, a pair or another format among them take launches of their own; results that do
    not fit the page-locked stage (256 KB)."""
    n_in = 1280
    outs = [1, 128, 129, 300, 33000]
    devs = [backend.upload(make_pair(fmt, n, n_in, 700 + n % 89)[0], n, n_in) for n in outs]
    other = backend.upload(make_pair("q8_0", 96, n_in, 790)[0], 96, n_in)
    x = synth.activations(t, n_in, 701)

    def run(ds, ns, ups=None):
        ys = [np.full((t, n), np.nan, np.float32) for n in ns]
        before = backend.launch_count()
        assert backend.matvec_rows(x, [ob.RowsJob(d, y, up=u) for d, y, u in zip(ds, ys, ups or [None] * len(ds))])
        return ys, backend.launch_count() - before

    alone = [run([d], [n])[0][0] for d, n in zip(devs, outs)]
    for pick, launches in (((0, 1), 1), ((3, 0, 2), 1), ((2, 4, 1, 0), 1), ((0, 1, 2, 3, 4), 5)):
        ys, count = run([devs[k] for k in pick], [outs[k] for k in pick])
        assert count == launches
        for k, y in zip(pick, ys):
            assert np.array_equal(y, alone[k]), (pick, k)
    pair = run([devs[1]], [128], [devs[1]])[0][0]
    ys, _ = run([devs[1], devs[2], other], [128, 129, 96], [devs[1], None, None])
    assert np.array_equal(ys[0], pair) and np.array_equal(ys[1], alone[2]) and np.isfinite(ys[2]).all()
