"""Products of two to eight tokens (`dmvk_*`, src/cuda_decode.cu:176-232) whose CTAs split the activations themselves, and the ones over records, on both sides of
the lines between them and between the forms: every row has the bits of its one-token product."""
import numpy as np
import pytest

import oxinfer_b200 as ob
from oxinfer_b200 import synth

from test_gemv_gpu import TIGHT, make_pair
from util import FORMATS, row_err

pytestmark = pytest.mark.gpu


# 256 .. 1024: short rows (1024: 32 blocks of eight tokens); 1280: five blocks (six tokens split by the product, seven not); 4096: two tokens and three
@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("n_out,n_in", [(33, 256), (300, 768), (257, 1024), (130, 1280), (96, 4096)])
def test_rows_keep_their_bits_with_and_without_records(backend, fmt, n_out, n_in):
    torch = pytest.importorskip("torch")
    ref, m = make_pair(fmt, n_out, n_in, 40 + n_in % 61)
    dev = backend.upload(ref, n_out, n_in)
    x = synth.activations(8, n_in, 41)
    ones = np.zeros((8, n_out), np.float32)
    for i in range(8):
        assert backend.matvec_rows(x[i:i + 1], [ob.RowsJob(dev, ones[i:i + 1])])
    assert row_err(ones, m.matmul_f64(x)) < TIGHT
    backend.set_stream(torch.cuda.current_stream().cuda_stream)
    try:
        xd = torch.from_numpy(x).cuda()
        for t in range(1, 9):
            y = torch.full((t, n_out), float("nan"), device="cuda")
            assert backend.matmul_dev(dev, xd[:t].contiguous(), y)
            assert np.array_equal(y.cpu().numpy(), ones[:t]), t
    finally:
        backend.set_stream(0)
    for t in (2, 3, 4):
        y, z = np.full((t, n_out), np.nan, np.float32), np.full((t, n_out), np.nan, np.float32)
        assert backend.matvec_rows(x[:t], [ob.RowsJob(dev, y), ob.RowsJob(dev, z)])
        assert np.array_equal(y, ones[:t]) and np.array_equal(z, ones[:t]), t
    for t in (5, 8):
        y = np.full((t, n_out), np.nan, np.float32)
        assert backend.matmul(x[:t], [ob.Job(dev, y)])
        assert np.array_equal(y, ones[:t]), t


# one, two, three and four blocks of activations, and five (the form on tcgen05 for every call)
@pytest.mark.parametrize("fmt", ["q4_k", "mlx4"])
@pytest.mark.parametrize("n_in", [256, 512, 768, 1024, 1280])
def test_jobs_of_short_rows_have_the_bits_of_each_by_itself(backend, fmt, n_in):
    """Several matrices of a call may share a launch of the other form; extreme activations, whose sums round everywhere, among them."""
    outs = [1, 129, 700, 64]
    devs = [backend.upload(make_pair(fmt, n, n_in, 60 + n % 53)[0], n, n_in) for n in outs]
    for seed, scale in ((71, 1.0), (72, 1e6), (73, 1e-6)):
        x = synth.activations(4, n_in, seed) * np.float32(scale)
        x[:, ::97] *= 1000.0
        for t in (1, 2, 4):
            alone = [np.full((t, n), np.nan, np.float32) for n in outs]
            for d, y in zip(devs, alone):
                assert backend.matvec_rows(x[:t], [ob.RowsJob(d, y)])
            ys = [np.full((t, n), np.nan, np.float32) for n in outs]
            assert backend.matvec_rows(x[:t], [ob.RowsJob(d, y) for d, y in zip(devs, ys)])
            for a, y in zip(alone, ys):
                assert np.array_equal(a, y), (scale, t, a.shape)
