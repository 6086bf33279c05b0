"""The small-batch products (one to eight tokens, gemv_mma.cu) where tiles, rounds and parts of K end unevenly.

Bound: an activation keeps 23 bits of the largest value of its block of 256 (2^-24 of it at most is lost per value) and a row's sums
are f32 sums in at most eight slices, each of K / 8 / 32 terms or fewer: 2e-6 of a row of N(0, 1) activations covers K = 14336.
"""
import numpy as np
import pytest
import torch

import oxinfer_b200 as ob
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
