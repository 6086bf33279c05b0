"""What the host side does when a kernel's bounded wait has given up: the mark is left from the host (nothing runs into a limit here). The call that finds it
fails with B2_ERR_TIMEOUT and leaves y alone, whatever the results' size ("in both non-zero cases no output was written"), and the next call works."""
import numpy as np
import pytest

import oxinfer_b200 as ob
from oxinfer_b200 import synth
from oxinfer_b200._lib import ERR_TIMEOUT

from test_gemv_gpu import make_pair
from test_plan_multi_gpu import rope_rows, two_plans

pytestmark = pytest.mark.gpu

K = 512
# rows per matrix; results of t = 4 rows within the page-locked stage (256 KB), a part (128 KB) and odd bytes behind it, several parts, a job over parts' edges
JOBS = [(96,), (300, 129), (16385,), (24000, 1, 9000), (65, 40000, 33, 20000)]


@pytest.mark.parametrize("fmt", ["q4_k", "mlx4", "q8_0", "q6_k"])
@pytest.mark.parametrize("outs", JOBS, ids=str)
def test_host_products_leave_their_results_alone(backend, fmt, outs):
    devs = [backend.upload(make_pair(fmt, n, K, 30 + n % 83)[0], n, K) for n in outs]
    x = synth.activations(12, K, 31)
    for t in (1, 4, 12):
        rows = t <= 4
        ys = [np.full((t, n), np.nan, np.float32) for n in outs]
        jobs = [ob.RowsJob(d, y) if rows else ob.Job(d, y) for d, y in zip(devs, ys)]
        call = lambda: (backend.matvec_rows if rows else backend.matmul)(x[:t], jobs)
        assert call()
        want = [y.copy() for y in ys]
        for y in ys:
            y.fill(7.0)
        backend.inject_timeout()
        with pytest.raises(ob.BackendError) as e:
            call()
        assert e.value.code == ERR_TIMEOUT and all((y == 7.0).all() for y in ys), t
        assert call() and all(np.array_equal(y, w) for y, w in zip(ys, want)), t
        one = np.zeros((t, outs[-1]), np.float32)  # (the same product by itself)
        assert (backend.matvec_rows(x[:t], [ob.RowsJob(devs[-1], one)]) if rows else backend.matmul(x[:t], [ob.Job(devs[-1], one)])) and np.array_equal(one, want[-1])


def test_device_calls_report_it_when_asked(backend):
    backend.inject_timeout()
    with pytest.raises(ob.BackendError) as e:
        backend.check_status()
    assert e.value.code == ERR_TIMEOUT
    backend.check_status()


def test_plan_steps_report_it_and_go_on(backend):
    cfg = dict(n_layers=1, h=256, nh=4, nkv=2, hd=64, inter=256, vocab=256)
    one, many, inv_freq, _, keep = two_plans(backend, cfg, seed=1600, max_len=64)
    xs = np.random.default_rng(82).standard_normal((3, cfg["h"])).astype(np.float32)
    cs = rope_rows(0, 3, inv_freq)
    for step, plan in ((lambda: one.step(0, xs[0], cs[0]), one), (lambda: many.step_multi(0, xs, cs), many)):
        want = step()
        backend.inject_timeout(plan)
        with pytest.raises(ob.BackendError) as e:
            step()
        assert e.value.code == ERR_TIMEOUT
        got = step()
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    one.close()
    many.close()
