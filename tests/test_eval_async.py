"""The FP64 device eval stays asynchronous and capturable right after a prepare, with the sliced
products' operand not built yet, and a recorded eval follows its handle: through a new prepare,
a weight fit and other evals of the handle."""
import time

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from conftest import rel_err
from test_eval_q64 import PLAIN_TOL, _plain
from test_gpu_parity import _gpu_dist

pytestmark = pytest.mark.gpu


def _setup(ng, d, n, m, kernel=1):
    rng = np.random.default_rng(d + m)
    sd = _gpu_dist(ng, 1, kernel, d, X=rng.standard_normal((n, d)))
    s = torch.cuda.Stream()
    sd.set_stream(s.cuda_stream)
    sd.prepare()
    P = rng.standard_normal((m, d))
    x = torch.from_numpy(P).cuda()
    out = torch.empty(m, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    return rng, sd, s, P, x, out


def _capture(sd, s, x, out):
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        sd.eval_m2lnp_device(x.data_ptr(), len(x), out.data_ptr())
    return g


def _replay(g, out):
    out.zero_()
    torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    return out.cpu().numpy()


def test_first_call_does_not_wait(gpu):
    _, sd, s, P, x, out = _setup(gpu, 6, 500, 1500)
    sd.eval_m2lnp_device(x.data_ptr(), len(x), out.data_ptr())     # buffers
    torch.cuda.synchronize()
    sd.prepare()
    with torch.cuda.stream(s):
        torch.cuda._sleep(int(4e8))                                # some 0.2 s of work before it
    t0 = time.perf_counter()
    sd.eval_m2lnp_device(x.data_ptr(), len(x), out.data_ptr())
    took = time.perf_counter() - t0
    busy = not s.query()
    torch.cuda.synchronize()
    assert busy and took < 0.05
    assert rel_err(out.cpu().numpy(), _plain(sd, P)) < PLAIN_TOL


@pytest.mark.parametrize("m", [300, 1500])
def test_capture_after_prepare(gpu, m):
    """No warm call between the prepare and the capture; the first one made the buffers."""
    rng, sd, s, P, x, out = _setup(gpu, 6, 500, m)
    sd.eval_m2lnp_device(x.data_ptr(), m, out.data_ptr())
    torch.cuda.synchronize()
    sd.set_sample(1.3 * rng.standard_normal((500, 6)))
    sd.prepare()
    g = _capture(sd, s, x, out)
    assert rel_err(_replay(g, out), _plain(sd, P)) < PLAIN_TOL


@pytest.mark.parametrize("warm", [False, True])
def test_replay_follows_the_handle(gpu, warm):
    """Recorded with and without the operand; then new fits and evals of other sizes."""
    rng, sd, s, P, x, out = _setup(gpu, 6, 500, 1500)
    sd.eval_m2lnp_device(x.data_ptr(), 1500, out.data_ptr())
    torch.cuda.synchronize()
    if not warm:
        sd.prepare()
    g = _capture(sd, s, x, out)
    for step in range(3):
        X = (1.0 + 0.1 * step) * rng.standard_normal((500, 6))
        sd.set_sample(X)
        sd.prepare_interp(np.sum(X ** 2, axis=1)) if step == 1 else sd.prepare()
        for _ in range(2):
            assert rel_err(_replay(g, out), _plain(sd, P)) < PLAIN_TOL
            sd.eval_m2lnp(P[:700])                                 # sliced products, smaller
            sd.eval_m2lnp(P[:300])                                 # tiles


def test_replay_on_another_stream_after_prepare(gpu):
    """The operand of a recorded eval is complete when a prepare returns."""
    rng, sd, s, P, x, out = _setup(gpu, 16, 4000, 1500)
    sd.eval_m2lnp_device(x.data_ptr(), 1500, out.data_ptr())
    torch.cuda.synchronize()
    g = _capture(sd, s, x, out)
    other = torch.cuda.Stream()
    for _ in range(3):
        sd.set_sample(rng.standard_normal((4000, 16)))
        torch.cuda.synchronize()
        sd.prepare()
        with torch.cuda.stream(other):
            g.replay()
        torch.cuda.synchronize()
        assert rel_err(out.cpu().numpy(), _plain(sd, P)) < PLAIN_TOL


def test_plain_capture_keeps_its_scratch(gpu):
    """A recorded tile eval and later sliced-product evals of the same handle."""
    _, sd, s, P, x, out = _setup(gpu, 6, 500, 300)
    sd.eval_m2lnp_device(x.data_ptr(), 300, out.data_ptr())
    torch.cuda.synchronize()
    g = _capture(sd, s, x, out)
    want = _replay(g, out)
    sd.eval_m2lnp(np.resize(P, (2000, 6)))
    guard = [torch.full((k * 1024,), 7.0, dtype=torch.float64, device="cuda") for k in (16, 64, 256, 512, 1024) * 4]
    assert np.array_equal(_replay(g, out), want)
    assert all(bool((b == 7.0).all()) for b in guard)


@pytest.mark.parametrize("kernel", [0, 1])
def test_operand_out_of_range(gpu, kernel):
    """Kernels too narrow for the fixed point: first call (range not known yet), host call (known)."""
    rng = np.random.default_rng(5)
    d, n = 5, 600
    X = rng.standard_normal((n, d))
    X[: n // 2] = 3.0 + X[: n // 2] * 1e-7
    P = np.concatenate([X[::2] + 0.3e-7 * rng.standard_normal((n // 2, d)), rng.standard_normal((400, d))])
    sd = _gpu_dist(gpu, 1, kernel, d, X=X)
    sd.prepare()
    x = torch.from_numpy(P).cuda()
    out = torch.empty(len(P), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    sd.eval_m2lnp_device(x.data_ptr(), len(P), out.data_ptr())
    sd.synchronize()
    first, host = out.cpu().numpy(), sd.eval_m2lnp(P)
    assert np.array_equal(first, host)
    assert rel_err(host, _plain(sd, P), floor=1.0) < PLAIN_TOL


def test_replay_with_an_operand_out_of_range(gpu):
    """Recorded within the range, replayed after a fit that leaves it, and back."""
    rng, sd, s, P, x, out = _setup(gpu, 6, 500, 700)
    sd.eval_m2lnp_device(x.data_ptr(), 700, out.data_ptr())
    torch.cuda.synchronize()
    g = _capture(sd, s, x, out)
    for scale in (1e-7, 1.0):
        X = rng.standard_normal((500, 6))
        X[:250] = 3.0 + scale * X[:250]
        sd.set_sample(X)
        sd.prepare()
        assert np.array_equal(_replay(g, out), sd.eval_m2lnp(P))
