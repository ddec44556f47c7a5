"""A recorded FP64 device eval follows its handle through other evals of the handle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

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
