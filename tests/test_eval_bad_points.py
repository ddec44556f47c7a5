"""Points without a density (a NaN or infinite coordinate on the device, or finite ones so
far out that chi^2 leaves FP64) in every FP64 form: no kernel counts, -2 ln p = +inf, and
the other points of the call keep their values."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from test_gpu_parity import _gpu_dist

pytestmark = pytest.mark.gpu


def _dev(sd, P):
    x = torch.tensor(P, dtype=torch.float64, device="cuda")
    out = torch.empty(len(P), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    sd.eval_m2lnp_device(x.data_ptr(), len(P), out.data_ptr())
    sd.synchronize()
    return out.cpu().numpy()


# few-point kernel, tiles, sliced products (VKDE)
@pytest.mark.parametrize("m", [5, 60, 700])
@pytest.mark.parametrize("d", [5, 8])
@pytest.mark.parametrize("kernel", [0, 1])
@pytest.mark.parametrize("kind", [0, 1])
def test_bad_points(gpu, kind, kernel, d, m):
    rng = np.random.default_rng(10 * d + m)
    X, P = rng.standard_normal((500, d)), rng.standard_normal((m, d))
    sd = _gpu_dist(gpu, kind, kernel, d, X=X)
    sd.prepare()
    want = _dev(sd, P)
    bad = np.array([0, 1, 3, m - 1])
    P[bad, [1, 0, d - 1, 2]] = np.nan, np.inf, -np.inf, 1e200
    got = _dev(sd, P)
    assert np.all(np.isposinf(got[bad]))
    keep = np.setdiff1d(np.arange(m), bad)
    assert np.array_equal(got[keep], want[keep])
    # the host entry takes the finite one
    assert np.isposinf(sd.eval_m2lnp(np.vstack([P[keep], P[m - 1:]]))[-1])
    b = gpu.Batch()
    b.add(sd, m)
    g = b.eval_m2lnp([P])[0]
    assert np.all(np.isposinf(g[bad])) and np.all(np.isfinite(g[keep]))
