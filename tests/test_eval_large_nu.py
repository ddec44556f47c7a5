"""Student-t kernels with many degrees of freedom in every FP64 form: ln K = -(nu + d) / 2
log (1 + chi^2 / nu) keeps its accuracy where chi^2 / nu is far below 1.  Compared with the
oracle by differences of -2 ln p between points, since the constant of the kernels
(lgamma differences) loses digits at such nu and is common to all points.  The bound: chi^2 of
some 30 with unit covariances is rounded 3 d times or so at 2^-53 (2e-13 at d = 16), the same on
both sides, and the sums and the logarithm add a few units of the result (1e-14 each)."""
import numpy as np
import pytest

from test_gpu_parity import _gpu_dist, _orc_dist

pytestmark = pytest.mark.gpu

TOL = 2e-12


# few-point kernel, tiles, sliced products (VKDE from 640 points)
@pytest.mark.parametrize("m", [7, 200, 700])
@pytest.mark.parametrize("kind,d", [(0, 2), (0, 9), (1, 6), (1, 16)])
@pytest.mark.parametrize("nu", [9.0, 1e3, 1e6, 1e9])
def test_large_nu(gpu, oracle, nu, kind, d, m):
    rng = np.random.default_rng(d + m)
    X, P = rng.standard_normal((80 * d + 300, d)), 1.2 * rng.standard_normal((m, d))
    o = _orc_dist(oracle, kind, 1, d, nu=nu, X=X, **({"local_frac": 0.3} if kind else {}))
    sd = _gpu_dist(gpu, kind, 1, d, nu=nu, X=X, **({"local_frac": 0.3} if kind else {}))
    assert o.prepare() == 0
    sd.prepare()
    want, got = o.eval_m2lnp(P), sd.eval_m2lnp(P)
    assert np.max(np.abs((got - got[0]) - (want - want[0]))) < TOL
    b = gpu.Batch()
    b.add(sd, m)
    g = b.eval_m2lnp([P])[0]
    assert np.max(np.abs((g - g[0]) - (want - want[0]))) < TOL
