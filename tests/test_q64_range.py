"""The sliced products hold chi^2 in a fixed point of the sample's scale: points (and kernels) far
outside it take the plain form inside the same call.  Against the plain kernels, to 1e-14
relative (test_eval_q64.py: 100 units of both forms' roundings)."""
import numpy as np
import pytest

from conftest import rel_err
from test_eval_q64 import PLAIN_TOL, _plain
from test_gpu_parity import FP64_TOL, _gpu_dist

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [0, 1])
def test_outlying_kernels(gpu, kernel):
    """Global coordinates by a fixed covariance: a group of kernels hundreds of widths out."""
    ng = gpu
    rng = np.random.default_rng(21)
    d, n = 6, 600
    X = rng.standard_normal((n, d))
    X[:60] = 150.0 + 0.2 * X[:60]
    P = np.concatenate([X[:60] + 0.1 * rng.standard_normal((60, d)) for _ in range(5)] + [rng.standard_normal((400, d))])
    sd = _gpu_dist(ng, 1, kernel, d, X=X, cov_type=ng.StatsDistKDECovType.FIXED, cov_fixed=np.eye(d))
    sd.prepare()
    # (-2 ln p crosses zero)
    assert rel_err(sd.eval_m2lnp(P), _plain(sd, P), floor=3.0) < PLAIN_TOL


@pytest.mark.parametrize("kernel,nu", [(0, 3.0), (1, 3.0), (1, 500.0)])
@pytest.mark.parametrize("d,n,m", [(5, 384, 640), (16, 1009, 700), (17, 1021, 8192 + 100), (32, 1700, 641)])
def test_far_points(gpu, kernel, nu, d, n, m):
    """None, some, a whole tile and nearly all of a call's points far out; the last one too."""
    rng = np.random.default_rng(d)
    X, P = rng.standard_normal((n, d)), rng.standard_normal((m, d))
    sd = _gpu_dist(gpu, 1, kernel, d, nu=nu, X=X, local_frac=0.1)
    sd.prepare()
    near = sd.eval_m2lnp(P)
    for far in (np.array([m - 1]), np.arange(0, m, 37), np.arange(96, 160), np.arange(1, m)):
        Q = P.copy()
        Q[far] *= 10.0 ** rng.uniform(3, 6, (len(far), 1))
        got = sd.eval_m2lnp(Q)
        assert rel_err(got, _plain(sd, Q)) < PLAIN_TOL
        keep = np.setdiff1d(np.arange(m), far)
        assert np.array_equal(got[keep], near[keep])
    assert rel_err(sd.eval(Q), np.exp(-0.5 * got), floor=1e-300) < FP64_TOL
