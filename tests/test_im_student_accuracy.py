"""Elements of the Student-t interpolation matrix far out in the kernels' tails, against the same
power in extended precision.  (1 + chi^2 / nu)^kappa carries kappa times the relative error of
chi^2: coordinates and bandwidth are rounded some five times, so 2 * 5 units of 2^-53, and the
power itself adds about 2; the logarithm, 60 there, must not."""
import numpy as np
import pytest

from test_gpu_parity import _gpu_dist

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [0, 1])
def test_tail_elements(gpu, kind):
    ng = gpu
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip("no extended precision here")
    rng = np.random.default_rng(2)
    nu, n = 3.0, 96
    X = 1e3 * rng.standard_normal((n, 1))
    if kind:   # pairs: tight local covariances of their own
        X[1::2] = X[::2] + 1e-10 * rng.standard_normal((n // 2, 1))
    sd = _gpu_dist(ng, kind, 1, 1, nu=nu, X=X, cov_type=ng.StatsDistKDECovType.FIXED, cov_fixed=np.array([[1e-20]]),
                   **({"local_frac": 2.5 / n} if kind else {}))
    sd.prepare()
    IM = sd.compute_IM()                                        # observations x kernels
    L = np.longdouble
    u = np.array([sd.peek_cov_decomp(i)[0, 0] if kind else sd.peek_full_cov_decomp()[0, 0] for i in range(n)])
    x = X[:, 0].astype(L)
    chi2 = ((x[:, None] - x[None, :]) / (u.astype(L) * L(sd.get_href()))[None, :]) ** 2
    K = (1 + chi2 / L(nu)) ** L(-0.5 * (nu + 1))
    got = IM / np.diag(IM)[None, :]                             # K = 1 there
    far = (chi2 > 1e12) & (np.abs(x[:, None] - x[None, :]) > 0.5 * np.maximum(np.abs(x)[:, None], np.abs(x)[None, :]))
    assert far.sum() > n
    err = np.abs(got[far].astype(L) / K[far] - 1)
    assert err.max() < (0.5 * (nu + 1) * 10 + 4) * 2.0 ** -53
