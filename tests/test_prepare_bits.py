"""The prepare kernels' exact results: neighbour lists of the FP32-screened kNN
and the Welford covariances by products of reciprocals equal the oracle's, bit
for bit, also where the screen's list overflows or leaves the FP32 range and
where the product form of the quotient hands over to the division."""
import numpy as np
import pytest

from test_gpu_parity import _gpu_dist, _orc_dist

pytestmark = pytest.mark.gpu


def _fixed(gpu, X, scale, local_frac):
    sd = _gpu_dist(gpu, 1, 0, X.shape[1], X=X, local_frac=local_frac,
                   cov_type=gpu.StatsDistKDECovType.FIXED, cov_fixed=np.eye(X.shape[1]) * scale)
    sd.prepare()
    return sd


@pytest.mark.parametrize("d,n,frac", [(1, 41, 0.1), (2, 1026, 0.05), (3, 130, 0.5), (7, 4099, 0.02), (2, 16387, 0.004),
                                      (16, 1025, 0.3), (32, 2051, 0.05)])
def test_knn_screen_sizes(gpu, oracle, d, n, frac):
    rng = np.random.default_rng(n + d)
    X = rng.standard_normal((n, d)) + 300.0
    X[n // 2] = 1e4 * rng.standard_normal(d)      # one far point widens the screen's error bound
    sd = _fixed(gpu, X, 1.0, frac)
    assert np.array_equal(sd.get_knn(), oracle.knn(X, sd.get_knn_k()))


@pytest.mark.parametrize("scale", [1.0, 1e60, 1e-60])
def test_knn_screen_overflow(gpu, oracle, scale):
    """Corners of a hypercube: hundreds of equal distances around the k-th, so
    some queries' lists overflow; scaled out of the FP32 range all of them go
    to the FP64 kernel."""
    rng = np.random.default_rng(5)
    X = rng.choice([-1.0, 1.0], size=(2400, 16))
    X = np.unique(X, axis=0)
    rng.shuffle(X)
    sd = _fixed(gpu, X, scale, 0.05)
    assert np.array_equal(sd.get_knn(), oracle.knn(X, sd.get_knn_k()))


@pytest.mark.parametrize("d", [1, 2, 3, 5, 8, 11, 16, 17, 27, 32])
@pytest.mark.parametrize("n", [97, 1300])
def test_covariance_bits(gpu, oracle, d, n):
    if n < 40 * d:
        n = 40 * d
    rng = np.random.default_rng(d)
    X = rng.standard_normal((n, d)) @ rng.standard_normal((d, d)) + 7.0
    o = _orc_dist(oracle, 1, 1, d, X=X)
    sd = _gpu_dist(gpu, 1, 1, d, X=X)
    assert o.prepare() == 0
    sd.prepare()
    assert np.array_equal(sd.peek_full_cov(), o.cov())
    assert np.array_equal(np.triu(sd.peek_full_cov_decomp()), np.triu(o.U()))
    assert np.array_equal(sd.get_knn(), o.knn())
    for i in list(range(0, n, max(1, n // 60))) + [n - 1]:
        assert np.array_equal(np.triu(sd.peek_cov_decomp(i)), np.triu(o.Ui(i))), i


def test_covariance_bits_tiny(gpu, oracle):
    """Coordinates whose differences lie below the product form's range."""
    rng = np.random.default_rng(2)
    X = rng.standard_normal((200, 2)) * np.array([1e-285, 1.0])
    X[:, 0] *= 1e-20
    want = oracle.welford_cov(X)
    sd = _gpu_dist(gpu, 0, 0, 2, X=X)
    try:
        sd.prepare()
    except gpu.NcgError:
        pass                                       # the covariance underflows: not positive definite
    else:
        assert np.array_equal(sd.peek_full_cov(), want)
    X = rng.standard_normal((200, 2)) * np.array([1e-140, 1.0]) + np.array([0.0, 1e9])
    sd = _gpu_dist(gpu, 0, 0, 2, X=X)
    sd.prepare()
    assert np.array_equal(sd.peek_full_cov(), oracle.welford_cov(X))
