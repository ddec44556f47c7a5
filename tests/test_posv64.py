"""The FP64 weight fit on sliced tensor-core products at the edges of its tiles:
systems around multiples of the 32-row panels, the 32- and 128-column tiles
and more tiles than SMs, against the oracle (weights <= 1e-10 of the largest, the
FP64 form's bound) or, where the oracle would take long, against the mixed form's
conjugate gradients on the same matrix (1e-10 as well)."""
import numpy as np
import pytest

from test_gpu_parity import FP64_TOL, _gpu_dist, _orc_dist

pytestmark = pytest.mark.gpu


def _problem(n, d, scale=1.0):
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, d)) * np.linspace(1.0, 2.0, d)
    return X, scale * np.sum((X / np.linspace(1.0, 2.0, d)) ** 2, axis=1)


@pytest.mark.parametrize("n", [8, 31, 32, 33, 63, 65, 96, 127, 128, 129, 159, 161, 256, 289, 385, 515])
@pytest.mark.parametrize("kernel", [0, 1])
def test_fp64_fit_tile_edges(gpu, oracle, n, kernel):
    d = 6
    X, m2 = _problem(n, d)
    o = _orc_dist(oracle, 0, kernel, d, X=X, over_smooth=0.6)
    sd = _gpu_dist(gpu, 0, kernel, d, X=X, over_smooth=0.6)
    assert o.prepare_interp(m2) == 0
    sd.prepare_interp(m2)
    w, wo = sd.peek_weights(), o.weights()
    assert np.max(np.abs(w - wo)) <= FP64_TOL * np.max(wo)
    assert sd.get_rnorm() == pytest.approx(o.rnorm, rel=1e-10)


@pytest.mark.parametrize("n", [1100, 2500])
def test_fp64_fit_against_mixed(gpu, n):
    """A wide range of f (rows of the matrix scaled by up to e^60) and several
    tiles per SM."""
    d = 9
    X, m2 = _problem(n, d, scale=1.5)
    sd = _gpu_dist(gpu, 1, 1, d, X=X)
    sd.prepare_interp(m2)
    w, st = sd.peek_weights(), sd.get_interp_stats()
    assert st["fp64"] == st["solves"] > 0 and sd.get_interp_fallbacks() == {"lu": 0, "qr": 0}
    sd.set_precision(gpu.Precision.MIXED)
    sd.prepare_interp(m2)
    assert sd.get_interp_stats()["fp64"] == 0
    assert np.max(np.abs(w - sd.peek_weights())) <= FP64_TOL * np.max(w)
