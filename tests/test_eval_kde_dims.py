"""KDE's FP64 eval in every even number of coordinates it is built for, odd ones
within them: a few points (one kernel per thread) and the tiles, against the
oracle at 1e-10 relative, the FP64 form's bound."""
import numpy as np
import pytest

from conftest import rel_err
from test_gpu_parity import FP64_TOL, _gpu_dist, _orc_dist

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [0, 1])
@pytest.mark.parametrize("d", [2, 3, 5, 6, 7, 9, 10, 13, 14, 17, 18, 21, 22, 25, 26, 29, 30, 31])
def test_kde_dims(gpu, oracle, d, kernel):
    rng = np.random.default_rng(d)
    X = rng.standard_normal((300, d)) * np.linspace(0.5, 2.0, d)
    o = _orc_dist(oracle, 0, kernel, d, X=X)
    sd = _gpu_dist(gpu, 0, kernel, d, X=X)
    assert o.prepare() == 0
    sd.prepare()
    P = rng.standard_normal((70, d)) * np.linspace(0.5, 2.0, d)
    want = o.eval_m2lnp(P)
    for m in (1, 9, 70):
        assert rel_err(sd.eval_m2lnp(P[:m]), want[:m]) < FP64_TOL, m
