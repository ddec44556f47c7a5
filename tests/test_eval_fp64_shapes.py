"""FP64 eval over the shapes where its launch changes form: point counts around
the few-point kernel (16) and the 32-point tiles, kernel counts around its
128-kernel and 32-kernel slices and the staged chunks, every padded dimension
class, points whose kernel sums span the exponential's whole range.

Tolerance: 1e-10 relative, the FP64 form's bound against the oracle."""
import numpy as np
import pytest

from conftest import rel_err
from test_gpu_parity import FP64_TOL, _gpu_dist, _orc_dist

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,kernel", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("d,n", [(1, 41), (4, 127), (9, 129), (16, 1025), (29, 1300)])
def test_eval_fp64_shapes(gpu, oracle, kind, kernel, d, n):
    rng = np.random.default_rng(100 * d + 2 * kind + kernel)
    X = rng.standard_normal((n, d)) * np.linspace(0.3, 3.0, d)
    o = _orc_dist(oracle, kind, kernel, d, X=X, local_frac=0.1)
    sd = _gpu_dist(gpu, kind, kernel, d, X=X, **({"local_frac": 0.1} if kind else {}))
    assert o.prepare() == 0
    sd.prepare()
    P = rng.standard_normal((161, d)) * np.linspace(0.3, 3.0, d)
    P[:8] *= 10.0 ** np.arange(8)[:, None]        # from inside the sample to far outside
    P[8:24] = X[:16]                              # at kernel centres
    want = o.eval_m2lnp(P)
    for m in (1, 2, 16, 17, 31, 32, 33, 161):
        assert rel_err(sd.eval_m2lnp(P[:m]), want[:m]) < FP64_TOL, m
    assert rel_err(sd.eval(P[8:]), o.eval(P[8:]), floor=1e-300) < FP64_TOL


def test_eval_fp64_zero_weights(gpu, oracle):
    """Kernels of zero weight (ln w = -inf) at the start of every slice."""
    rng = np.random.default_rng(9)
    d, n = 3, 260
    X = rng.standard_normal((n, d))
    m2 = np.sum(X ** 2, axis=1)
    o = _orc_dist(oracle, 1, 0, d, X=X)
    sd = _gpu_dist(gpu, 1, 0, d, X=X, shrink=0.0)
    sd.prepare_interp(m2)
    assert (sd.peek_weights() == 0.0).any()
    o = _orc_dist(oracle, 1, 0, d, X=X, shrink=0.0)
    assert o.prepare_interp(m2) == 0
    P = rng.standard_normal((40, d))
    for m in (3, 40):
        assert rel_err(sd.eval_m2lnp(P[:m]), o.eval_m2lnp(P[:m])) < FP64_TOL
