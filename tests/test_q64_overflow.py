"""Kernels so narrow that the square of their whitening leaves FP64 (a cluster of width 1e-158
in a sample of width 1): their sliced-product operand is not finite, and the eval has to keep
the plain form, which only needs the whitening itself."""
import numpy as np
import pytest

from conftest import rel_err
from test_eval_q64 import _plain
from test_gpu_parity import FP64_TOL, _gpu_dist, _orc_dist

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [0, 1])
def test_operand_past_fp64(gpu, oracle, kernel):
    rng = np.random.default_rng(12)
    d, n = 5, 500
    X = rng.standard_normal((n, d))
    X[: n // 2] *= 1e-158
    X[n // 2 :, 0] += 20.0              # neighbourhoods of their own
    P = np.concatenate([X[: n // 2: 2] * 1.1, X[n // 2 :] + 0.3, rng.standard_normal((400, d))])
    o = _orc_dist(oracle, 1, kernel, d, X=X)
    sd = _gpu_dist(gpu, 1, kernel, d, X=X)
    assert o.prepare() == 0
    sd.prepare()
    want, got = o.eval_m2lnp(P), sd.eval_m2lnp(P)
    assert np.all(np.isfinite(want))
    assert rel_err(got, want) < FP64_TOL
    assert np.array_equal(got, _plain(sd, P))
