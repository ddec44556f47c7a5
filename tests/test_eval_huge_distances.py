"""Points so far out that chi^2 is above 1e300 but still a double: -2 ln p is that chi^2 (Gauss),
not infinity, in every FP64 form."""
import numpy as np
import pytest

from conftest import rel_err
from test_gpu_parity import FP64_TOL, _gpu_dist, _orc_dist

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [5, 60, 700])
@pytest.mark.parametrize("kind,kernel", [(0, 0), (1, 0), (1, 1)])
def test_huge_distances(gpu, oracle, kind, kernel, m):
    rng = np.random.default_rng(m)
    d = 5
    X, P = rng.standard_normal((500, d)), rng.standard_normal((m, d))
    P[1::2] *= 1e152
    o = _orc_dist(oracle, kind, kernel, d, X=X)
    sd = _gpu_dist(gpu, kind, kernel, d, X=X)
    assert o.prepare() == 0
    sd.prepare()
    want = o.eval_m2lnp(P)
    assert np.all(np.isfinite(want)) and (kernel == 1 or want.max() > 1e302)
    assert rel_err(sd.eval_m2lnp(P), want) < FP64_TOL
    b = gpu.Batch()
    b.add(sd, m)
    assert rel_err(b.eval_m2lnp([P])[0], want) < FP64_TOL
