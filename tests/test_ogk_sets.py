"""The OGK eigenvectors of many sets, several to a CTA: set counts that leave the last
CTA partly filled, and dimensions on either side of the group sizes (8, 16) and
odd.  Factors against the oracle's, normwise (two Jacobi orderings: 1e-10, the
FP64 form's bound)."""
import numpy as np
import pytest

from conftest import rel_err
from test_robust import FP64_TOL, _data, _pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,n,frac", [(2, 1221, 0.02), (7, 1219, 0.05), (8, 307, 0.1), (9, 613, 0.08), (17, 305, 0.3)])
def test_factors_of_many_sets(gpu, oracle, d, n, frac):
    X, P = _data(d, n, 17 * d)
    sd, o = _pair(gpu, oracle, 1, 0, d, X, 3, local_frac=frac)
    for i in list(range(0, n, 61)) + [n - 2, n - 1]:
        a, b = np.triu(sd.peek_cov_decomp(i)), np.triu(o.Ui(i))
        assert rel_err(a, b, floor=np.max(np.abs(b))) < FP64_TOL
    assert rel_err(sd.eval_m2lnp(P), o.eval_m2lnp(P), floor=1.0) < FP64_TOL
