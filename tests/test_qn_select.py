"""The Qn selection at the sizes where it changes its way: sets smaller than
the ranked remainder (no count at all), the last set of a warp and the first of a
whole CTA (1024, 1025 rows), power-of-two edges of the sort, and ranges far wider
than the scale (the octave steps) or far narrower.  ROBUST_DIAG is sigma^2 per
coordinate, and sigma is an order statistic of exact differences: the oracle's
bits."""
import numpy as np
import pytest

from test_robust import _pair

pytestmark = pytest.mark.gpu


def _values(rng, kind, n, d):
    if kind == "gauss":
        return rng.standard_normal((n, d))
    if kind == "cauchy":                       # a range of 1e12 scales and more
        return np.ldexp(rng.standard_cauchy((n, d)), rng.integers(0, 40, (n, d)) * (rng.random((n, d)) < 0.02))
    if kind == "ties":
        return np.floor(3.0 * rng.standard_normal((n, d))) + 0.25
    return 1.0 + rng.integers(0, 50, (n, d)) * 2.0 ** -50   # a few ulps apart


@pytest.mark.parametrize("kind", ["gauss", "cauchy", "ties", "ulps"])
@pytest.mark.parametrize("n", [4, 5, 8, 9, 32, 33, 65, 512, 1023, 1024, 1025, 2048, 2049, 5000])
def test_diagonal_scale_is_the_oracles(gpu, oracle, n, kind):
    d = 2
    rng = np.random.default_rng(n)
    X = _values(rng, kind, n, d)
    if n < 10 and kind in ("ties", "ulps"):
        X += np.arange(n)[:, None] * (1.0 if kind == "ties" else 2.0 ** -46)   # a positive scale
    sd, o = _pair(gpu, oracle, 0, 0, d, X, 2)
    assert np.array_equal(sd.peek_full_cov(), o.cov())


@pytest.mark.parametrize("frac", [0.01, 0.06, 0.4])
@pytest.mark.parametrize("kind", ["gauss", "cauchy"])
def test_neighbourhood_factors_are_the_oracles(gpu, oracle, kind, frac):
    d, n = 2, 700
    rng = np.random.default_rng(int(100 * frac))
    X = _values(rng, kind, n, d)
    sd, o = _pair(gpu, oracle, 1, 0, d, X, 2, local_frac=frac)
    for i in range(0, n, 37):
        a, b = np.triu(sd.peek_cov_decomp(i)), np.triu(o.Ui(i))
        # sqrt(sigma^2) on the diagonal: one rounding of each side
        assert np.max(np.abs(a - b)) <= 4e-16 * np.max(np.abs(b))
