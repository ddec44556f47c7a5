"""The FP64 branch schedule runs each problem as its own eval does, bit for bit, also where
that eval takes the sliced products (VKDE, d >= 5, from 640 points and 384 kernels), and after
the handles were prepared again."""
import numpy as np
import pytest

from test_batch import _problem

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 8, 600, 700), (1, 0, 16, 1009, 1000), (1, 1, 27, 1700, 641), (1, 1, 5, 384, 640), (1, 1, 5, 383, 640),
          (1, 0, 6, 500, 639), (1, 1, 4, 500, 900), (0, 1, 9, 700, 800), (1, 1, 12, 900, 9000), (1, 0, 7, 800, 3)]


def test_branches_equal_own_evals(gpu):
    ng = gpu
    F = ng.Precision.FP64
    probs = [_problem(ng, *s, seed=80 + i) for i, s in enumerate(SHAPES)]
    pts = [P for _, _, P in probs]
    b = ng.Batch()
    for sd, _, P in probs:
        b.add(sd, len(P))
    b.set_params(F, tc=2)
    for scale in (1.0, 1.4):
        if scale != 1.0:
            for sd, X, _ in probs:
                sd.set_sample(X * scale)
                sd.prepare()
        for _ in range(2):
            got = b.eval_m2lnp(pts, F)
            assert all(np.array_equal(g, sd.eval_m2lnp(P)) for g, (sd, _, P) in zip(got, probs))
