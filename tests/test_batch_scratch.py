"""A batch's captured graph keeps to memory of its own: an own eval of one of its handles, which
moves the handle's scratch, neither changes the batch's results nor leaves the graph
writing where that scratch was; and a handle may stand in one batch twice."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from test_batch import _problem

pytestmark = pytest.mark.gpu

# (kind, kernel, d, n, m): VKDE sizes whose own FP64 eval takes the sliced products, and others
SHAPES = [(1, 0, 5, 384, 640), (1, 1, 16, 1300, 900), (0, 1, 7, 500, 700), (1, 1, 8, 600, 90)]


@pytest.mark.parametrize("precision,tc", [(0, 2), (1, 2), (1, 1)])
def test_own_evals_between_batches(gpu, precision, tc):
    ng = gpu
    prec = ng.Precision(precision)
    probs = [_problem(ng, *s, seed=40 + i) for i, s in enumerate(SHAPES)]
    b = ng.Batch()
    for sd, _, P in probs:
        b.add(sd, len(P))
    b.set_params(prec, tc=tc)
    pts = [P for _, _, P in probs]
    first = b.eval_m2lnp(pts, prec)
    captures = b.get_stats(prec)["captures"]
    for m in (700, 2000):
        for sd, X, P in probs:
            for p in (ng.Precision.FP64, ng.Precision.MIXED):
                sd.set_precision(p)
                sd.eval_m2lnp(np.resize(P, (m, P.shape[1])))
        # blocks of many sizes where freed scratch would be
        guard = [torch.full((k * 1024,), 7.0, dtype=torch.float64, device="cuda") for k in (8, 16, 64, 256, 1024, 4096) * 4]
        torch.cuda.synchronize()
        again = b.eval_m2lnp(pts, prec)
        assert all(np.array_equal(x, y) for x, y in zip(first, again))
        assert all(bool((g == 7.0).all()) for g in guard)
        del guard
    assert b.get_stats(prec)["captures"] == captures


@pytest.mark.parametrize("precision,tc", [(0, 2), (1, 2), (1, 1)])
def test_one_handle_twice(gpu, precision, tc):
    ng = gpu
    prec = ng.Precision(precision)
    sd, _, P = _problem(ng, 1, 1, 8, 600, 600, seed=3)
    b = ng.Batch()
    for k in (600, 333):
        b.add(sd, k)
    b.set_params(prec, tc=tc)
    for _ in range(3):
        one, two = b.eval_m2lnp([P, P[:333]], prec)
        assert np.max(np.abs(one[:333] - two)) <= 1e-6 * np.max(np.abs(two))
        if precision == 0:
            assert np.max(np.abs(one[:333] - two)) <= 1e-13 * np.max(np.abs(two))


def test_both_plans_follow_a_new_prepare(gpu):
    """The FP64 and the mixed plan are each rebuilt after their handles were prepared again."""
    ng = gpu
    F, M = ng.Precision.FP64, ng.Precision.MIXED
    probs = [_problem(ng, *s, seed=60 + i) for i, s in enumerate(SHAPES)]
    pts = [P for _, _, P in probs]
    b = ng.Batch()
    for sd, _, P in probs:
        b.add(sd, len(P))
    b.eval_m2lnp(pts, F)
    b.eval_m2lnp(pts, M)
    for sd, X, _ in probs:
        sd.set_sample(X[::-1] * 1.3 + 0.2)
        sd.prepare()
    got = b.eval_m2lnp(pts, F), b.eval_m2lnp(pts, M)
    fresh = ng.Batch()
    for sd, _, P in probs:
        fresh.add(sd, len(P))
    for g, p in zip(got, (F, M)):
        assert all(np.array_equal(x, y) for x, y in zip(g, fresh.eval_m2lnp(pts, p)))
