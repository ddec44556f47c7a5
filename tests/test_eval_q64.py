"""The FP64 eval whose chi^2 comes from sliced tensor-core products: against the
oracle (1e-10 relative, the FP64 form's bound) and against the plain FP64
kernels (the no-allocation entry keeps them): both forms round chi^2 and the
sums at about 1e-16 of -2 ln p, so 100 units of that, 1e-14, separates rounding
from a lost digit (2^-40 or more)."""
import ctypes as C

import numpy as np
import pytest

from conftest import rel_err
from test_gpu_parity import FP64_TOL, _gpu_dist, _orc_dist

pytestmark = pytest.mark.gpu

PLAIN_TOL = 1e-14


def _plain(sd, P):
    import torch

    from numcosmo_gb300 import _lib

    x = torch.tensor(P, dtype=torch.float64, device="cuda")
    out = torch.empty(len(P), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    _lib.check(_lib.load().ncg_sd_eval_m2lnp_device_noalloc(sd._h, C.c_void_p(x.data_ptr()), len(P),
                                                            C.c_void_p(out.data_ptr())), "noalloc")
    sd.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("kernel", [0, 1])
@pytest.mark.parametrize("d,n,m", [(5, 384, 640), (6, 431, 641), (8, 576, 767), (15, 960, 640), (16, 1009, 1000),
                                   (17, 1021, 769), (24, 1441, 640), (32, 1700, 700)])
def test_q64_shapes(gpu, oracle, kernel, d, n, m):
    rng = np.random.default_rng(d + n)
    S = rng.standard_normal((d, d)) / np.sqrt(d) + np.eye(d)
    X = rng.standard_normal((n, d)) @ S + 50.0
    P = rng.standard_normal((m, d)) @ S + 50.0
    P[:12] = X[:12]                                             # at kernel centres
    P[12:20] = 50.0 + (P[12:20] - 50.0) * 10.0 ** np.arange(1, 9)[:, None]   # far outside
    o = _orc_dist(oracle, 1, kernel, d, X=X, local_frac=0.1)
    sd = _gpu_dist(gpu, 1, kernel, d, X=X, local_frac=0.1)
    assert o.prepare() == 0
    sd.prepare()
    got = sd.eval_m2lnp(P)
    assert rel_err(got, o.eval_m2lnp(P)) < FP64_TOL
    assert rel_err(got, _plain(sd, P)) < PLAIN_TOL
    assert np.array_equal(got, sd.eval_m2lnp(P))
    assert rel_err(sd.eval(P), o.eval(P), floor=1e-300) < FP64_TOL


def test_q64_point_chunks(gpu):
    """More points than one launch takes, the last one short."""
    rng = np.random.default_rng(3)
    X, P = rng.standard_normal((600, 7)), rng.standard_normal((8192 + 8192 + 130, 7))
    sd = _gpu_dist(gpu, 1, 1, 7, X=X)
    sd.prepare()
    got = sd.eval_m2lnp(P)
    assert rel_err(got, _plain(sd, P)) < PLAIN_TOL
    assert np.array_equal(got[:8192], sd.eval_m2lnp(P[:8192]))


@pytest.mark.parametrize("scale", [1e-3, 1e-7])
def test_q64_narrow_kernels(gpu, oracle, scale):
    """A tight cluster far from the rest: kernels narrow against the global
    covariance, within the fixed point's range and beyond it (plain form)."""
    rng = np.random.default_rng(4)
    d, n = 5, 600
    X = rng.standard_normal((n, d))
    X[: n // 2] = 3.0 + X[: n // 2] * scale
    P = np.concatenate([X[::2] + 0.3 * scale * rng.standard_normal((n // 2, d)), rng.standard_normal((400, d))])
    o = _orc_dist(oracle, 1, 0, d, X=X)
    sd = _gpu_dist(gpu, 1, 0, d, X=X)
    assert o.prepare() == 0
    sd.prepare()
    assert rel_err(sd.eval_m2lnp(P), o.eval_m2lnp(P), floor=1.0) < FP64_TOL


def test_q64_state_changes(gpu, oracle):
    """The operand follows the bandwidth and the sample; the weights are not in it."""
    rng = np.random.default_rng(6)
    d, n = 6, 500
    X, X2, P = rng.standard_normal((n, d)), rng.standard_normal((n + 90, d)) * 2.0, rng.standard_normal((700, d))
    sd = _gpu_dist(gpu, 1, 1, d, X=X)
    for X_, os_, interp in ((X, 1.0, False), (X, 1.0, True), (X, 0.7, True), (X2, 0.7, False)):
        o = _orc_dist(oracle, 1, 1, d, X=X_, over_smooth=os_)
        sd.set_over_smooth(os_)
        sd.set_sample(X_)
        m2 = np.sum(X_ ** 2, axis=1)
        if interp:
            assert o.prepare_interp(m2) == 0
            sd.prepare_interp(m2)
        else:
            assert o.prepare() == 0
            sd.prepare()
        assert rel_err(sd.eval_m2lnp(P), o.eval_m2lnp(P)) < FP64_TOL


def test_q64_bad_points(gpu):
    """The device entry does not check its points: a NaN or infinite coordinate
    gives what the plain form gives, and leaves the others alone."""
    import torch

    rng = np.random.default_rng(8)
    X, P = rng.standard_normal((500, 5)), rng.standard_normal((640, 5))
    sd = _gpu_dist(gpu, 1, 0, 5, X=X)
    sd.prepare()
    want = sd.eval_m2lnp(P)
    P[3, 1], P[130, 0], P[639, 4] = np.nan, np.inf, -np.inf
    x = torch.tensor(P, dtype=torch.float64, device="cuda")
    out = torch.empty(640, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    sd.eval_m2lnp_device(x.data_ptr(), 640, out.data_ptr())
    sd.synchronize()
    got = out.cpu().numpy()
    keep = np.ones(640, dtype=bool)
    keep[[3, 130, 639]] = False
    assert np.array_equal(got[keep], want[keep])
    assert np.array_equal(got[~keep], _plain(sd, P)[~keep])
