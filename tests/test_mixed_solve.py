"""The mixed weight fit at the edges of its blocks: the 64-column panels of the
FP32 factor, the 128-row blocks of its triangular solves and the set sizes around
them, against the FP64 form on the same matrix (weights <= 1e-10 of the largest, the
FP64 form's bound), without a fallback to FP64."""
import numpy as np
import pytest

from test_gpu_parity import FP64_TOL, _gpu_dist
from test_posv64 import _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 63, 64, 65, 126, 127, 128, 129, 191, 193, 255, 257, 383, 385, 520])
@pytest.mark.parametrize("kernel", [0, 1])
def test_mixed_fit_block_edges(gpu, n, kernel):
    d = 6
    X, m2 = _problem(n, d)
    sd = _gpu_dist(gpu, 0, kernel, d, X=X, over_smooth=0.6)
    sd.prepare_interp(m2)
    w = sd.peek_weights()
    sd.set_precision(gpu.Precision.MIXED)
    sd.prepare_interp(m2)
    st = sd.get_interp_stats()
    assert st["fp64"] == 0 and st["solves"] > 0
    assert np.max(np.abs(w - sd.peek_weights())) <= FP64_TOL * np.max(w)
