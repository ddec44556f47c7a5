"""The FP64 eval recorded in a CUDA graph: its launches depend on one another by
programmatic edges there too, and a replay gives the bits of the plain call, for the
few-point kernel, the tiles and the sliced-product form (warm before the capture)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from test_gpu_parity import _gpu_dist

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,d,n,m", [(0, 4, 500, 3), (0, 6, 500, 300), (1, 6, 500, 300), (1, 6, 500, 1500)])
def test_captured_eval(gpu, kind, d, n, m):
    rng = np.random.default_rng(n + m)
    sd = _gpu_dist(gpu, kind, 1, d, X=rng.standard_normal((n, d)))
    s = torch.cuda.Stream()
    sd.set_stream(s.cuda_stream)
    sd.prepare()
    P = torch.from_numpy(rng.standard_normal((m, d))).cuda()
    want, out = (torch.empty(m, dtype=torch.float64, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    sd.eval_m2lnp_device(P.data_ptr(), m, want.data_ptr())
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        sd.eval_m2lnp_device(P.data_ptr(), m, out.data_ptr())
    for _ in range(3):
        out.zero_()
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
