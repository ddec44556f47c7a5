"""Host evals around the sizes where the points change their way to the device
(read in place, moved by the checking kernel, copied) against the same points on
the device: the same kernels, so the same bits; non-finite points are refused on
each way and leave the handle usable."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from test_gpu_parity import _gpu_dist

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
@pytest.mark.parametrize("kind,d", [(0, 4), (1, 27), (1, 3)])
def test_host_eval_is_the_device_eval(gpu, kind, d, precision):
    rng = np.random.default_rng(d)
    sd = _gpu_dist(gpu, kind, 1, d, X=rng.standard_normal((400, d)))
    sd.set_precision(gpu.Precision[precision])
    sd.prepare()
    edge = 8192 // d
    for m in sorted({1, 2, 16, 17, min(edge, 2048), min(edge, 2048) + 1, 2049}):
        P = rng.standard_normal((m, d))
        dP = torch.from_numpy(P).cuda()
        out = torch.empty(m, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        sd.eval_m2lnp_device(dP.data_ptr(), m, out.data_ptr())
        torch.cuda.synchronize()
        assert np.array_equal(sd.eval_m2lnp(P), out.cpu().numpy()), m
        P[-1, -1] = np.inf if m % 2 else np.nan
        with pytest.raises(gpu.NcgError):
            sd.eval_m2lnp(P)
