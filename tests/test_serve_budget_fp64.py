"""An FP64 chain whose operand of the sliced products does not fit the memory budget is served
in the plain form, as it was before that operand existed, instead of being refused."""
import numpy as np
import pytest

from test_serve import _add_all, _final

pytestmark = pytest.mark.gpu


def test_chain_that_fits_without_the_operand(gpu):
    ng = gpu
    chains = [(1, 1, 16, 2048)]
    fin = []
    budget = 40 << 30
    for _ in range(2):
        srv = ng.Server(slots=1, precision=ng.Precision.FP64, hbm_budget=budget)
        (c,) = _add_all(srv, chains)
        res = [srv.result(srv.submit(c)) for _ in range(2)]
        st = srv.stats()
        assert all(r["status"] == 0 for r in res) and st["failed"] == 0
        assert st["peak_reserved_bytes"] <= budget
        fin.append(_final(srv, [c])[0])
        budget = st["peak_reserved_bytes"] - 1          # the next one: a byte short of the operand's
        srv.close()
    (Xa, ma), (Xb, mb) = fin
    assert np.array_equal(Xa, Xb) and np.max(np.abs(ma - mb)) < 1e-10 * np.max(np.abs(ma))
