"""The SW day list of small launches (k_daylist_small, one CTA up to 2,048 columns) against the general kernels: a request
solved alone, and in a batch whose column total takes the general path, gives the same bits, at sizes around a warp's,
the CTA's and the rule's edges, all day, all night and mixed, with windows that cut the day list."""
from __future__ import annotations

import numpy as np
import pytest

from woof_nam_b200.columns import Columns, make_columns

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,sun,window", [(1, "day", 0), (2, "mixed", 0), (63, "mixed", 8), (65, "mixed", 13),
                                          (2047, "mixed", 100), (2048, "day", 0), (2048, "mixed", 77), (100, "night", 0)])
def test_small_day_list_equals_the_general_one(n, sun, window):
    import torch
    from woof_nam_b200.solver import RadSolver
    cols = make_columns(n, 40 + n)
    d = {k: np.ascontiguousarray(v) for k, v in cols.arrays().items()}
    if sun == "day":
        d["coszen"] = np.abs(d["coszen"]) + np.float32(0.01)
    elif sun == "night":
        d["coszen"] = -np.abs(d["coszen"])
    cols = Columns(**d, solcon=cols.solcon)
    other = make_columns(2100, 7)
    s = RadSolver(parts="sw", window_cols=window)
    dev, dev2 = s.to_device(cols), s.to_device(other)
    alone = s.solve(dev, cols.solcon)
    batch = s.solve_batch([dev2, dev], [other.solcon, cols.solcon])[1]
    torch.cuda.synchronize()
    assert s.device_error() == 0
    for k in alone:
        assert np.array_equal(alone[k].cpu().numpy(), batch[k].cpu().numpy()), k
