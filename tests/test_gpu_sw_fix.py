"""The float64 queue of the chunked SW (sw4_rt_kernel's queue, sw4_fix_kernel): columns whose sun sits at a two-stream
resonance k mu0 = 1 that every strongly absorbing layer shares (PIFM k = 2, discrete ordinates k = sqrt(3)), so that
thousands of g-points of a column are queued, beside ordinary ones, over several tiles with a ragged last one, at layer
counts at and off the item size -- against the float64 oracle within the path's tolerances (0.05 W/m^2, 0.01 K/day) and
tile-independent to the bit."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_within
from oracle import oracle
from woof_nam_b200.columns import Columns, make_columns

pytestmark = pytest.mark.gpu


def _resonant(n, nlay, mode, seed):
    cols = make_columns(n, seed)
    d = {k: np.ascontiguousarray(v[..., -nlay:, :] if v.ndim > 1 and v.shape[-2] == 61 else v) for k, v in cols.arrays().items()}
    for k in ("plvl", "tlvl"):
        d[k] = np.ascontiguousarray(d[k][-(nlay + 1):])
    mu = 0.5 if mode == 2 else 1.0 / np.sqrt(3.0)
    cz = d["coszen"].copy()
    cz[::3] = mu * (1.0 + np.linspace(-4e-3, 4e-3, cz[::3].size))      # inside |1 - (k mu0)^2| < 1e-2
    cz[1::3] = np.abs(cz[1::3])
    d["coszen"] = cz.astype(np.float32)
    return Columns(**d, solcon=cols.solcon)


@pytest.mark.parametrize("nlay,mode,tile", [(61, 2, 100), (61, 3, 90), (2, 2, 37), (16, 2, 64), (33, 3, 128)])
def test_resonant_columns(nlay, mode, tile):
    import torch
    from woof_nam_b200.solver import RadSolver
    cols = _resonant(301, nlay, mode, 900 + nlay)
    outs = []
    for t in (tile, 0):
        s = RadSolver(parts="sw", nlay=nlay, iswmode=mode, sw_sweep_chunk=t)
        out = s.solve(s.to_device(cols), cols.solcon)
        torch.cuda.synchronize()
        assert s.device_error() == 0
        outs.append({k: v.cpu().numpy() for k, v in out.items()})
    ref = oracle.solve(cols, precision="double", iswmode=mode)
    assert_within(outs[0], {k: ref[k] for k in outs[0]}, what=f"resonant columns, {nlay} layers, mode {mode}")
    for k in outs[0]:
        assert np.array_equal(outs[0][k], outs[1][k]), k


def test_recompute_lists_and_their_overflow():
    """A tile of 4,096 columns or more hands its float64 recomputes to sw4_exact_kernel through per-band lists (here
    with more resonant g-points in some bands than a list holds, so that some stay with sw4_fix_kernel, and fewer in
    others); smaller tiles run them all in sw4_fix_kernel.  Same bits either way, and within tolerance of the oracle."""
    import torch
    from woof_nam_b200.solver import RadSolver
    cols = _resonant(4600, 61, 2, 77)
    outs = []
    for t in (0, 4096, 1000):
        s = RadSolver(parts="sw", sw_sweep_chunk=t)
        out = s.solve(s.to_device(cols), cols.solcon)
        torch.cuda.synchronize()
        assert s.device_error() == 0
        counts, cap = s.sw_recomputes()
        if t == 0:                                   # one tile of all the columns
            assert cap == 4600 and max(counts) > cap and any(0 < c <= cap for c in counts), counts
        else:
            assert cap == (t if t >= 4096 else 0)
        outs.append({k: v.cpu().numpy() for k, v in out.items()})
    for o in outs[1:]:
        for k in o:
            assert np.array_equal(o[k], outs[0][k]), k
    head = cols.slice(0, 256)
    ref = oracle.solve(head, precision="double")
    assert_within({k: outs[0][k][..., :256] for k in outs[0]}, {k: ref[k] for k in outs[0]}, what="recompute lists")
