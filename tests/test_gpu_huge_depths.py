"""Cloud and aerosol optical depths given directly far beyond the last entry of the exponential tables, up to 3e38, the
largest a float holds: such a layer is opaque.  The mixed kernels take a depth's table position from a reciprocal of the
depth itself, and its albedo and asymmetry from reciprocals of depths, which must not be flushed to zero (a reciprocal of
more than 2^126 = 8.5e37 is below the smallest normal float), and a finite depth times 1 / mu0 or the diffusivity may pass
the largest float.  Against the float64 oracle, where none of this happens, within the path's tolerances
(0.05 W/m^2, 0.01 K/day)."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_within
from oracle import oracle
from woof_nam_b200.columns import Columns, make_columns

pytestmark = pytest.mark.gpu

DEPTHS = (1.0e30, 8.0e37, 9.0e37, 1.5e38, 3.0e38)
N = 24 * len(DEPTHS)


def _columns(depth: bool, seed: int) -> Columns:
    """Direct cloud optics, every fourth column with its sun at the two-stream resonance (whose g-points take the
    float64 fix-up); depth: each cloudy layer holds one of DEPTHS, by column."""
    cols = make_columns(N, seed, stress=True)
    d = {k: v.copy() for k, v in cols.arrays().items()}
    cf, tau, ssa = d["clouds"][0], d["clouds"][1], d["clouds"][2]
    cf[np.diff(d["plvl"], axis=0) < 2.0] = 0.0                          # no column for the float64 LW kernel
    rng = np.random.default_rng(seed)
    ssa[:] = rng.choice(np.array([0.0, 0.3, 0.9, 0.999], np.float32), ssa.shape)
    if depth:
        tau[:] = np.where(cf > 0, np.array(DEPTHS, np.float32)[np.arange(N) % len(DEPTHS)][None], tau)
    d["coszen"] = rng.uniform(0.05, 1.0, N).astype(np.float32)
    d["coszen"][::4] = 0.5
    return Columns(**d, solcon=cols.solcon, diagnostic_clouds=True)


def _run(cols, faersw=None, faerlw=None, **kw):
    import torch
    from woof_nam_b200.solver import RadSolver
    s = RadSolver(diagnostic=True, **kw)
    dev = s.to_device(cols)
    if faersw is not None:
        dev["faersw"], dev["faerlw"] = torch.from_numpy(faersw).cuda(), torch.from_numpy(faerlw).cuda()
    out = s.solve(dev, cols.solcon)
    torch.cuda.synchronize()
    assert s.device_error() == 0
    return {k: v.cpu().numpy() for k, v in out.items()}


FORMS = [dict(), dict(lw_chunk=-1, sw_sweep_chunk=-1)]


@pytest.mark.parametrize("form", FORMS, ids=["chunked", "single"])
@pytest.mark.parametrize("mode,iovrlw", [(2, 1), (2, 0), (3, 1)])
def test_cloud(mode, iovrlw, form):
    cols = _columns(True, 61 + mode)
    ref = oracle.solve(cols, precision="double", iswmode=mode, iovrlw=iovrlw)
    assert all(np.isfinite(v).all() for v in ref.values())
    assert_within(_run(cols, iswmode=mode, iovrlw=iovrlw, **form), ref, what=f"mode {mode}, overlap {iovrlw}")


@pytest.mark.parametrize("form", FORMS, ids=["chunked", "single"])
def test_aerosol(form):
    cols = _columns(False, 71)
    rng = np.random.default_rng(72)
    fsw, flw = np.zeros((3, 14, 61, N), np.float32), np.zeros((3, 16, 61, N), np.float32)
    for f in (fsw, flw):
        f[0] = 0.01
        f[0, :, 40:] = np.array(DEPTHS, np.float32)[np.arange(N) % len(DEPTHS)]
        f[0, :, 40:][:, cols.clouds[0, 40:] > 0] = 0.01                 # the layer's sum stays finite
        f[1] = rng.choice(np.array([0.0, 0.5, 0.95], np.float32), f[1].shape)
        f[2] = 0.6
    ref = oracle.solve(cols, precision="double", faersw=fsw, faerlw=flw)
    assert all(np.isfinite(v).all() for v in ref.values())
    assert_within(_run(cols, fsw, flw, **form), ref, what="aerosol")
