"""A kernel's dynamic shared-memory limit belongs to the kernel on the device, for all threads of the process.  A launch
path that sets it to its own call's size can lower it between another thread's call and its larger launch, which then does
not run, and the kernels after it read a scratch that was not written.  So no launch path sets it: the solve's limits are
set once per device to their largest value, the front end's are only raised.  Read from the sources, then (GPU) two threads
with a handle each, one with aerosol, whose kernels need more, and one without."""
from __future__ import annotations

import re
import threading
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "woof_nam_b200" / "csrc"
SETTERS = {"set_smem_limits", "raise_smem"}


def _functions_setting_limits():
    for f in sorted(CSRC.glob("*.cu*")):
        name = None
        for line in f.read_text().splitlines():
            m = re.match(r"(?:[\w:<>*&]+\s+)+(\w+)\(", line)               # a definition starts in the first column
            if m:
                name = m.group(1)
            if re.search(r"\bcudaFuncSetAttribute\b", line.split("//")[0]):
                yield f.name, name


def test_no_launch_path_sets_a_limit():
    found = list(_functions_setting_limits())
    assert {n for _, n in found} == SETTERS, found


@pytest.mark.gpu
@pytest.mark.parametrize("form", [dict(), dict(lw_chunk=-1, sw_sweep_chunk=-1)], ids=["chunked", "single"])
def test_two_threads(form):
    import torch
    from woof_nam_b200.columns import make_columns
    from woof_nam_b200.solver import RadSolver
    cols = make_columns(8, 31)
    aer = torch.full((3, 14, 61, 8), 0.1, device="cuda")
    errors = []

    def work(with_aer):
        try:
            s = RadSolver(parts="sw", **form)
            d = s.to_device(cols)
            if with_aer:
                d["faersw"] = aer
            st = torch.cuda.Stream()
            st.wait_stream(torch.cuda.current_stream())
            ref = None
            for _ in range(300):
                with torch.cuda.stream(st):
                    out = s.solve(d, cols.solcon, stream=st)
                st.synchronize()
                got = {k: v.cpu().numpy() for k, v in out.items()}
                ref = ref or got
                assert all(np.array_equal(got[k], ref[k]) for k in ref)
        except BaseException as e:  # noqa: BLE001 -- reported by the main thread
            errors.append(e)

    ts = [threading.Thread(target=work, args=(a,)) for a in (False, True)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors
