"""gradient_schedule 'auto' sizes the launch to the free memory: the largest balanced one that fits.
(On the host: plans are described and measured, no workspace is made.)"""
import ctypes as C
import types

import numpy as np
import pytest

from pysit_gb300 import _native, engine
from test_workspace_limits import _desc


@pytest.fixture(scope="module")
def lib():
    from pysit_gb300 import build
    build.build()
    return _native.load()


@pytest.mark.parametrize("share", [0.02, 0.1, 0.3, 0.7])
@pytest.mark.parametrize("n,pml,steps,S", [((141, 1, 81), ((10, 10), (0, 0), (10, 10)), 20000, 283),
                                           ((401, 1, 151), ((20, 20), (0, 0), (20, 20)), 20000, 283)])
def test_checkpointed_fallback_takes_the_largest_launch_that_fits(lib, monkeypatch, n, pml, steps, S, share):
    import torch
    nshots, keep = 90, []
    d = _desc(keep, 2, n, pml, 4, _native.PYSIT_F32)
    d.nsteps, d.checkpoint_every, d.nshots = steps, S, nshots
    ptr = np.arange(nshots + 1, dtype=np.int64)
    amp, one, zero = np.ones((nshots, steps, 1)), np.ones(nshots), np.zeros(nshots, np.int32)
    cell = np.full(nshots, int(np.prod(n)) // 2, np.int64)
    keep += [ptr, amp, one, zero, cell]
    for k, v, t in (("src_tap_ptr", ptr, C.c_int64), ("src_tap_cell", cell, C.c_int64), ("src_tap_point", zero, C.c_int32),
                    ("src_tap_w", one, C.c_double), ("src_amp", amp, C.c_double), ("rec_tap_ptr", ptr, C.c_int64),
                    ("rec_tap_cell", cell, C.c_int64), ("rec_tap_point", zero, C.c_int32),
                    ("rec_tap_wsample", one, C.c_double), ("rec_tap_winject", one, C.c_double)):
        setattr(d, k, v.ctypes.data_as(C.POINTER(t)))
    size = lambda g: engine.WavePlan._workspace_for(lib, d, g, False)  # noqa: E731
    budget = int(share * size(nshots))
    reserve = 3 * nshots * steps * 4 + (2 << 30)
    monkeypatch.setattr(_native, "require_cuda", lambda: torch)
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda: (budget + reserve, 0))
    me = types.SimpleNamespace(nshots=nshots, nsteps=steps, tdtype=torch.float32, shots_per_launch=nshots, lanes=1,
                               _workspace_for=engine.WavePlan._workspace_for)
    made = []
    me._workspace_for = lambda *a: made.append(a) or engine.WavePlan._workspace_for(*a)
    assert engine.WavePlan._choose_schedule(me, lib, d, False, 1) == "checkpoint"
    g = me.shots_per_launch
    assert size(g) <= budget and len(made) < 40
    # no smaller number of equal launches fits
    fewest = next(k for k in range(1, nshots + 1) if size(-(-nshots // k)) <= budget)
    assert g == -(-nshots // fewest)
