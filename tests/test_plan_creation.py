"""Host cost of creating a plan: the task table is built once for its shots, not once for every
tile length and extent that the tuner could ask for."""
import ctypes as C
import time

import numpy as np
import pytest

from pysit_gb300 import _native
from test_task_tables import _desc


@pytest.fixture(scope="module")
def lib():
    from pysit_gb300 import build
    build.build()
    return _native.load()


@pytest.mark.parametrize("dim,n,pml,nshots", [(2, (1232, 1, 464), ((40, 40), (0, 0), (40, 40)), 1000),
                                              (3, (220, 220, 170), ((20, 20),) * 3, 300)])
def test_creation_does_not_rebuild_the_table(lib, dim, n, pml, nshots):
    keep = []
    d = _desc(keep, dim, n, pml, 8, _native.PYSIT_F32)
    d.nshots = d.shots_per_launch = nshots
    cells = np.random.default_rng(0).integers(0, int(np.prod(n)), nshots)
    arrs = dict(src_tap_ptr=np.arange(nshots + 1, dtype=np.int64), src_tap_cell=cells, src_tap_w=np.ones(nshots),
                src_tap_point=np.zeros(nshots, np.int32), src_amp=np.ones((nshots, 8, 1)),
                rec_tap_ptr=np.arange(nshots + 1, dtype=np.int64), rec_tap_cell=cells[::-1].copy(),
                rec_tap_point=np.zeros(nshots, np.int32), rec_tap_wsample=np.ones(nshots), rec_tap_winject=np.ones(nshots))
    ct = {np.int64: C.c_int64, np.int32: C.c_int32, np.float64: C.c_double}
    for k, v in arrs.items():
        keep.append(v)
        setattr(d, k, v.ctypes.data_as(C.POINTER(ct[v.dtype.type])))
    best = 1e9
    for _ in range(5):
        t = time.process_time()
        h = C.c_void_p()
        _native.check(lib.pysit_plan_create(C.byref(d), C.byref(h)))
        best = min(best, time.process_time() - t)
        lib.pysit_plan_destroy(h)
    # about 10 ms; building the table sixty times took 160 ms and more
    assert best < 0.06
