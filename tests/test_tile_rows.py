"""Rows of the step kernels' tiles against the threads that step them: a row past the last thread's would
not be stepped.  Tables and block shapes read back on the host (no GPU), for launches small and large
enough for every block size and number of rows per thread."""
import ctypes as C

import numpy as np
import pytest

from pysit_gb300 import _native
from test_task_tables import _desc


@pytest.fixture(scope="module")
def lib():
    from pysit_gb300 import build
    build.build()
    return _native.load()


def _plan(lib, keep, dim, n, pml, order, dtype, tiles, nshots):
    d = _desc(keep, dim, n, pml, order, dtype, *tiles)
    d.nshots = d.shots_per_launch = nshots
    ptr, one = np.zeros(nshots + 1, np.int64), np.ones((nshots, 8, 1))  # no taps
    keep += [ptr, one]
    d.src_tap_ptr = d.rec_tap_ptr = ptr.ctypes.data_as(C.POINTER(C.c_int64))
    d.src_amp = one.ctypes.data_as(C.POINTER(C.c_double))
    h, k, t, r = C.c_void_p(), C.c_uint64(), C.c_int(), C.c_int()
    _native.check(lib.pysit_plan_create(C.byref(d), C.byref(h)))
    _native.check(lib.pysit_plan_task_table(h, None, 0, C.byref(k), None))
    tab = np.zeros(k.value, np.int32)
    _native.check(lib.pysit_plan_task_table(h, tab.ctypes.data_as(C.POINTER(C.c_int32)), k.value, None, None))
    _native.check(lib.pysit_plan_get_blocks(h, C.byref(t), C.byref(r)))
    lib.pysit_plan_destroy(h)
    return tab.reshape(-1, 6 if dim == 3 else 5), t.value, r.value


def _too_tall_2d(tasks, threads, rows):
    cells = np.where(tasks[:, 4] == 0, 4, 2)  # of a thread along z
    columns = -(-(tasks[:, 3] - tasks[:, 2]) // cells)
    return (tasks[:, 1] - tasks[:, 0]) > threads // columns * rows


def _too_tall_3d(tasks, threads, dtype):
    vectors = -(-(tasks[:, 5] - tasks[:, 4]) // (4 if dtype == _native.PYSIT_F32 else 2))
    return (vectors > 32) | ((tasks[:, 3] - tasks[:, 2]) > threads // 32 * (32 // np.minimum(vectors, 32)))


@pytest.mark.parametrize("dtype", [_native.PYSIT_F32, _native.PYSIT_F64])
@pytest.mark.parametrize("order", [2, 8])
@pytest.mark.parametrize("tiles", [(0, 0), (5, 0), (8, 16), (64, 96)])
def test_2d_rows(lib, order, dtype, tiles):
    seen = set()
    for (nx, nz), nshots in (((141, 81), 1), ((141, 81), 12), ((461, 203), 9), ((1232, 464), 1), ((1232, 464), 20),
                             ((57, 433), 40), ((70, 19), 3)):
        tasks, threads, rows = _plan(lib, [], 2, (nx, 1, nz), ((9, 9), (0, 0), (9, 9)), order, dtype, tiles, nshots)
        seen.add((threads, rows))
        assert threads in (32, 64, 128) and not _too_tall_2d(tasks, threads, rows).any()
        worst = tasks.copy()
        full = int(np.argmax(tasks[:, 1] - tasks[:, 0]))
        columns = -(-(tasks[full, 3] - tasks[full, 2]) // (4 if tasks[full, 4] == 0 else 2))
        worst[full, 1] = worst[full, 0] + threads // columns * rows + 1  # one row too tall: seen
        assert _too_tall_2d(worst, threads, rows).any()
    assert len(seen) >= 3


@pytest.mark.parametrize("dtype", [_native.PYSIT_F32, _native.PYSIT_F64])
@pytest.mark.parametrize("order", [2, 8])
@pytest.mark.parametrize("tiles", [(0, 0), (1, 0), (8, 16), (16, 36), (64, 96)])
def test_3d_rows(lib, order, dtype, tiles):
    seen = set()
    for n, nshots in (((53, 49, 45), 2), ((121, 107, 95), 4), ((30, 44, 171), 1), ((24, 26, 45), 60)):
        tasks, threads, planes = _plan(lib, [], 3, n, ((6, 6),) * 3, order, dtype, tiles, nshots)
        seen.add((threads, planes))
        assert threads in (64, 128) and not _too_tall_3d(tasks, threads, dtype).any()
        worst = tasks.copy()
        vectors = -(-(worst[0, 5] - worst[0, 4]) // (4 if dtype == _native.PYSIT_F32 else 2))
        worst[0, 3] = worst[0, 2] + threads // 32 * (32 // vectors) + 1
        assert _too_tall_3d(worst, threads, dtype).any()
    assert seen == {(64, 1), (128, 4)}
