"""Workspace of checkpointed plans of small launches: the second replay buffer, into which a segment is
recomputed while the adjoint reads the one after it, is bounded."""
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


def _bytes(lib, dim, n, pml, nsteps, S, nshots=1):
    keep = []
    d = _desc(keep, dim, n, pml, 8, _native.PYSIT_F32)
    d.nsteps, d.checkpoint_every, d.nshots, d.shots_per_launch = nsteps, S, nshots, nshots
    ptr = np.arange(nshots + 1, dtype=np.int64)
    amp, one, zero = np.ones((nshots, nsteps, 1)), np.ones(nshots), np.zeros(nshots, np.int32)
    cell = np.full(nshots, int(np.prod(n)) // 2, np.int64)
    keep += [ptr, amp, one, zero, cell]
    for k, v, t in (("src_tap_ptr", ptr, C.c_int64), ("src_tap_cell", cell, C.c_int64), ("src_tap_point", zero, C.c_int32),
                    ("src_tap_w", one, C.c_double), ("src_amp", amp, C.c_double), ("rec_tap_ptr", ptr, C.c_int64),
                    ("rec_tap_cell", cell, C.c_int64), ("rec_tap_point", zero, C.c_int32),
                    ("rec_tap_wsample", one, C.c_double), ("rec_tap_winject", one, C.c_double)):
        setattr(d, k, v.ctypes.data_as(C.POINTER(t)))
    h, b = C.c_void_p(), C.c_uint64()
    _native.check(lib.pysit_plan_create(C.byref(d), C.byref(h)))
    _native.check(lib.pysit_plan_workspace_bytes(h, C.byref(b)))
    lib.pysit_plan_destroy(h)
    return b.value


@pytest.mark.parametrize("dim,n,pml,nsteps,S,nshots,rows", [
    (2, (1232, 1, 464), ((40, 40), (0, 0), (40, 40)), 4000, 2000, 2, 1232 + 8),
    (1, (1, 1, 500000), ((0, 0), (0, 0), (40, 40)), 2000, 600, 4, 1),
    (3, (90, 90, 90), ((10, 10),) * 3, 3000, 1500, 1, 98 * 98)])
def test_long_segments_have_one_replay_buffer(lib, dim, n, pml, nsteps, S, nshots, rows):
    field = rows * (-(-(4 + n[2] + 12) // 32) * 32) * 4 * nshots
    fields = S + {1: 3, 2: 4, 3: 6}[dim] * -(-nsteps // S) + 40  # replay, checkpoints, states and the rest
    assert _bytes(lib, dim, n, pml, nsteps, S, nshots) < fields * field


def test_short_segments_have_two(lib):
    """(the rule's other side: a default segment of a small launch still overlaps)"""
    n, pml = (141, 1, 81), ((10, 10), (0, 0), (10, 10))
    field = (141 + 8) * 128 * 4
    a, b = _bytes(lib, 2, n, pml, 360, 38), _bytes(lib, 2, n, pml, 38, 38)  # ten segments; one: nothing to overlap
    assert a - b > 38 * field
