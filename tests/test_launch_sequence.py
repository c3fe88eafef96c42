"""The order of a plan's copies, launches, events and waits, read on any host from a stand-in for the
CUDA runtime (fake_cudart.cpp, preloaded into a child process): no device, no kernel runs."""
import os
import shutil
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

CHILD = """
import ctypes as C, sys
import numpy as np
sys.path[:0] = [%r, %r]
from pysit_gb300 import _native
from test_task_tables import _desc
lib = _native.load()
fake = C.CDLL(None)
fake.fake_log.restype = C.c_char_p
keep = []
def plan(d):
    h, n = C.c_void_p(), C.c_uint64()
    _native.check(lib.pysit_plan_create(C.byref(d), C.byref(h)))
    _native.check(lib.pysit_plan_workspace_bytes(h, C.byref(n)))
    raw = np.empty(n.value + 256, np.uint8)
    keep.append(raw)
    p = (raw.ctypes.data + 255) // 256 * 256
    _native.check(lib.pysit_plan_bind_workspace(h, C.c_void_p(p), n, C.c_void_p(7)))
    return h
def model(h, d):
    c = np.full(d.n[0] * d.n[1] * d.n[2], 2000.0)
    keep.append(c)
    _native.check(lib.pysit_plan_set_model(h, C.c_void_p(c.ctypes.data), C.c_void_p(7)))
def log():
    return fake.fake_log().decode().splitlines()
""" % (ROOT, HERE)


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    from pysit_gb300 import build
    build.build()
    so = str(tmp_path_factory.mktemp("fake") / "fake_cudart.so")
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build._nvcc()))), "include")
    subprocess.run([shutil.which("g++"), "-shared", "-fPIC", "-std=c++17", "-I", inc,
                    os.path.join(HERE, "fake_cudart.cpp"), "-o", so], check=True)
    return so


def _run(fake, code, **env):
    r = subprocess.run([sys.executable, "-c", CHILD + code], capture_output=True, text=True,
                       env={**os.environ, "LD_PRELOAD": fake, **env})
    assert r.returncode == 0, r.stderr
    return r.stdout.splitlines()


@pytest.mark.parametrize("dim,n", [(1, (1, 1, 120)), (2, (40, 1, 36)), (3, (20, 18, 24))])
def test_bind_returns_with_the_workspace_complete(fake, dim, n):
    """Everything that bind enqueues is waited for before it returns, so that another stream may
    use the plan next."""
    out = _run(fake, f"d = _desc(keep, {dim}, {n}, ((4, 4),) * 3, 4, _native.PYSIT_F64)\n"
                     "plan(d)\nprint('\\n'.join(log()))")
    work = [i for i, l in enumerate(out) if l.split()[0] in ("launch", "memcpy", "memset")]
    assert any("one_sigma" in out[i] for i in work)
    assert "sync 7" in out[work[-1] + 1:]


TUNE = """
d = _desc(keep, {dim}, {n}, ((4, 4),) * 3, 4, _native.PYSIT_F64)
h = plan(d); model(h, d)
tile = C.c_int(); _native.check(lib.pysit_plan_get_tiles(h, C.byref(tile), None)); before = tile.value
cx, cz = (C.c_int * {nx})(*{cx}), (C.c_int * 1)(0)
x, z, ms = C.c_int(), C.c_int(), (C.c_double * {nx})()
fake.fake_clear()
_native.check(lib.pysit_plan_autotune_tiles(h, cx, {nx}, cz, 1, 3, C.byref(x), C.byref(z), ms, C.c_void_p(7)))
_native.check(lib.pysit_plan_get_tiles(h, C.byref(tile), None))
print(before, x.value, tile.value, sum(l.startswith("record") for l in log()) // 2, *ms)
"""


@pytest.mark.parametrize("times,chosen", [("1,2,2,1", 0), ("2,1,1,2", 8)])
def test_the_tuner_may_keep_the_default_length(fake, times, chosen):
    """A small 3D plan's default of one plane is a candidate (0), kept when it is the fastest."""
    out = _run(fake, TUNE.format(dim=3, n=(20, 18, 24), nx=2, cx=(0, 8)), FAKE_MS=times)
    before, x, tile, timed, *ms = out[-1].split()
    assert int(before) == 1 and int(x) == chosen and int(tile) == (chosen or 1)
    assert int(timed) == 4 and [float(v) for v in ms] == [float(v) for v in times.split(",")[:2]]


def test_the_3d_tuner_takes_lengths_down_to_one_plane(fake):
    out = _run(fake, TUNE.format(dim=3, n=(20, 18, 24), nx=4, cx=(64, 4, 2, 1)), FAKE_MS="4,3,2,1,1,2,3,4")
    assert out[-1].split()[:4] == ["1", "1", "1", "8"]


def test_lengths_that_give_the_same_2d_table_are_timed_once(fake):
    # blocks of three rows: every length gives the same tiles
    out = _run(fake, TUNE.format(dim=2, n=(300, 1, 36), nx=4, cx=(8, 64, 200, 0)), FAKE_MS="2,1")
    before, x, tile, timed, *ms = out[-1].split()
    assert (int(before), int(x), int(timed)) == (32, 8, 2) and [float(v) for v in ms] == [1, 1, 1, 1]


def test_the_tuner_tries_the_default():
    from pysit_gb300 import engine
    assert all(c[0] == 0 for c in engine.TILE_CANDIDATES.values()) and 1 in engine.TILE_CANDIDATES[3]


@pytest.mark.parametrize("nz,dtype,largest,cluster", [(1500, "F64", 16, 16), (1500, "F64", 8, 0), (1200, "F64", 16, 16),
                                                      (1200, "F64", 8, 8), (1200, "F64", 0, 0), (300, "F32", 16, 1),
                                                      (300, "F32", 0, 0)])
def test_1d_runs_use_a_cluster_that_the_device_places(fake, nz, dtype, largest, cluster):
    """Where the device places no cluster of a run's size, a smaller one is taken, or a launch per step."""
    out = _run(fake, f"d = _desc(keep, 1, (1, 1, {nz}), ((0, 0), (0, 0), (9, 9)), 4, _native.PYSIT_{dtype})\n"
                     "h = plan(d); model(h, d); fake.fake_clear()\n"
                     "tr = np.zeros(8)\n"
                     "_native.check(lib.pysit_plan_forward(h, C.c_void_p(tr.ctypes.data), C.c_void_p(7)))\n"
                     "print('\\n'.join(log()))", FAKE_MAX_CLUSTER=str(largest))
    runs = [l for l in out if "wave1d_sweep_kernel" in l]
    steps = [l for l in out if "wave1d_kernel" in l]
    assert [int(l.split()[-1]) for l in runs] == ([cluster] if cluster else [])
    assert len(steps) == (0 if cluster else 8)


@pytest.mark.parametrize("nshots,dtype,runs", [(64, "F64", 1), (128, "F64", 0), (128, "F32", 1), (512, "F32", 0)])
def test_1d_launches_that_fill_the_gpu_step_one_launch_at_a_time(fake, nshots, dtype, runs):
    out = _run(fake, f"d = _desc(keep, 1, (1, 1, 799), ((0, 0), (0, 0), (10, 10)), 4, _native.PYSIT_{dtype})\n"
                     f"n = {nshots}\nd.nshots = d.shots_per_launch = n\n"
                     "ptr = np.arange(n + 1, dtype=np.int64); one = np.ones(n); pt = np.zeros(n, np.int32)\n"
                     "cell = np.full(n, 400, np.int64); amp = np.ones((n, 8, 1))\n"
                     "P = lambda a, t: a.ctypes.data_as(C.POINTER(t))\n"
                     "d.src_tap_ptr = d.rec_tap_ptr = P(ptr, C.c_int64); d.src_tap_cell = d.rec_tap_cell = P(cell, C.c_int64)\n"
                     "d.src_tap_point = d.rec_tap_point = P(pt, C.c_int32); d.src_amp = P(amp, C.c_double)\n"
                     "d.src_tap_w = d.rec_tap_wsample = d.rec_tap_winject = P(one, C.c_double)\n"
                     "h = plan(d); model(h, d); fake.fake_clear()\n"
                     "tr = np.zeros(8 * n)\n"
                     "_native.check(lib.pysit_plan_forward(h, C.c_void_p(tr.ctypes.data), C.c_void_p(7)))\n"
                     "print('\\n'.join(log()))")
    assert sum("wave1d_sweep_kernel" in l for l in out) == runs
    assert sum("wave1d_kernel" in l for l in out) == (0 if runs else 8)


@pytest.mark.parametrize("nz,cluster", [(1200, 8), (1500, 0)])
def test_a_refused_cluster_attribute_is_no_error_of_the_plan(fake, nz, cluster):
    out = _run(fake, f"d = _desc(keep, 1, (1, 1, {nz}), ((0, 0), (0, 0), (9, 9)), 4, _native.PYSIT_F64)\n"
                     "h = plan(d); model(h, d); fake.fake_clear()\n"
                     "tr = np.zeros(8)\n"
                     "_native.check(lib.pysit_plan_forward(h, C.c_void_p(tr.ctypes.data), C.c_void_p(7)))\n"
                     "print('\\n'.join(log()))", FAKE_PORTABLE="1")
    assert [int(l.split()[-1]) for l in out if "wave1d_sweep_kernel" in l] == ([cluster] if cluster else [])
