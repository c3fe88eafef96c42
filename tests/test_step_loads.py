"""Loads of the overlapping step kernels, checked in the source (no GPU).

A step kernel starts while the one before it runs, so what that one writes (wavefields, Phi, psi,
dWaveOp, the image) may change while this one lives.  ``__ldg`` is defined only for data that stay
constant as long as a kernel lives; here it may reach C^2, m1, the sigma tables, the tile tables, the
injection operators with their amplitudes, and the recorder's taps, and nothing else."""
import os
import re

import pytest

from pysit_gb300 import build

# read-only data: members of WaveParams (p), Inject (inj), Record (p.rec), and locals that point into them
CONSTANT = re.compile(r"p\.(c2|m1|(sg|mg|fc)[xyz]|rec\.(rowptr|off|w))\b|\binj\.(w|pt)\b|^\s*(bx|rp|amp)\b|\btiles\b")
WRITTEN = re.compile(r"\b(u_cur|u_prev|ph[xyz]_(in|out)|psi_(in|out)|dw_(in|out)|ic)\b|^\s*(u|ur|q)\b")


def _calls(text, name):
    """Argument texts of the calls of `name` in a source without comments."""
    for m in re.finditer(r"(?<![\w.])" + name + r"\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        yield m.start(), text[m.end():i - 1]


def _source(name):
    with open(os.path.join(build.CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


@pytest.mark.parametrize("name", ["wave.cuh", "pairs.cuh", "wave2d_tile.cuh", "wave3d_tile.cuh"])
def test_the_read_only_path_reaches_only_what_no_step_writes(name):
    text = _source(name)
    seen = 0
    helper = [m.span() for m in re.finditer(r"void ldr\([^{]*\{[^}]*\}", text)]  # ldr's own definition
    for at, arg in list(_calls(text, "__ldg")):
        if any(a <= at < b for a, b in helper):
            continue
        arg = re.sub(r"reinterpret_cast<[^>]*>\(", "", arg)
        assert CONSTANT.search(arg) and not WRITTEN.search(arg), f"{name}: __ldg({arg})"
        seen += 1
    for at, arg in _calls(text, "ldr"):
        if any(a <= at < b for a, b in helper):
            continue
        src = arg.split(",", 1)[1]
        assert CONSTANT.search(src) and not WRITTEN.search(src), f"{name}: ldr({arg})"
        seen += 1
    assert seen > 0 or name == "pairs.cuh"


def test_the_check_sees_a_wavefield_behind_the_read_only_path():
    for arg in ("u + off[q]", "p.u_cur + sh + o", "p.phx_in + sh + o", "p.dw_in + sh + o", "q + j * 2 * NP"):
        assert WRITTEN.search(arg) or not CONSTANT.search(arg)
