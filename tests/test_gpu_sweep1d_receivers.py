"""1D runs in one cluster launch with many receivers: a warp per receiver up to four times the blocks, a
thread per receiver above (whole and ragged groups of 32, several rounds a block), taps across blocks and at
both ends of the grid; against the CPU oracle in FP64, and FP32 against FP64."""
import numpy as np
import pytest

import pipeline
import problems
from pysit_gb300.engine import WavePlan
from test_gpu_sweep1d import _build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nshots,nrec", [(480, 1, 31), (480, 1, 33), (480, 2, 130), (480, 1, 480), (50, 3, 50),
                                           (1300, 1, 1025), (1300, 1, 1300), (9, 2, 9)])
def test_traces_of_many_receivers(n, nshots, nrec):
    steps = 20
    rng = np.random.default_rng(n + nrec)
    dobs = rng.standard_normal((nshots, steps, nrec))
    out = {}
    for precision in ("double", "single"):
        solver, shots = _build(n, 4, precision, steps, nshots, nrec, 6)
        plan = WavePlan(solver, shots, checkpoint_every=6, use_graph=False)
        plan.load_observed(dobs)
        g, _ = plan.gradient(with_traces=True)
        out[precision] = plan.traces.cpu().numpy().copy(), g.cpu().numpy().copy()
        assert plan.launches() < 3 * steps  # runs of steps, not steps
        if precision == "double":
            P = [problems.oracle_problem(solver, s) for s in shots]
            ref_tr = np.stack([pipeline.forward(p)[0] for p in P])
            ref_g, _ = pipeline.gradient(P, list(dobs))
    close = lambda a, b, tol: np.linalg.norm(a - b) <= tol * np.linalg.norm(b)  # noqa: E731
    assert close(out["double"][0], ref_tr, 1e-11) and close(out["double"][1], ref_g, 1e-9)
    assert close(out["single"][0], out["double"][0], 1e-4) and close(out["single"][1], out["double"][1], 1e-3)
