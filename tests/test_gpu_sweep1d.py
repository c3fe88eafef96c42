"""1D runs of steps in one cluster launch against the same runs stepped one launch at a time.

Grids that fill one block, straddle two, fill a cluster of eight with a short last block, and one
longer than a cluster takes (stepped launch by launch on both sides); several shots, receivers whose
taps straddle blocks, ragged segments, imaging periods and record lengths.  The reference is the CPU
oracle in FP64; in FP32 the FP64 run, at the parity tolerances of the other tests."""
import numpy as np
import pytest

import pipeline
import problems
import pysit_gb300 as api
from pysit_gb300.engine import WavePlan

pytestmark = pytest.mark.gpu


def _build(n, order, precision, steps, nshots, nrec, npml):
    dx = 10.0
    pml = api.PML(npml * dx, 200.0)
    m = api.CartesianMesh(api.RectangularDomain((0.0, (n - 1) * dx, pml, pml)), n)
    rng = np.random.default_rng(n)
    C = 1500.0 + 2000.0 * rng.random((n, 1))
    dt = 0.5 * dx / C.max()
    w = api.RickerWavelet(25.0, shift_deviations=1)
    z = np.linspace(0.0, (n - 1) * dx, nrec)
    shots = [api.Shot(api.PointSource(m, ((n - 1) * dx * (i + 0.3) / nshots,), w),
                      api.ReceiverSet(m, [api.PointReceiver(m, (float(v),)) for v in z])) for i in range(nshots)]
    solver = api.ConstantDensityAcousticWave(m, spatial_accuracy_order=order, trange=(0.0, (steps - 0.5) * dt),
                                             kernel_implementation="cuda", precision=precision, cfl_safety=0.5)
    solver.model_parameters = solver.ModelParameters(m, {"C": C})
    return solver, shots


@pytest.mark.parametrize("order", [2, 8])
@pytest.mark.parametrize("n,nshots,nrec,npml", [(20, 1, 3, 5), (53, 2, 5, 6), (490, 3, 17, 7), (1201, 1, 40, 20),
                                                (4200, 1, 2, 10), (4200, 2, 60, 10)])
def test_runs_of_steps_match_the_oracle(n, nshots, nrec, npml, order):
    steps = 45
    rng = np.random.default_rng(1)
    out = {}
    for precision in ("double", "single"):
        solver, shots = _build(n, order, precision, steps, nshots, nrec, npml)
        dobs = rng.standard_normal((nshots, steps, nrec)) if precision == "double" else dobs
        for schedule, S in (("checkpoint", 7), ("store", 7)):
            plan = WavePlan(solver, shots, gradient_schedule=schedule, checkpoint_every=S)
            for _ in range(3):  # eager, captured, replayed
                plan.load_observed(dobs)
                g, rn = plan.gradient(with_traces=True)
            out[precision, schedule] = (plan.traces.cpu().numpy().copy(), g.cpu().numpy().copy(), float(rn.item()))
            assert plan.check_status() == 0
        if precision == "double":
            P = [problems.oracle_problem(solver, s) for s in shots]
            ref_tr = np.stack([pipeline.forward(p)[0] for p in P])
            ref_g, _ = pipeline.gradient(P, list(dobs))
    close = lambda a, b, tol: np.linalg.norm(a - b) <= tol * np.linalg.norm(b)  # noqa: E731
    tr, g, rn = out["double", "checkpoint"]
    assert close(tr, ref_tr, 1e-11) and close(g, ref_g, 1e-9)
    for precision in ("double", "single"):  # both schedules compute the same numbers
        a, b = out[precision, "checkpoint"], out[precision, "store"]
        np.testing.assert_array_equal(a[0], b[0])
        np.testing.assert_array_equal(a[1], b[1])
    tr32, g32, _ = out["single", "checkpoint"]
    assert close(tr32, tr, 1e-4) and close(g32, g, 1e-3)
