"""2D step kernel on the GPU: the rows per thread follow from the launch's size, and every choice
gives the same numbers to the last bit.

One plan steps all shots in one launch (more rows per thread), the other one shot at a time (one
row per thread on these grids; the parity tests hold that path to the oracle).  The sizes put the
edges of tiles everywhere: interiors of no whole tile, one-row remainders, z extents that are not
a multiple of the vector, several z segments, a grid that is all PML shell."""
import numpy as np
import pytest

import pysit_gb300 as api
from pysit_gb300.engine import WavePlan

pytestmark = pytest.mark.gpu

# (nx, nz, PML cells, shots): padded cells x shots of about 0.33, 1.3 and 2.6 million
SIZES = [(131, 77, 8, 24), (257, 143, 9, 30), (61, 391, 7, 80), (1003, 18, 30, 42)]


def _build(nx, nz, npml, nshots, order, precision, steps):
    dx = 10.0
    pml = api.PML(npml * dx, 3000.0 / npml)
    d = api.RectangularDomain((0.0, (nx - 1) * dx, pml, pml), (0.0, (nz - 1) * dx, pml, pml))
    m = api.CartesianMesh(d, nx, nz)
    rng = np.random.default_rng(nx)
    C = 1500.0 + 2500.0 * rng.random((nx * nz, 1))
    dt = 0.4 * dx / C.max()
    w = api.RickerWavelet(25.0, shift_deviations=1)
    rec = [api.PointReceiver(m, (x, z)) for x, z in zip(np.linspace(0, (nx - 1) * dx, 23),
                                                        np.linspace(0, (nz - 1) * dx, 23))]
    shots = [api.Shot(api.PointSource(m, ((nx - 1) * dx * (i + 0.5) / nshots, (nz - 1) * dx * ((i * 7) % nshots) / nshots), w),
                      api.ReceiverSet(m, rec)) for i in range(nshots)]
    solver = api.ConstantDensityAcousticWave(m, spatial_accuracy_order=order, trange=(0.0, (steps - 0.5) * dt),
                                             kernel_implementation="cuda", precision=precision, cfl_safety=0.4)
    solver.model_parameters = solver.ModelParameters(m, {"C": C})
    return solver, shots


@pytest.mark.parametrize("precision", ["single", "double"])
@pytest.mark.parametrize("order", [2, 6, 8])
@pytest.mark.parametrize("size", range(len(SIZES)))
def test_rows_per_thread_do_not_change_the_results(size, order, precision):
    import torch
    nx, nz, npml, nshots = SIZES[size]
    steps = 12
    solver, shots = _build(nx, nz, npml, nshots, order, precision, steps)
    rng = np.random.default_rng(5)
    dobs = rng.standard_normal((nshots, steps, 23)) * 1e-3
    m1 = 1e-9 * rng.standard_normal(nx * nz)
    out = []
    for G in (nshots, 1):
        plan = WavePlan(solver, shots, shots_per_launch=G, checkpoint_every=5, use_graph=False)
        tr = plan.forward().cpu().numpy().copy()
        plan.load_observed(dobs)
        g, rn = plan.gradient()
        born = plan.born(torch.as_tensor(m1)).cpu().numpy().copy()
        out.append((tr, born, g.cpu().numpy().copy(), float(rn.item())))
        assert plan.check_status() == 0
        del plan
    (tr, born, g, rn), (tr1, born1, g1, rn1) = out
    assert np.abs(tr).max() > 0 and np.abs(born).max() > 0 and np.abs(g).max() > 0
    np.testing.assert_array_equal(tr, tr1)
    np.testing.assert_array_equal(born, born1)
    # the shots' images are summed in FP64 in the same order, in launches of all or of one:
    # the rounding of a sum of nshots terms
    assert np.linalg.norm(g - g1) <= nshots * 2.3e-16 * np.linalg.norm(g1) * 10
    assert rn == pytest.approx(rn1, rel=1e-12)
