"""3D step kernel on the GPU: the planes per thread and the tile length follow from the launch's
size, and every choice gives the same numbers to the last bit.

One plan steps all shots in one launch (four planes per thread), one steps a shot at a time (one
plane), one has a fixed tile length.  The sizes put remainders everywhere: x chunks that are no
multiple of four, z extents that are not a multiple of the vector, one- and two-row y groups."""
import numpy as np
import pytest

import pysit_gb300 as api
from pysit_gb300.engine import WavePlan

pytestmark = pytest.mark.gpu

# (nx, ny, nz, PML cells, shots): 1.3 million padded cells x shots and more
SIZES = [(31, 29, 37, 5, 24), (22, 35, 18, 6, 40), (19, 17, 131, 4, 16)]


@pytest.mark.parametrize("pml_psi", ["reference", "consistent"])
@pytest.mark.parametrize("precision", ["single", "double"])
@pytest.mark.parametrize("order", [2, 4, 8])
@pytest.mark.parametrize("size", range(len(SIZES)))
def test_planes_per_thread_do_not_change_the_results(size, order, precision, pml_psi):
    nx, ny, nz, npml, nshots = SIZES[size]
    steps, dx = 10, 10.0
    pml = api.PML(npml * dx, 5.0)
    ext = [(n - 1) * dx for n in (nx, ny, nz)]
    m = api.CartesianMesh(api.RectangularDomain(*[(0.0, e, pml, pml) for e in ext]), nx, ny, nz)
    rng = np.random.default_rng(nx)
    C = 1500.0 + 2500.0 * rng.random((nx * ny * nz, 1))
    dt = 0.3 * dx / C.max()
    w = api.RickerWavelet(25.0, shift_deviations=1)
    at = lambda f: tuple(e * v for e, v in zip(ext, f))  # noqa: E731
    rec = [api.PointReceiver(m, at(rng.random(3))) for _ in range(11)]
    shots = [api.Shot(api.PointSource(m, at(rng.random(3)), w), api.ReceiverSet(m, rec)) for _ in range(nshots)]
    solver = api.ConstantDensityAcousticWave(m, spatial_accuracy_order=order, trange=(0.0, (steps - 0.5) * dt),
                                             kernel_implementation="cuda", precision=precision, cfl_safety=0.3,
                                             pml_psi=pml_psi)
    solver.model_parameters = solver.ModelParameters(m, {"C": C})
    dobs = rng.standard_normal((nshots, steps, 11)) * 1e-3
    out = []
    for G in (nshots, 1):
        plan = WavePlan(solver, shots, shots_per_launch=G, checkpoint_every=4, use_graph=False)
        tr = plan.forward().cpu().numpy().copy()
        plan.load_observed(dobs)
        g, rn = plan.gradient()
        out.append((tr, g.cpu().numpy().copy(), float(rn.item())))
        if G > 1:  # any tile length gives the same
            plan.autotune(candidates=(23,), nsteps=1, z_candidates=(16,))
            np.testing.assert_array_equal(plan.forward().cpu().numpy(), tr)
        assert plan.check_status() == 0
        del plan
    (tr, g, rn), (tr1, g1, rn1) = out
    assert np.abs(tr).max() > 0 and np.abs(g).max() > 0
    np.testing.assert_array_equal(tr, tr1)
    # the shots' images are summed in FP64 in the same order, in launches of all or of one:
    # the rounding of a sum of nshots terms
    assert np.linalg.norm(g - g1) <= nshots * 2.3e-16 * np.linalg.norm(g1) * 10
    assert rn == pytest.approx(rn1, rel=1e-12)
