"""2D launches of more than 48 MB of wavefields, whose blocks fetch the next shot's tile into L2: the same
numbers to the last bit as in launches of a few shots, which do not."""
import numpy as np
import pytest

from pysit_gb300.engine import WavePlan
from test_gpu_tiles2d import _build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,nshots", [("single", 81), ("double", 41)])
@pytest.mark.parametrize("nx,nz,npml", [(301, 201, 9)])
def test_fetching_ahead_changes_nothing(nx, nz, npml, precision, nshots):
    import torch
    steps = 8
    solver, shots = _build(nx, nz, npml, nshots, 8, precision, steps)
    field = (nx + 2 * npml + 8) * 256 * (4 if precision == "single" else 8)
    assert 2 * field * nshots > 48 << 20 > 2 * field * 9
    rng = np.random.default_rng(7)
    dobs = rng.standard_normal((nshots, steps, 23)) * 1e-3
    m1 = torch.as_tensor(1e-9 * rng.standard_normal(nx * nz))
    out = []
    for G in (nshots, 9):
        plan = WavePlan(solver, shots, shots_per_launch=G, checkpoint_every=3, use_graph=False)
        tr = plan.forward().cpu().numpy().copy()
        plan.load_observed(dobs)
        g, _ = plan.gradient()
        out.append((tr, plan.born(m1).cpu().numpy().copy(), g.cpu().numpy().copy()))
        assert plan.check_status() == 0
        del plan
    (tr, born, g), (tr1, born1, g1) = out
    assert np.abs(tr).max() > 0 and np.abs(born).max() > 0 and np.abs(g).max() > 0
    np.testing.assert_array_equal(tr, tr1)
    np.testing.assert_array_equal(born, born1)
    # the shots' images are summed in FP64 in the same order: the rounding of a sum of nshots terms
    assert np.linalg.norm(g - g1) <= nshots * 2.3e-16 * np.linalg.norm(g1) * 10
