"""dJ/dC for an FP32 C is the FP64 result for the same values, rounded to FP32."""
import numpy as np
import pytest

import problems
import pysit_gb300 as api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["o2", "3d", "1d"])
def test_fp32_model_gives_the_rounded_gradient(name):
    import torch
    from pysit_gb300.autograd import FWIMisfit
    m, shots, solver, C, C0 = problems.build(api, name)
    api.generate_seismic_data(shots, solver, solver.ModelParameters(m, {"C": C}))
    obs = torch.as_tensor(np.stack([s.receivers.data for s in shots]))
    ts = solver.ts()
    values = torch.as_tensor(np.asarray(C0), dtype=torch.float32)
    grads = []
    for dtype in (torch.float32, torch.float64):
        c = values.to(dtype).clone().requires_grad_()
        FWIMisfit(solver, shots, obs, ts)(c).backward()
        assert c.grad.dtype == dtype
        grads.append(c.grad.double())
    assert grads[1].abs().max() > 0
    # one rounding to FP32 (2^-24 relative), the rest is FP64 rounding; 2^-149 for subnormals
    assert ((grads[0] - grads[1]).abs() <= 6.0e-8 * grads[1].abs() + 1.5e-45).all()
