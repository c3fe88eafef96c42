"""Device pointers of the stacked solver vector: the same as those of the sliced views."""
import types

import pytest
import torch

from pysit_gb300.solvers.cda_time import _CDATimeScalarCuda


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("shape", [(28, 1), (28,), (4, 7), (25, 1), (21, 1)])
def test_pointer_is_that_of_the_view(shape, dtype):
    dof = 7
    me = types.SimpleNamespace(mesh=types.SimpleNamespace(dof=lambda include_bc: dof))
    t = torch.zeros(shape, dtype=dtype)
    for i in range(5):
        want = t.reshape(-1)[i * dof:(i + 1) * dof].data_ptr()
        assert _CDATimeScalarCuda._field_ptr(me, t, i) == want
