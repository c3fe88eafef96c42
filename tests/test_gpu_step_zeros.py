"""Per-step kernels where derivative terms drop out: PML fields that are zero outside the
padding, a psi that is not finite beside cells without a product of sigmas, and dWaveOp on grids
with few rows.  Same tolerances as the parity of the full step."""
import ctypes as C

import numpy as np
import pytest

import pipeline
from test_gpu_step import _gpu_step, _inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("dim,shape,order", [(1, [259], 4), (2, [9, 33], 2), (3, [11, 9, 34], 4), (3, [12, 13, 32], 8)])
def test_fields_zero_outside_the_padding(dim, shape, order, dtype):
    rng = np.random.default_rng(dim + order)
    km1, aux, k, Cm, rhs, prof = _inputs(dim, shape, dtype, rng)
    pad = np.zeros(shape, bool)
    for ax, n in enumerate(shape):
        pos = np.arange(n).reshape([-1 if a == ax else 1 for a in range(dim)])
        pad |= (pos < 3) | (pos >= n - 4)
    for name in aux:
        aux[name] = (aux[name].reshape(shape) * (pad if name != "psi" else 1)).ravel().astype(dtype)
    deltas = [7.0, 9.0, 11.0][:dim]
    ref_u, ref_aux = pipeline.step("oracle", dim, order, km1, aux, k, Cm, rhs, prof, 1e-3, deltas, shape)
    u, a = _gpu_step(dim, order, km1, aux, k, Cm, rhs, prof, 1e-3, deltas, shape)
    tol = 1e-13 if dtype == np.float64 else 3e-5
    assert np.abs(u - ref_u).max() <= tol * np.abs(ref_u).max()
    for name in aux:
        assert np.abs(a[name] - ref_aux[name]).max() <= tol * max(np.abs(ref_aux[name]).max(), 1e-30), name


@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("name", ["psi", "Phiz"])
def test_not_finite_spreads_as_in_the_oracle(name, value):
    shape = [13, 12, 15]
    km1, aux, k, Cm, rhs, prof = _inputs(3, shape, np.float64, np.random.default_rng(5))
    aux[name] = aux[name].reshape(shape).copy()
    aux[name][1, 6, 7] = value  # one axis in the padding: every product of sigmas is zero
    aux[name] = aux[name].ravel()
    args = (km1, aux, k, Cm, rhs, prof, 1e-3, [7.0, 9.0, 11.0], shape)
    ref_u, ref_aux = pipeline.step("oracle", 3, 4, *args)
    u, a = _gpu_step(3, 4, *args)
    np.testing.assert_array_equal(np.isfinite(u), np.isfinite(ref_u))
    for f in aux:
        np.testing.assert_array_equal(np.isfinite(a[f]), np.isfinite(ref_aux[f]))


@pytest.mark.parametrize("dim,shape", [(1, [5]), (1, [1031]), (2, [7, 257]), (2, [9, 31]), (3, [3, 3, 300])])
def test_dwaveop_few_rows(dim, shape):
    import torch
    from pysit_gb300 import _native
    rng = np.random.default_rng(6)
    um, uc, up, psi = (rng.standard_normal(int(np.prod(shape))) for _ in range(4))
    maps = [np.abs(rng.standard_normal(n)) * (np.arange(n) < 4) * 10 for n in shape]
    ref = pipeline.dwaveop(dict(dim=dim, dt=1e-3, shape=shape, sigmaps=maps), um, uc, up, psi if dim == 3 else None)
    dev = [torch.as_tensor(a, device="cuda") for a in (um, uc, up, psi)]
    sg = [torch.as_tensor(m, device="cuda") for m in maps]
    sg, dims = {1: ([None, None] + sg, [1, 1] + shape), 2: (sg[:1] + [None] + sg[1:], [shape[0], 1, shape[-1]]),
                3: (sg, shape)}[dim]
    ptr = lambda x: None if x is None else C.c_void_p(x.data_ptr())  # noqa: E731
    out = torch.zeros_like(dev[0])
    _native.check(_native.load().pysit_cda_dwaveop(
        _native.PYSIT_F64, dim, *[ptr(x) for x in dev[:3]], ptr(dev[3]) if dim == 3 else None,
        *[ptr(x) for x in sg], *dims, 1e-3, ptr(out), _native.stream_handle()))
    np.testing.assert_allclose(out.cpu().numpy(), ref, rtol=1e-12, atol=1e-12 * np.abs(ref).max())
