"""Rounding of the per-step kernels in FP64: the error against extended precision is no larger than
that of the reference's own order of operations (taps summed one by one, 1/h last, three quotients
in the padding), evaluated here with a rounding after every fused multiply-add."""
import numpy as np
import pytest

import pipeline
from test_gpu_step import _gpu_step

pytestmark = pytest.mark.gpu
L = np.longdouble
W1 = {2: [(1, 2)], 4: [(2, 3), (-1, 12)], 6: [(3, 4), (-3, 20), (1, 60)], 8: [(4, 5), (-1, 5), (4, 105), (-1, 280)]}
W2 = {2: [(-2, 1), (1, 1)], 4: [(-5, 2), (4, 3), (-1, 12)], 6: [(-49, 18), (3, 2), (-3, 20), (1, 90)],
      8: [(-205, 72), (8, 5), (-1, 5), (8, 315), (-1, 560)]}


def _fma(a, b, c):
    return (L(a) * b + c).astype(np.float64)


@pytest.mark.parametrize("spacing", [10.0, 7.3])
@pytest.mark.parametrize("order", [2, 4, 6, 8])
@pytest.mark.parametrize("dim", [2, 3])
def test_error_is_no_larger_than_in_the_reference_order(dim, order, spacing):
    shape = [230, 240] if dim == 2 else [40, 42, 44]
    R, h, dt = order // 2, spacing, 1.1e-3
    rng = np.random.default_rng(order + dim)
    pos = np.meshgrid(*[np.arange(n) for n in shape], indexing="ij")
    wave = lambda a: a * sum(np.sin(rng.uniform(0, 6) + sum(rng.uniform(-.8, .8) * p for p in pos))  # noqa: E731
                             for _ in range(4))
    u, um = wave(1.0), None
    um = u + 0.05 * rng.standard_normal(shape)
    aux = {a: wave(0.02) for a in pipeline.AUX[dim]}
    C = rng.uniform(1500, 3500, shape)
    rhs = 1e-3 * rng.standard_normal(shape)
    npad = shape[0] // 2  # half of the axis is padding on x, none on the others
    prof = [(np.linspace(150.0, 1.0, npad), np.zeros(0))] + [(np.zeros(0), np.zeros(0))] * (dim - 1)
    got_u, got = _gpu_step(dim, order, um.ravel(), {k: v.ravel() for k, v in aux.items()}, u.ravel(), C.ravel(),
                           rhs.ravel(), prof, dt, [h] * dim, shape)
    core = tuple(slice(R, n - R) for n in shape)

    def tap(v, ax, m):
        return v[tuple(slice(R + (m if a == ax else 0), n - R + (m if a == ax else 0)) for a, n in enumerate(shape))]

    names = ["Phix", "Phiz"] if dim == 2 else ["Phix", "Phiy", "Phiz"]
    s = np.zeros(shape)
    s[:npad] = prof[0][0].reshape([-1] + [1] * (dim - 1))
    s, uc, up, Cc, rc, phi = (v[core] for v in (s, u, um, C, rhs, aux["Phix"]))
    # extended precision, exact weights
    F, dux = L(1) * rc, None
    for ax in range(dim):
        d1 = lambda v: sum(L(n) / d * (L(1) * tap(v, ax, m) - tap(v, ax, -m))  # noqa: E731
                           for m, (n, d) in enumerate(W1[order], 1)) / L(h)
        F = F + sum(L(W2[order][abs(m)][0]) / W2[order][abs(m)][1] * tap(u, ax, m) for m in range(-R, R + 1)) / (L(h) * h)
        F = F + d1(aux[names[ax]])
        if ax == 0:
            dux = d1(u)
    a = L(dt) * s
    true_phi = phi - a * phi - a * dux
    true_u = (2 * L(dt) * dt * (L(1) * Cc * Cc * F) + 2 * (2 * L(1) * uc - up) + a * up) / (2 + a)
    # the reference's order in FP64
    def seq(v, ax, w):
        acc = np.zeros(uc.shape)
        for m in range(-R, R + 1):
            if w is W1 and m == 0:
                continue
            n, d = W1[order][abs(m) - 1] if w is W1 else W2[order][abs(m)]
            acc = _fma((np.sign(m) if w is W1 else 1) * (n / d), tap(v, ax, m), acc)
        return acc
    lap = np.zeros(uc.shape)
    for ax in range(dim):
        lap = _fma(seq(u, ax, W2), 1 / (h * h), lap)
    Fr = rc + lap
    for ax in range(dim):
        Fr = _fma(seq(aux[names[ax]], ax, W1), 1 / h, Fr)
    ref_phi = _fma(-(dt * s), seq(u, 0, W1) * (1 / h), _fma(-(dt * s), phi, phi))
    dt2 = dt * dt
    plain = _fma(dt2 * (Cc * Cc), Fr, -(up - 2 * uc))
    pml = 2 * dt2 / (2 + dt * s) * (_fma(Cc * Cc, Fr, -((up - 2 * uc) / dt2)) + s * up / (2 * dt))
    rms = lambda e: float(np.sqrt(np.mean(e.astype(np.float64) ** 2)))  # noqa: E731
    out_u, out_phi = got_u.reshape(shape)[core], got["Phix"].reshape(shape)[core]
    pad = s != 0
    # 3 %: the spread of such a ratio over a few ten thousand cells
    assert rms((out_phi - true_phi)[pad]) <= 1.03 * rms((ref_phi - true_phi)[pad])
    assert rms((out_u - true_u)[~pad]) <= 1.03 * rms((plain - true_u)[~pad])
    assert rms((out_u - true_u)[pad]) <= 1.03 * rms((pml - true_u)[pad])
