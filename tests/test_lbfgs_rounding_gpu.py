"""A pass of the L-BFGS recursion rounds x + k u once to FP64 and once to FP32, with coefficient and sums in
FP64: bit for bit against exact fractions, where the sum cancels to its last bits (q = g - alpha y with
g = alpha y rounded to FP32) and at the ends of FP32's range.  The data are such that every dot product
but the last pass's is exact in FP64 in any order: y and s small whole numbers, g of 24 bits.  The old model's
pair is s, the new model zero, so that the updated model is the direction itself; where s is zero the
direction is gamma q."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [41, 64])
@pytest.mark.parametrize("exponent", [0, -115, 100])
def test_axpy_rounds_as_fp64(nx, exponent):
    import fwi_gb300 as f
    nz, rng = 40, np.random.default_rng([nx, exponent + 200])
    y = rng.integers(1, 2048, (3, nz, nx)).astype(np.float64) * rng.choice([-1.0, 1.0], (3, nz, nx))
    s = np.where(rng.random((3, nz, nx)) < 0.5, 0.0, np.rint(0.25 * y) + rng.integers(1, 3, (3, nz, nx)))
    g1 = (np.rint(0.62890625 * y * 4096.0 + rng.integers(-1, 2, (3, nz, nx))) / 4096.0)  # 24 bits, about 0.63 y
    g0 = g1 - y
    unit = 2.0 ** exponent
    ctx = f.Context(nx=nx, nz=nz, dh=10.0, dt=1e-3, cpml=8, f_cpml=20.0, nt_max=4, max_shots=1)
    f32 = lambda a: [np.ascontiguousarray(v, np.float32) for v in a]  # noqa: E731
    for a in (g0, g1, y):
        assert np.array_equal(np.float32(a * unit).astype(np.float64), a * unit)
    # the pair's old model is the one that the first step started from
    ctx.set_model(*f32(-s))
    ctx.set_gradient(*f32(g0 * unit))
    ctx.first_step(0.0, 0.0, 0.0)
    ctx.set_model(*f32(0.0 * s))
    ctx.set_gradient(*f32(g1 * unit))
    ctx.lbfgs_direction(1)
    ctx.lbfgs_update(1.0, 1.0, 1.0, False, False)
    got = -np.asarray(ctx.get_model()[1]).astype(np.float64)  # v_po: no other bound acts on it
    y, s, g = y[1], s[1], g1[1]
    ys, yy, sg = float((y * s).sum()) * unit, float((y * y).sum()) * unit ** 2, float((s * g).sum()) * unit
    rho = 1.0 / ys
    alpha, gamma = rho * sg, ys / yy
    r = np.zeros((nz, nx), np.float32)
    for i in np.ndindex(nz, nx):
        q = np.float32(float(Fraction(g[i]) * Fraction(unit) - Fraction(alpha) * Fraction(y[i]) * Fraction(unit)))
        r[i] = np.float32(float(Fraction(gamma) * Fraction(float(q))))
    rows, free = slice(16, None), (s == 0)[16:]
    assert np.abs(r[rows][free]).max() > 0
    assert np.array_equal(got[rows][free], r[rows].astype(np.float64)[free])
    # where s is not zero: + (alpha - beta) s, beta from a sum whose order is free, 2^-50 of the value
    beta = rho * float((y * unit * r.astype(np.float64)).sum())
    want = r.astype(np.float64) + (alpha - beta) * s
    assert np.all(np.abs(got - want)[rows] <= 2.0 ** -23 * np.abs(want)[rows])
