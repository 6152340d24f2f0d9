"""The L-BFGS recursion over several pairs, its ring of slots wrapping, on grids whose rows are padded,
against the two-loop recursion in NumPy (FP64) on the same models and gradients.  A model value of
4e6 is rounded to 0.25 (FP32) and moves by about 1e4, so that an update is off by 1e-5 of itself a
rounding; ten roundings a value: 1e-4.  FP64: 1e-10."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def two_loop(g, pairs):
    q, al = g.copy(), []
    for s, y in reversed(pairs):
        a = (s * q).sum() / (y * s).sum()
        al.append(a)
        q -= a * y
    s, y = pairs[-1]
    r = q * (s * y).sum() / (y * y).sum()
    for (s, y), a in zip(pairs, reversed(al)):
        r += s * (a - (y * r).sum() / (y * s).sum())
    return r


@pytest.mark.parametrize("prec", ["FP32", "FP64"])
@pytest.mark.parametrize("nx,nz,m", [(33, 40, 3), (64, 29, 1), (101, 33, 5)])
def test_directions_match_two_loop(prec, nx, nz, m):
    import fwi_gb300 as f
    dtype = np.float64 if prec == "FP64" else np.float32
    rng = np.random.default_rng(nx)
    ctx = f.Context(nx=nx, nz=nz, dh=10.0, dt=1e-3, cpml=8, f_cpml=20.0, nt_max=4, max_shots=1,
                    precision=getattr(f, "PREC_" + prec))
    model = [np.full((nz, nx), v, dtype) for v in (4e6, 3e6, 2.5e6)]  # v_hor, v_po, v_nmo
    ctx.set_model(*model)
    g0 = [rng.standard_normal((nz, nx)) for _ in range(3)]
    pairs = [[], [], []]
    for k in range(6):
        g = [(a * 0.6 ** k + 0.01 * 0.6 ** k * rng.standard_normal((nz, nx))).astype(dtype) for a in g0]
        ctx.set_gradient(*g)
        if k == 0:
            ctx.first_step(2e5, 2e5, 2e5)
        else:
            for p in range(3):
                pairs[p].append((model[p].astype(np.float64) - back[p], g[p].astype(np.float64) - gback[p]))
                pairs[p] = pairs[p][-m:]
            ctx.lbfgs_direction(m)
            ctx.lbfgs_update(1.0, 1.0, 1.0, False, False)
        back, gback = [a.astype(np.float64) for a in model], [a.astype(np.float64) for a in g]
        model = [np.asarray(a).copy() for a in ctx.get_model()]
        if k:
            for p in range(3):
                r = two_loop(gback[p], pairs[p])[16:]
                step = back[p][16:] - model[p].astype(np.float64)[16:]
                assert np.linalg.norm(step - r) <= (1e-10 if prec == "FP64" else 1e-4) * np.linalg.norm(r)
                assert np.array_equal(model[p][:16], back[p].astype(dtype)[:16])
