"""Shots resident on chip over the whole GPU (prop_resident.cuh) against the per-step passes
(environment FWI_CLUSTER=0), at the sizes where the row bands, column pairs and side layers are at
their limits: odd and narrow windows, layers of 4 and 5 points, few rows, windows of several widths
and lengths in one batch, several launches a batch, every image type, checkpoints and the
reference mode.  The forward rounds as the passes do, the adjoint in another order.
Tolerances (relative L2), 2^-24 a step adding up over nt steps as a random walk, ten of it a step:
10 x 2^-24 x sqrt(240) = 1e-5 for records and FP32-image gradients; with 16-bit images a last-bit
difference may move an image by 2^-9 where it lies at a rounding boundary, a chance of 2^-7 at such a
difference: 10 times as much."""
import numpy as np
import pytest

from test_native_gpu import exact_problem, wavelet

pytestmark = pytest.mark.gpu

CASES = [  # nx, nz, cpml, shots, store, images, mode, windows of several sizes
    (131, 77, 13, 3, "CHECKPOINT", "FP16", "EXACT", False),
    (333, 131, 15, 5, "FULL", "BF16", "EXACT", True),
    (51, 60, 20, 2, "CHECKPOINT", "NATIVE", "EXACT", False),
    (397, 90, 4, 2, "FULL", "NATIVE", "EXACT", False),
    (640, 60, 20, 1, "FULL", "FP16", "EXACT", False),
    (501, 47, 12, 2, "FULL", "NATIVE", "EXACT", False),
    (73, 33, 5, 2, "CHECKPOINT", "BF16", "EXACT", False),
    (72, 56, 12, 34, "CHECKPOINT", "FP16", "EXACT", True),
    (209, 200, 20, 24, "FULL", "FP16", "EXACT", False),
    (149, 90, 12, 2, "FULL", "NATIVE", "REF_COMPAT", False),
    (131, 77, 13, 4, "CHECKPOINT", "FP16", "REF_COMPAT", True),
    (501, 60, 20, 1, "FULL", "BF16", "REF_COMPAT", False),
    (53, 50, 5, 2, "CHECKPOINT", "NATIVE", "REF_COMPAT", False),
]


def rel(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


@pytest.mark.parametrize("nx,nz,cpml,n,store,images,mode,mixed", CASES)
def test_resident_path_matches_tile_passes(nx, nz, cpml, n, store, images, mode, mixed, monkeypatch):
    import fwi_gb300 as f
    nt = 240
    p = exact_problem(seed=nx, nx=nx, nz=nz, nt=nt)
    shots = []
    for k in range(n):
        w = nx if not mixed or k == 0 else max(2 * cpml + 9, nx - 13 * k % (nx // 2))
        shots.append(dict(sx=4 + (w - 9) * (k + 1) // (n + 1), sz=6, rz=5 + k % 3, rx0=max(4, cpml), rx1=w - max(4, cpml),
                          nt=nt - (17 * k % 90 if mixed else 0), x0=nx - w, nxw=w if mixed else 0))
        shots[-1]["sx"] += shots[-1]["x0"]
        shots[-1]["rx0"] += shots[-1]["x0"]
        shots[-1]["rx1"] += shots[-1]["x0"]
    obs = np.random.default_rng(1).standard_normal(sum(s["nt"] * (s["rx1"] - s["rx0"]) for s in shots)).astype(np.float32)
    out = {}
    for flag in ("1", "0"):
        monkeypatch.setenv("FWI_CLUSTER", flag)
        ctx = f.Context(nx=nx, nz=nz, dh=p["dh"], dt=p["dt"], cpml=cpml, f_cpml=p["f"], nt_max=nt, max_shots=n,
                        max_window=nx, mode=getattr(f, "MODE_" + mode), store=getattr(f, "STORE_" + store),
                        store_prec=getattr(f, "SPREC_" + images))
        ctx.set_wavelet(wavelet(p).astype(np.float32))
        ctx.set_model(*(np.ascontiguousarray(p[k], np.float32) for k in ("vh", "vp", "vn")))
        sh = f.make_shots(shots)
        first = ctx.gradient(sh, obs)
        again = ctx.gradient(sh, obs)
        assert first[0] == again[0] and all(np.array_equal(a, b) for a, b in zip(first[1:], again[1:]))
        launches = ctx.last_launches()
        out[flag] = (first, ctx.forward(sh), launches)
    (ga, ta, la), (gb, tb, lb) = out["1"], out["0"]
    assert la < lb
    tol = 1e-5 if images == "NATIVE" else 1e-4
    assert rel(ta, tb) <= 1e-5 and abs(ga[0] - gb[0]) <= 1e-5 * abs(gb[0])
    for a, b in zip(ga[1:], gb[1:]):
        assert rel(a, b) <= tol
