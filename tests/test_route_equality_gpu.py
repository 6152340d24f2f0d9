"""Traces do not depend on the path that runs a batch: the shots resident on chip over the whole GPU
(prop_resident.cuh) give, bit for bit, those of the path that would otherwise take the batch, the
per-step tile passes (environment FWI_CLUSTER=0; the layer tiles that advance psi themselves, the
strip pass where the window has no tile origin for that or FWI_INLINE_STRIP=0 asks for it, batches of
several windows) or the cluster path (FWI_RESIDENT=0).  Images follow from the same sums: gradients
differ by the adjoint's rounding only, whatever the image type, 10 x 2^-24 a step as a random walk over
240 steps = 1e-5 (relative L2)."""
import numpy as np
import pytest

from test_native_gpu import exact_problem, wavelet

pytestmark = pytest.mark.gpu

TILES, STRIP, CLUSTER = {"FWI_CLUSTER": "0"}, {"FWI_CLUSTER": "0", "FWI_INLINE_STRIP": "0"}, {"FWI_RESIDENT": "0"}
CASES = [  # nx, nz, cpml, shots, store, images, mode, windows of several sizes, the other path
    (131, 77, 13, 3, "CHECKPOINT", "FP16", "EXACT", False, TILES),
    (209, 200, 20, 8, "FULL", "BF16", "REF_COMPAT", False, TILES),
    (333, 131, 15, 2, "CHECKPOINT", "BF16", "EXACT", False, TILES),
    (73, 33, 5, 2, "CHECKPOINT", "NATIVE", "EXACT", False, TILES),
    (120, 87, 13, 12, "BOUNDARY", "BF16", "EXACT", False, TILES),   # the traces' call only
    (139, 100, 22, 3, "CHECKPOINT", "BF16", "EXACT", False, TILES),  # no tile origin: strip pass
    (300, 100, 24, 2, "CHECKPOINT", "NATIVE", "REF_COMPAT", False, TILES),
    (131, 77, 13, 3, "CHECKPOINT", "FP16", "EXACT", False, STRIP),
    (333, 131, 15, 5, "CHECKPOINT", "BF16", "EXACT", True, TILES),
    (131, 77, 13, 4, "CHECKPOINT", "NATIVE", "REF_COMPAT", True, TILES),
    (160, 120, 12, 2, "FULL", "FP16", "EXACT", False, CLUSTER),
    (209, 209, 20, 3, "FULL", "BF16", "EXACT", False, CLUSTER),
    (131, 140, 23, 4, "FULL", "NATIVE", "EXACT", True, CLUSTER),
    (211, 61, 5, 3, "FULL", "BF16", "EXACT", True, CLUSTER),
]


@pytest.mark.parametrize("nx,nz,cpml,n,store,images,mode,mixed,other", CASES)
def test_traces_equal_on_every_path(nx, nz, cpml, n, store, images, mode, mixed, other, monkeypatch):
    import fwi_gb300 as f
    nt = 240
    p = exact_problem(seed=nx, nx=nx, nz=nz, nt=nt)
    shots = []
    for k in range(n):
        w = nx if not mixed or k == 0 else max(2 * cpml + 9, nx - 13 * k % (nx // 2))
        x0 = nx - w
        shots.append(dict(sx=x0 + 4 + (w - 9) * (k + 1) // (n + 1), sz=6, rz=nz - cpml - 6 if k % 2 else 6, rx0=x0 + 4,
                          rx1=x0 + w - 4, nt=nt - (17 * k % 90 if mixed else 0), x0=x0, nxw=w if mixed else 0))
    obs = np.random.default_rng(1).standard_normal(sum(s["nt"] * (s["rx1"] - s["rx0"]) for s in shots)).astype(np.float32)
    out = []
    for env in ({}, other):
        for name in ("FWI_CLUSTER", "FWI_RESIDENT", "FWI_INLINE_STRIP"):
            monkeypatch.delenv(name, raising=False)
        for name, value in env.items():
            monkeypatch.setenv(name, value)
        if other is STRIP:  # (the choice the path would make holds for both)
            monkeypatch.setenv("FWI_INLINE_STRIP", "0")
        ctx = f.Context(nx=nx, nz=nz, dh=p["dh"], dt=p["dt"], cpml=cpml, f_cpml=p["f"], nt_max=nt, max_shots=n,
                        max_window=nx, mode=getattr(f, "MODE_" + mode), store=getattr(f, "STORE_" + store),
                        store_prec=getattr(f, "SPREC_" + images))
        ctx.set_wavelet(wavelet(p).astype(np.float32))
        ctx.set_model(*(np.ascontiguousarray(p[k], np.float32) for k in ("vh", "vp", "vn")))
        sh = f.make_shots(shots)
        out.append((ctx.forward(sh), ctx.gradient(sh, obs)))
    (ta, ga), (tb, gb) = out
    assert np.abs(tb).max() > 0
    assert np.array_equal(ta, tb)
    assert ga[0] == gb[0]  # the misfit of the same traces
    for a, b in zip(ga[1:], gb[1:]):
        a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
        assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b)
