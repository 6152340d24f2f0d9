"""The tile passes (environment FWI_CLUSTER=0) at widths whose tile grid starts left of the window: a
grid's first tile then holds the frame alone (width 200, layers 20 wide) or the window's first
columns (width 500).  Gradients with 16-bit images against those with FP32 images: an image is
off by at most 2^-12 (FP16) or 2^-9 (BF16) of its value, and the imaging sums (at most a few times
the gradient in absolute terms) by no more: 2e-3 and 1.6e-2 in the L2 norm."""
import numpy as np
import pytest

from test_native_gpu import exact_problem, wavelet

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz", [(200, 90), (500, 110)])
def test_sixteen_bit_images_at_offset_tile_grids(nx, nz, monkeypatch):
    from fwi_gb300 import Context, MODE_EXACT, SPREC_BF16, SPREC_FP16, SPREC_NATIVE, make_shots
    monkeypatch.setenv("FWI_CLUSTER", "0")
    p = exact_problem(seed=5, nx=nx, nz=nz, nt=200)
    shots = make_shots([dict(sx=k, sz=6, rz=6, rx0=4, rx1=nx - 4, nt=p["nt"], x0=0, nxw=0) for k in (20, nx // 2)])
    obs = np.random.default_rng(3).standard_normal(2 * p["nt"] * (nx - 8)).astype(np.float32)
    g = {}
    for sprec in (SPREC_NATIVE, SPREC_FP16, SPREC_BF16):
        ctx = Context(nx=nx, nz=nz, dh=p["dh"], dt=p["dt"], cpml=20, f_cpml=p["f"], nt_max=p["nt"], max_shots=2,
                      mode=MODE_EXACT, store_prec=sprec)
        ctx.set_wavelet(wavelet(p).astype(np.float32))
        ctx.set_model(*(np.ascontiguousarray(p[k], np.float32) for k in ("vh", "vp", "vn")))
        g[sprec] = [np.asarray(a, np.float64) for a in ctx.gradient(shots, obs)[1:]]
    for sprec, tol in ((SPREC_FP16, 2e-3), (SPREC_BF16, 1.6e-2)):
        for a, b in zip(g[sprec], g[SPREC_NATIVE]):
            assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b)
