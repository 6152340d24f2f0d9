"""The cluster kernels themselves (prop_cluster.cuh) at the sizes of test_cluster_gpu.py: windows past 12000
points take the resident path unless FWI_RESIDENT=0 says otherwise, so that these cases set it.  Two
shots of different windows and lengths, 16-bit images, 16 CTAs of unequal rows, wide layers, against the
FP64 oracle and the tile passes, with that file's tolerances.  And, as the library dispatches them
itself, windows of up to 12000 points with every image type."""
import numpy as np
import pytest

import test_cluster_gpu as sizes
from test_cluster_gpu import c1_case, case  # noqa: F401 (fixtures)
from test_native_gpu import exact_problem, oracle_exact

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def clusters_only(request, monkeypatch):
    if "dispatched" not in request.node.name:
        monkeypatch.setenv("FWI_RESIDENT", "0")


def test_oracle_and_tile_passes(case, monkeypatch):  # noqa: F811
    sizes.test_cluster_path_matches_fp64_oracle_and_tile_passes(case, monkeypatch)


@pytest.mark.parametrize("sprec,tol", [(1, 2e-3), (2, 2e-2)])
def test_reduced_precision_images(case, sprec, tol, monkeypatch):  # noqa: F811
    sizes.test_cluster_path_reduced_precision_images(case, sprec, tol, monkeypatch)


@pytest.mark.parametrize("sprec,tol_tile", [(0, 1e-5), (1, 2e-3), (2, 2e-2)])
def test_unequal_rows(c1_case, sprec, tol_tile, monkeypatch):  # noqa: F811
    sizes.test_cluster_path_c1_grid_unequal_rows(c1_case, sprec, tol_tile, monkeypatch)


def test_wide_layers(monkeypatch):
    sizes.test_cluster_path_edge_shapes(dict(nx=96, nz=200, cpml=30, nt=80), monkeypatch)


@pytest.mark.parametrize("nx,nz", [(110, 100), (72, 56), (120, 100)])
@pytest.mark.parametrize("sprec,tol", [(0, 1e-5), (1, 2e-3), (2, 2e-2)])
def test_dispatched_windows(nx, nz, sprec, tol, monkeypatch):
    p = exact_problem(seed=9, nx=nx, nz=nz, nt=200)
    shots = [dict(sx=nx // 3, sz=6, rz=6, rx0=4, rx1=nx - 4, nt=200, x0=0, nxw=0),
             dict(sx=nx // 2, sz=nz - 10, rz=5, rx0=14, rx1=nx - 16, nt=150, x0=7, nxw=nx - 17)]
    obs = 1e-3 * np.random.default_rng(2).standard_normal(sum(s["nt"] * (s["rx1"] - s["rx0"]) for s in shots))
    mask = np.ones(sum(s["rx1"] - s["rx0"] for s in shots), np.uint8)
    (Jc, *gc), lc, _ = sizes.run(p, shots, obs, mask, sprec=sprec)
    (Jt, *gt), lt, _ = sizes.run(p, shots, obs, mask, sprec=sprec, cluster=False, monkeypatch=monkeypatch)
    J, g = oracle_exact(p, shots, obs, mask)
    assert lc < 10 < lt
    assert abs(Jc - J) <= 1e-5 * J and abs(Jc - Jt) <= 1e-6 * Jt
    for a, b, c in zip(gc, gt, g):
        assert sizes.rel(a, b) <= tol and sizes.rel(a, c) <= (1e-4 if sprec == 0 else tol)
