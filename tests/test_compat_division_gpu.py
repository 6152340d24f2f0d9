"""The drop-in stencils' division by dh^2 at the divisors and values where its rounding could go wrong,
bit for bit against NumPy's FP64 division, at grids that end inside a tile, at its edge and past it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dh2", [100.0, 0.3, 1.9999999, 7.0, 3e-3, 1e30, 1.1e-31, 1e-38, -25.0, float("inf")])
@pytest.mark.parametrize("nx,nz", [(33, 17), (48, 40), (17, 25)])
def test_second_derivative_divides_as_ieee(dh2, nx, nz):
    from fwi_gb300 import native
    rng = np.random.default_rng(int(nx + nz))
    f = [(rng.standard_normal((nz, nx)) * 10.0 ** rng.uniform(-44, 30, (nz, nx))).astype(np.float32) for _ in range(2)]
    for a in f:
        a[rng.random((nz, nx)) < 0.3] = 0.0
        a[rng.random((nz, nx)) < 0.05] = -0.0
        a[nz - 6, nx - 6] = np.inf
    t = [torch.from_numpy(a).cuda() for a in f]
    out = [torch.zeros(nz, nx, device="cuda") for _ in range(2)]
    d32 = np.float32(dh2)
    native.lib().SecondDerivate_P_h(t[0].data_ptr(), t[1].data_ptr(), out[0].data_ptr(), out[1].data_ptr(), float(d32), nx, nz)
    torch.cuda.synchronize()
    with np.errstate(all="ignore"):
        for a, got, axis in ((f[0], out[0], 1), (f[1], out[1], 0)):
            at = lambda k: np.roll(a, -k, axis)  # noqa: E731
            pair = lambda k: (at(k) + at(-k)).astype(np.float64)  # noqa: E731
            s = -(205 / 72.) * a.astype(np.float64) + (8 / 5.) * pair(1) - (1 / 5.) * pair(2) + (8 / 315.) * pair(3)
            want = ((s - (1 / 560.) * pair(4)) / np.float64(d32)).astype(np.float32)[4:nz - 4, 4:nx - 4]
            got = got.cpu().numpy()[4:nz - 4, 4:nx - 4]
            nan = np.isnan(want)
            assert np.array_equal(np.isnan(got), nan)
            assert np.array_equal(got[~nan].view(np.int32), want[~nan].view(np.int32))
