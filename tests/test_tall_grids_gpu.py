"""Grids of more than 524280 rows, where tiles of 8 rows pass the 65535 blocks a launch takes along y: an
FP64 shot near the bottom of a uniform model against the same shot on a grid of 64 rows, and the drop-in
second derivative against that of the bottom rows alone.  The points compared see the same values in the
same operations: bit for bit equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

TALL, LOW = 524280 + 41, 64


def test_fp64_shot_at_the_bottom():
    import fwi_gb300
    from fwi_gb300 import Context, make_shots
    nx, cpml, nt = 24, 6, 8
    dt = torch.float64
    got = []
    for nz in (TALL, LOW):
        ctx = Context(nx=nx, nz=nz, dh=10.0, dt=1e-3, cpml=cpml, f_cpml=10.0, nt_max=nt, max_shots=1,
                      precision=fwi_gb300.PREC_FP64)
        ctx.set_wavelet(np.linspace(1.0, 2.0, nt).astype(ctx.dtype))
        ctx.set_model(*(torch.full((nz, nx), v, dtype=dt, device="cuda") for v in (5.2e6, 4e6, 4.4e6)))
        shots = make_shots([dict(sx=11, sz=nz - 20, rz=nz - 20, rx0=4, rx1=nx - 4, nt=nt, x0=0, nxw=0)])
        out = [torch.zeros(nz, nx, dtype=dt, device="cuda") for _ in range(3)]
        traces = torch.zeros(nt * (nx - 8), dtype=dt, device="cuda")
        ctx.forward(shots, out=traces)
        ctx.gradient(shots, torch.zeros_like(traces), None, out=out)
        got.append([traces.cpu()] + [o[-40:].cpu() for o in out])
        del ctx, out
        torch.cuda.empty_cache()
    for tall, low in zip(*got):
        assert bool(low.abs().max() > 0) and torch.equal(tall, low)


def test_drop_in_second_derivative():
    from fwi_gb300 import native
    nx, rows = 19, 96
    g = torch.Generator(device="cuda").manual_seed(2)
    f = [torch.randn(TALL, nx, generator=g, device="cuda") for _ in range(2)]
    out = []
    for nz in (TALL, rows):
        part = [a[-nz:].contiguous() for a in f]
        d = [torch.zeros(nz, nx, device="cuda") for _ in range(2)]
        native.lib().SecondDerivate_P_h(*(native.ptr(a) for a in part + d), 100.0, nx, nz)
        torch.cuda.synchronize()
        out.append([a[-rows + 4:-4].cpu() for a in d])
    for tall, low in zip(*out):
        assert bool(low.abs().max() > 0) and torch.equal(tall, low)
