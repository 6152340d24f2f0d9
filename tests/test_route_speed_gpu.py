"""The built-in routes and group sizes against the other ones on calls that a wrong choice makes an eighth to
two thirds slower (the FP32 shapes where rules drawn from fewer shapes did so): device time of the call, or of
its adjoint where that is what the choice changes, the least of five, within 12 % of the other choice's."""
import numpy as np
import pytest

from test_native_gpu import wavelet

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# name: grid, shots, layer, mode, storage, images, windows of several sizes and lengths, the other choice
CASES = {
    "forward in three launches": (338, 123, 37, 14, "exact", "forward", "fp16", False, {"FWI_CLUSTER": "0"}),
    "forward in fourteen launches": (250, 822, 27, 21, "exact", "forward", "fp16", False, {"FWI_CLUSTER": "0"}),
    "checkpointed in five launches": (310, 336, 17, 15, "exact", "checkpoint", "fp16", False, {"FWI_CLUSTER": "0"}),
    "small shots of several lengths": (226, 238, 11, 12, "exact", "full", "fp32", True, {"FWI_RESIDENT": "0"}),
    "reference adjoint": (552, 139, 6, 21, "ref", "full", "fp32", False,
                          {"FWI_SHOTS_PER_GROUP": "1", "FWI_LAYER_SHOTS_PER_GROUP": "1"}),
    "layer tiles of tall windows": (201, 757, 30, 20, "exact", "boundary", "fp16", False,
                                    {"FWI_SHOTS_PER_GROUP": "3", "FWI_LAYER_SHOTS_PER_GROUP": "8"}),
}


@pytest.mark.parametrize("name", CASES)
def test_not_slower_than_the_other_choice(name, monkeypatch):
    import fwi_gb300 as fw
    nx, nz, n, cpml, mode, call, images, uneven, other = CASES[name]
    nt, rng = 160, np.random.default_rng([3, nx, nz, n])
    shots = []
    for k in range(n):
        w = int(rng.integers(max(2 * cpml + 16, nx // 10), 2 * nx // 5)) if uneven else nx
        x0 = int(rng.integers(0, nx - w + 1))
        t = int(rng.integers(nt // 4, nt + 1)) if uneven and k else nt
        lo, hi = (x0 + cpml, x0 + w - cpml) if mode == "ref" else (x0 + 4, x0 + w - 4)
        shots.append(dict(sx=x0 + w // 2, sz=6, rz=6, rx0=lo, rx1=hi, nt=t, x0=x0, nxw=w if uneven else 0))
    ctx = fw.Context(nx=nx, nz=nz, dh=10.0, dt=1e-3, cpml=cpml, f_cpml=10.0, nt_max=nt, max_shots=n,
                     mode=fw.MODE_REF_COMPAT if mode == "ref" else fw.MODE_EXACT,
                     store={"full": fw.STORE_FULL, "boundary": fw.STORE_BOUNDARY}.get(call, fw.STORE_CHECKPOINT),
                     store_prec=fw.SPREC_FP16 if images == "fp16" else fw.SPREC_NATIVE)
    ctx.set_wavelet(wavelet(dict(nt=nt, f=10.0, dt=1e-3)).astype(np.float32))
    ctx.set_model(*(torch.full((nz, nx), v, device="cuda") for v in (5.2e6, 4e6, 4.4e6)))
    obs = torch.zeros(sum(s["nt"] * (s["rx1"] - s["rx0"]) for s in shots), device="cuda")
    made = fw.make_shots(shots)
    out = [torch.zeros(nz, nx, device="cuda") for _ in range(3)]

    phase = 2 if "FWI_SHOTS_PER_GROUP" in other else 0  # (the adjoint; the call)

    def least():
        t = []
        for k in range(8):  # the first two before their graphs are captured
            if call == "forward":
                ctx.forward(made, out=obs)
            else:
                ctx.gradient(made, obs, None, out=out)
            t.append(float(ctx.last_timing()[phase]) if k > 2 else np.inf)
        return min(t)

    built_in = least()
    for key, value in other.items():
        monkeypatch.setenv(key, value)
    assert built_in <= 1.12 * least()
