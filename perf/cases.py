"""What the library is timed on: the calls an inversion makes, over the sizes it makes them at.

Grids, steps, frequencies and storage modes are those of the benchmark's
configurations (fwi_gb300/synth.py: C1 .. C5), of the tests' small problems,
and of the reference's single-shot driver loop.  Models are seeded smooth
layered VTI models; observed records are hyperbolic events of a Ricker
wavelet (a direct arrival and reflections), so that the inputs depend on the
seed alone and not on any propagator.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import fwi_gb300
from fwi_gb300 import native

DEV = "cuda"
DH, DT, VMAX, R_COEF = 10.0, 1e-3, 6000.0, 1e-6
FLOPS_FWD, FLOPS_ADJ = 50, 62  # per point update: two 8th-order stencils and the update; with imaging
STORES = {"full": fwi_gb300.STORE_FULL, "checkpoint": fwi_gb300.STORE_CHECKPOINT,
          "boundary": fwi_gb300.STORE_BOUNDARY}
IMAGES = {"fp32": fwi_gb300.SPREC_NATIVE, "fp16": fwi_gb300.SPREC_FP16, "bf16": fwi_gb300.SPREC_BF16}


def _case(name, call, nx, nz, nt, shots, **kw):
    c = dict(name=name, call=call, nx=nx, nz=nz, nt=nt, shots=shots, cpml=20, freq=10.0, mode="exact",
             precision="fp32", store="full", images="fp32", uneven=False, dropout=False)
    c.update(kw)
    return c


def listed():
    return [
        # a test-sized problem (one shot on a 72 x 56 grid): latency and launches, the smallest call
        _case("small shot gradient", "gradient", 72, 56, 260, 1, cpml=12, freq=20.0),
        # C1, the reference's plain single-shot gradient, default storage (every image in FP32)
        _case("C1 shot gradient", "gradient", 209, 209, 2000, 1),
        # C1-sized shots side by side, 16-bit images: a small survey on one GPU
        _case("C1 x 8 shots gradient", "gradient", 209, 209, 2000, 8, images="fp16"),
        # C2, the headline configuration: 32 shots, checkpointed, FP16 images
        _case("C2 x 32 shots gradient", "gradient", 609, 309, 3000, 32, freq=8.0, store="checkpoint",
              images="fp16"),
        # one C2 shot at a time (max_shots 1), FP32 images: how the reference's rank works
        _case("C2 shot gradient", "gradient", 609, 309, 3000, 1, freq=8.0),
        # forward modelling of C2 shots: observed data, and a line-search trial's cost
        _case("C2 x 16 shots forward", "forward", 609, 309, 3000, 16, freq=8.0, store="checkpoint"),
        # C3's large grid, checkpointed (a few hundred of its steps)
        _case("C3 x 4 shots gradient", "gradient", 2009, 809, 400, 4, store="checkpoint", images="fp16"),
        # C4: apertures and record lengths of every size, boundary storage, dropped traces
        _case("C4 x 8 windows gradient", "gradient", 4009, 1209, 900, 8, freq=12.0, store="boundary",
              images="fp16", uneven=True, dropout=True),
        # the reference's own gradient (its CPML adjoint), one C1 shot
        _case("C1 reference-mode gradient", "gradient", 209, 209, 2000, 1, mode="ref"),
        # FP64 contexts: the accuracy check of an FP32 run
        _case("FP64 shot gradient", "gradient", 209, 209, 400, 1, precision="fp64"),
        # the drop-in entry points in the reference's per-step sequence, one C1 shot
        _case("drop-in shot loop", "compat", 209, 209, 300, 1),
        # the optimizer between gradients: first step, then L-BFGS directions and updates (C3's grid)
        _case("L-BFGS updates", "optimizer", 2009, 809, 6, 1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["gradient"] * 7 + ["forward", "optimizer", "compat"])
    cpml = rng.randint(10, 24)
    nx, nz = max(_log_int(rng, 72, 1400), 2 * cpml + 24), max(_log_int(rng, 56, 900), cpml + 24)
    c = _case("", call, nx, nz, 0, 1, cpml=cpml, freq=round(rng.uniform(5.0, 14.0), 2))
    del c["name"]
    if call == "optimizer":
        c["nt"] = rng.randint(3, 8)
        return c
    if call == "compat":
        c["nx"], c["nz"], c["nt"] = min(nx, 700), min(nz, 400), rng.randint(60, 240)
        return c
    c["shots"] = _log_int(rng, 1, 40)
    # at most about a third of the largest listed case's point updates
    c["nt"] = max(120, min(_log_int(rng, 260, 3000), int(6e9 / (nx * nz * c["shots"]))))
    c["store"] = rng.choice(["full", "checkpoint", "checkpoint", "boundary"])
    c["images"] = rng.choice(["fp32", "fp16", "fp16", "bf16"])
    if call == "gradient":
        c["mode"] = rng.choice(["exact"] * 5 + ["ref"])
        c["uneven"] = c["shots"] > 1 and nx > 2 * cpml + 60 and rng.random() < 0.3
        c["dropout"] = rng.random() < 0.3
    if c["store"] == "full" and nx * nz * c["nt"] * c["shots"] > 3e9:
        c["store"] = "checkpoint"
    return c


# ------------------------------------------------------------------ inputs

def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _host_rng(case, seed):
    return np.random.default_rng([int(seed), case["nx"], case["nz"], case["shots"]])


def _smooth(a, n):
    k = torch.ones(1, 1, 1, 2 * n + 1, dtype=a.dtype, device=a.device) / (2 * n + 1)
    a = a[None, None]
    for _ in range(2):
        a = torch.nn.functional.conv2d(torch.nn.functional.pad(a, (n, n, 0, 0), mode="replicate"), k)
        a = torch.nn.functional.conv2d(torch.nn.functional.pad(a, (0, 0, n, n), mode="replicate"),
                                       k.transpose(2, 3))
    return a[0, 0]


def _model(case, seed):
    """Squared velocities (v_hor, v_po, v_nmo), FP32 [nz][nx]: speed growing with depth in smoothed
    layers with anomalies, 1500 to 3700 m/s; epsilon up to 0.2, delta below epsilon."""
    g = _generator(seed)
    nx, nz = case["nx"], case["nz"]
    layers = torch.rand(12, generator=g, device=DEV).cumsum(0)
    layers = 1500.0 + 1900.0 * layers / layers[-1]
    z = torch.arange(nz, device=DEV)[:, None] + 0.04 * torch.arange(nx, device=DEV)[None, :]
    vel = layers[(12 * z / (z.max() + 1)).long()]
    vel = vel + 120.0 * torch.randn(nz, nx, generator=g, device=DEV)
    vel = _smooth(vel, 4).clamp(1500.0, 3700.0)
    eps = 0.1 + 0.1 * _smooth(torch.rand(nz, nx, generator=g, device=DEV) * 2 - 1, 3)
    dl = 0.5 * eps
    vp = vel * vel
    return [(vp * (1 + 2 * eps)).contiguous(), vp.contiguous(), (vp * (1 + 2 * dl)).contiguous()]


def _shots(case, seed):
    """Surface shots evenly spread over the model with a receiver at every interior column of
    their window (the reference mode: between the layers, as the reference places them); `uneven`:
    windows of a tenth to two fifths of the model and steps of a quarter to all, drawn from the seed."""
    rng = _host_rng(case, seed)
    nx, nz, nt, n, cp = (case[k] for k in ("nx", "nz", "nt", "shots", "cpml"))
    sz = 4 if case["mode"] == "ref" else 6
    out = []
    for k in range(n):
        x0, w, t = 0, nx, nt
        if case["uneven"]:
            w = int(rng.integers(max(2 * cp + 16, nx // 10), max(2 * cp + 17, 2 * nx // 5)))
            w = min(w, nx)
            x0 = int(rng.integers(0, nx - w + 1))
            t = nt if k == 0 else int(rng.integers(max(1, nt // 4), nt + 1))
            sx = x0 + w // 2
        else:
            sx = 4 + int((nx - 9) * (k + 0.5) / n)
        lo, hi = (x0 + cp, x0 + w - cp) if case["mode"] == "ref" else (x0 + 4, x0 + w - 4)
        out.append(dict(sx=sx, sz=sz, rz=sz, rx0=lo, rx1=hi, nt=t, x0=x0, nxw=w if case["uneven"] else 0))
    return out


def _ricker(case):
    """The reference's Ricker wavelet, its time accumulated in FP32 (src/main.c:328-332)."""
    f, dt, t = np.float32(case["freq"]), np.float32(DT), np.float32(0)
    w = np.zeros(max(case["nt"], 1))
    for k in range(case["nt"]):
        t = np.float32(t + dt)
        a = math.pi * float(f) * float(np.float32(t - np.float32(1) / f))
        w[k] = (1 - 2 * a * a) * math.exp(-a * a)
    return w


def _records(case, seed, shots, dtype):
    """Observed records [nt][nrec] of every shot, concatenated: a direct arrival and three
    reflections, Ricker pulses along hyperbolas with 1/sqrt(distance) amplitudes."""
    rng = _host_rng(case, seed + 7)
    parts = []
    for s in shots:
        x = (torch.arange(s["rx0"], s["rx1"], device=DEV, dtype=torch.float32) - s["sx"]) * DH
        t = torch.arange(s["nt"], device=DEV, dtype=torch.float32)[:, None] * DT
        rec = torch.zeros(s["nt"], x.numel(), device=DEV)
        for e in range(4):
            v = 1600.0 + 350.0 * e + 100.0 * rng.random()
            t0 = 0.0 if e == 0 else (0.25 * e + 0.15 * rng.random()) * max(s["nt"] * DT, 0.4)
            path = torch.sqrt((t0 * v) ** 2 + x * x)
            a = (math.pi * case["freq"] * (t - 1.2 / case["freq"] - path / v)) ** 2
            amp = (8.0 if e == 0 else 4.0 * (0.5 - rng.random())) / torch.sqrt(1.0 + path / 50.0)
            rec += amp * (1 - 2 * a) * torch.exp(-a)
        parts.append(rec.reshape(-1))
    return torch.cat(parts).to(dtype)


def _mask(case, seed, shots):
    if not case["dropout"]:
        return None
    rng = _host_rng(case, seed + 3)
    return (rng.random(sum(s["rx1"] - s["rx0"] for s in shots)) >= 0.1).astype(np.uint8)


# ------------------------------------------------------------------ prepare and run

def prepare(case, seed):
    if case["call"] == "compat":
        return _prepare_compat(case, seed)
    fp64 = case["precision"] == "fp64"
    dtype = torch.float64 if fp64 else torch.float32
    shots = _shots(case, seed)
    ctx = fwi_gb300.Context(
        nx=case["nx"], nz=case["nz"], dh=DH, dt=DT, cpml=case["cpml"], f_cpml=case["freq"], vmax=VMAX, r_coef=R_COEF,
        nt_max=case["nt"], max_shots=case["shots"], max_window=max(s["nxw"] or case["nx"] for s in shots),
        max_receivers=max(s["rx1"] - s["rx0"] for s in shots),
        mode=fwi_gb300.MODE_REF_COMPAT if case["mode"] == "ref" else fwi_gb300.MODE_EXACT,
        precision=fwi_gb300.PREC_FP64 if fp64 else fwi_gb300.PREC_FP32,
        store=STORES[case["store"]], store_prec=IMAGES[case["images"]])
    ctx.set_wavelet(_ricker(case).astype(ctx.dtype))
    model = [m.to(dtype) for m in _model(case, seed)]
    state = dict(case=case, ctx=ctx, out=[torch.zeros(case["nz"], case["nx"], dtype=dtype, device=DEV)
                                          for _ in range(3)])
    state["shots"] = fwi_gb300.make_shots(shots)
    if case["call"] == "optimizer":
        state.update(model=model, gradients=_gradients(case, seed, model))
        torch.cuda.synchronize()
        ctx.set_model(*model)  # an inversion has computed a gradient before its first update: a few steps here
        ctx.gradient(state["shots"], torch.zeros(sum(s["nt"] * (s["rx1"] - s["rx0"]) for s in shots), device=DEV))
        return state
    if case["call"] == "gradient":
        state.update(obs=_records(case, seed, shots, dtype), mask=_mask(case, seed, shots))
    else:
        state["traces"] = torch.zeros(sum(s["nt"] * (s["rx1"] - s["rx0"]) for s in shots), dtype=dtype, device=DEV)
    torch.cuda.synchronize()
    ctx.set_model(*model)
    return state


def run(state):
    case = state["case"]
    if case["call"] == "compat":
        return _run_compat(state)
    ctx = state["ctx"]
    if case["call"] == "gradient":
        j, gh, gp, gn = ctx.gradient(state["shots"], state["obs"], state["mask"], out=state["out"])
        return {"misfit": j, "v_hor": gh, "v_po": gp, "v_nmo": gn}
    if case["call"] == "forward":
        return {"traces": ctx.forward(state["shots"], out=state["traces"])}
    # optimizer: a steepest first step, then L-BFGS directions, each followed by an update
    g = state["gradients"]
    ctx.set_model(*state["model"])
    ctx.set_gradient(*g[0])
    ctx.first_step(3e5, 2e5, 2.5e5)
    for k in range(1, case["nt"]):
        ctx.set_gradient(*g[k])
        ctx.lbfgs_direction(5)
        ctx.lbfgs_update(1.0, 1.0, 1.0)
    if native.lib().fwi_get_model(ctx.handle, *[native.ptr(o) for o in state["out"]]) != 0:
        raise RuntimeError("fwi_get_model failed")
    return {"v_hor": state["out"][0], "v_po": state["out"][1], "v_nmo": state["out"][2]}


def _gradients(case, seed, model):
    """Gradients of successive iterations, each half of the last one but for a little noise: every
    pair has positive curvature, and the steps stay about as long as the first."""
    g = _generator(seed + 1)
    d = [_smooth(torch.randn(case["nz"], case["nx"], generator=g, device=DEV), 3) for _ in range(3)]
    return [[(x * 0.5 ** k + 1e-3 * 0.5 ** k * torch.randn(case["nz"], case["nx"], generator=g, device=DEV)).contiguous()
             for x in d] for k in range(case["nt"])]


# The drop-in entry points: one shot as the reference's main.c sequences it (src/main.c:408-495),
# its buffers (F = P + nx nz in one allocation, the adjoint's CPML arrays aliasing the forward's).

def _prepare_compat(case, seed):
    nx, nz, nt, cp = (case[k] for k in ("nx", "nz", "nt", "cpml"))
    n = nx * nz
    f32 = np.float32
    L = cp * DH
    d0 = float(f32(-3 * math.log(R_COEF) / (2 * L)))
    lib = native.lib()
    z = lambda k: torch.zeros(k, dtype=torch.float32, device=DEV)  # noqa: E731
    ax, bx, az, bz = z(nx), z(nx), z(nz), z(nz)
    lib.CPML_x_h(native.ptr(ax), native.ptr(bx), cp, VMAX, nx, DT, DH, case["freq"], d0, L)
    lib.CPML_z_h(native.ptr(az), native.ptr(bz), cp, VMAX, nz, DT, DH, case["freq"], d0, L)
    shot = dict(sx=nx // 2, rx0=0, rx1=nx, nt=nt)
    st = dict(case=case, lib=lib, n=n, coef=(ax, bx, az, bz), model=_model(case, seed),
              source=torch.from_numpy(_ricker(case).astype(f32)).to(DEV),
              obs=_records(case, seed, [shot], torch.float32), snap=torch.zeros(nt * 2 * n).pin_memory(),
              dh2=float(f32(DH) * f32(DH)), C=float(f32(DT) * f32(DT) / (f32(DH) * f32(DH))),
              lvl=[z(2 * n), z(2 * n)], pre2=z(2 * n), PF=z(n), p2=z(n), r2=z(n), cpml=[z(n) for _ in range(6)],
              adj=[z(n) for _ in range(6)], aux=[z(n) for _ in range(4)], d2=[z(n) for _ in range(4)],
              syn=z(nt * nx), res=z(nt * nx), grad=[z(n) for _ in range(3)])
    torch.cuda.synchronize()
    return st


def _run_compat(s):
    case, lib, n = s["case"], s["lib"], s["n"]
    nx, nz, nt, cp = (case[k] for k in ("nx", "nz", "nt", "cpml"))
    P = native.ptr
    sx, sz = nx // 2 + 1, 5
    for t in s["lvl"] + s["cpml"] + s["adj"] + s["grad"] + [s["PF"], s["syn"]]:
        t.zero_()
    coef, mod = [P(t) for t in s["coef"]], [P(t) for t in s["model"]]
    psx, psz, zx, zz, ap, af = (P(t) for t in s["cpml"])
    pre, past = P(s["lvl"][0]), P(s["lvl"][1])
    snap, fo = s["snap"].data_ptr(), 4 * n
    for it in range(nt):
        lib.launchPropagation(None, None, snap + 2 * it * fo, P(s["PF"]), past, pre, past + fo, pre + fo, P(s["p2"]),
                              P(s["r2"]), s["dh2"], nx, nz, *coef, psx, psz, DH, cp, zx, zz, ap, af, *mod,
                              P(s["source"]), P(s["syn"]), s["C"], sx, sz, it)
        pre, past = past, pre
    lib.res_h(P(s["res"]), P(s["obs"]), P(s["syn"]), nx, nt)
    for t in s["lvl"] + s["cpml"]:
        t.zero_()
    a1, a2, a3, a4, a5, a6 = (P(t) for t in s["adj"])
    pre, past = P(s["lvl"][0]), P(s["lvl"][1])
    pre2 = P(s["pre2"])
    for it in range(nt):
        lib.launchBackPropagation(None, None, nx, nz, nt, snap + 2 * (nt - it - 1) * fo, pre, past, pre + fo, past + fo,
                                  *[P(t) for t in s["aux"]], *mod, *[P(t) for t in s["d2"]], s["dh2"], pre2, pre2 + fo,
                                  *coef, a1, a2, psx, psz, DH, cp, zx, zz, af, ap, a3, a4, a5, a6, P(s["res"]), s["C"],
                                  P(s["PF"]), it, sx, sz, DT, *[P(t) for t in s["grad"]])
        pre, past = past, pre
    return {"traces": s["syn"], "residual": s["res"], "v_hor": s["grad"][0], "v_po": s["grad"][1], "v_nmo": s["grad"][2]}


# ------------------------------------------------------------------ the least work, and the values in 64 bits

def _updates(case):
    """Point updates of one phase, from the shots of seed 0."""
    return sum(((s["nxw"] or case["nx"]) - 8) * (case["nz"] - 8) * s["nt"] for s in _shots(case, 0))


def work(case):
    e = 8 if case["precision"] == "fp64" else 4
    n = case["nx"] * case["nz"]
    if case["call"] == "optimizer":
        k = case["nt"]  # models in and out, gradients in; the two loops' axpys and dots over the pairs
        pairs = sum(min(j, 5) for j in range(1, k))
        return {"bytes": 3 * 4 * n * (2 + k), "flops": 3 * n * (8 * pairs + 12 * k)}
    if case["call"] == "compat":
        upd = (case["nx"] - 8) * (case["nz"] - 8) * case["nt"]
        return {"bytes": 4 * (6 * n + 3 * case["nx"] * case["nt"]) + 16 * n * case["nt"],
                "flops": upd * (FLOPS_FWD + FLOPS_ADJ + 40)}
    records = sum(s["nt"] * (s["rx1"] - s["rx0"]) for s in _shots(case, 0))
    grad = case["call"] == "gradient"
    return {"bytes": e * (3 * n + records + (3 * n if grad else 0)),
            "flops": _updates(case) * (FLOPS_FWD + (FLOPS_ADJ if grad else 0))}


D1 = (4 / 5, -1 / 5, 4 / 105, -1 / 280)
D2 = (-205 / 72, 8 / 5, -1 / 5, 8 / 315, -1 / 560)


def _taps(f, dim, c, sign, scale):
    """Sum of c[k] (f(+k) + sign f(-k)) along dim inside the 4-point frame, zero on it."""
    n = f.shape[dim]
    acc = None
    for k, w in enumerate(c, 1):
        t = f.narrow(dim, 4 + k, n - 8) + sign * f.narrow(dim, 4 - k, n - 8)
        acc = t * w if acc is None else acc.add_(t, alpha=w)
    out = torch.zeros_like(f)
    out.narrow(dim, 4, n - 8).copy_(acc.mul_(scale))
    return out


def _d1(f, dim):
    return _taps(f, dim, D1, -1.0, 1.0 / DH)


def _d2(f, dim):
    out = _taps(f, dim, D2[1:], 1.0, 1.0 / (DH * DH))
    n = f.shape[dim]
    out.narrow(dim, 4, n - 8).add_(f.narrow(dim, 4, n - 8), alpha=D2[0] / (DH * DH))
    return out


def _layers(case):
    """CPML a, b along x and z, the interior and the layer points, in 64 bits."""
    nx, nz, cp = case["nx"], case["nz"], case["cpml"]
    dt, f = float(np.float32(DT)), float(np.float32(case["freq"]))
    L = cp * DH
    d0 = -3 * math.log(float(np.float32(R_COEF))) / (2 * L)

    def table(dist):
        dist = dist.double()
        d = d0 * VMAX * (dist * DH / L) ** 2
        al = math.pi * f * (L - dist * DH) / L
        b = torch.exp(-(d + al) * dt)
        return torch.where(dist > 0, d * (b - 1) / (d + al), 0.0), torch.where(dist > 0, b, 0.0)
    ix, iz = torch.arange(nx, device=DEV), torch.arange(nz, device=DEV)
    dx = torch.clamp(torch.maximum(cp - ix, ix - nx + cp + 1), min=0)
    dz = torch.clamp(iz - nz + cp + 1, min=0)
    inner = ((ix > 3) & (ix < nx - 4))[None, :] & ((iz > 3) & (iz < nz - 4))[:, None]
    strip = inner & ((dx > 0)[None, :] | (dz > 0)[:, None])
    ax, bx = table(dx)
    az, bz = table(dz)
    return ax[None, :], bx[None, :], az[:, None], bz[:, None], inner.double(), strip.double()


def exact(case, seed):
    call, upd = case["call"], _updates(case) if case["call"] in ("gradient", "forward") else 0
    if call == "optimizer":
        return _exact_optimizer(case, seed)
    # the reference's adjoint, the boundary store's zero layers and the drop-in functions' mixed
    # precision have no plain 64-bit value here; nor have long batches, for their time and images
    if call == "compat" or case["uneven"] or (call == "gradient" and (case["mode"] == "ref" or case["store"] == "boundary")):
        return None
    if case["nt"] * 2.5e-3 + upd * (4e-10 if call == "forward" else 1e-9) > 18 or (call == "gradient" and upd > 4e9):
        return None
    shots = _shots(case, seed)
    nx, nz, nt, B = case["nx"], case["nz"], case["nt"], len(shots)
    vh, vp, vn = (m.double() for m in _model(case, seed))
    ax, bx, az, bz, inner, strip = _layers(case)
    w = _ricker(case)
    if case["precision"] == "fp32":
        w = w.astype(np.float32).astype(np.float64)
    dt2 = float(np.float32(DT)) ** 2
    zero = lambda: torch.zeros(B, nz, nx, dtype=torch.float64, device=DEV)  # noqa: E731
    P, F, VP, VF, psx, psz, zx, zz = (zero() for _ in range(8))
    sb = torch.arange(B, device=DEV)
    ssx, ssz = (torch.tensor([s[k] for s in shots], device=DEV) for k in ("sx", "sz"))
    rz, rx0, rx1 = shots[0]["rz"], shots[0]["rx0"], shots[0]["rx1"]
    rec = torch.zeros(nt, B, rx1 - rx0, dtype=torch.float64, device=DEV)
    grad = call == "gradient"
    img = torch.zeros(nt, 2, B, nz, nx, dtype=torch.float64, device=DEV) if grad else None
    for it in range(nt):
        psx = strip * (bx * psx + ax * _d1(P, 2))
        psz = strip * (bz * psz + az * _d1(F, 1))
        p2, r2 = inner * _d2(P, 2), inner * _d2(F, 1)
        tx, tz = strip * _d1(psx, 2), strip * _d1(psz, 1)
        zx = strip * (bx * zx + ax * (p2 + tx))
        zz = strip * (bz * zz + az * (r2 + tz))
        G, H = p2 + tx + zx, r2 + tz + zz
        VP += dt2 * (vh * G + vp * H)
        VF += dt2 * (vn * G + vp * H)
        VP[sb, ssz, ssx] += w[it]
        VF[sb, ssz, ssx] += w[it]
        P, F = P + VP, F + VF
        rec[it] = P[:, rz, rx0:rx1] + F[:, rz, rx0:rx1]
        if grad:
            img[it, 0], img[it, 1] = G, H
    if not grad:
        return {"traces": rec.permute(1, 0, 2).reshape(-1)}
    dtype = torch.float64 if case["precision"] == "fp64" else torch.float32
    obs = _records(case, seed, shots, dtype).double().reshape(B, nt, rx1 - rx0).permute(1, 0, 2)
    res = rec - obs
    mask = _mask(case, seed, shots)
    if mask is not None:
        res = res * torch.from_numpy(mask.reshape(B, -1)).to(DEV).double()
    J = 0.5 * float((res * res).sum())
    lP, lF, WP, WF, Zx, Zz, Yx, Yz = (zero() for _ in range(8))
    g = [torch.zeros(nz, nx, dtype=torch.float64, device=DEV) for _ in range(3)]
    for m in range(nt - 1, -1, -1):
        gx, hz = dt2 * inner * (vh * lP + vn * lF), dt2 * inner * vp * (lP + lF)
        Zx, Zz = strip * (gx + bx * Zx), strip * (hz + bz * Zz)
        wx, wz = strip * (gx + ax * Zx), strip * (hz + az * Zz)
        Yx = strip * (-_d1(wx, 2) + bx * Yx)
        Yz = strip * (-_d1(wz, 1) + bz * Yz)
        WP += inner * (_d2(gx + ax * strip * Zx, 2) - _d1(ax * Yx, 2))
        WF += inner * (_d2(hz + az * strip * Zz, 1) - _d1(az * Yz, 1))
        WP[:, rz, rx0:rx1] += res[m]
        WF[:, rz, rx0:rx1] += res[m]
        lP, lF = lP + WP, lF + WF
        G, H = img[m, 0], img[m, 1]
        g[0] += dt2 * (G * lP).sum(0)
        g[1] += dt2 * (H * (lP + lF)).sum(0)
        g[2] += dt2 * (G * lF).sum(0)
    return {"misfit": J, "v_hor": g[0], "v_po": g[1], "v_nmo": g[2]}


def _exact_optimizer(case, seed):
    """The first step and the two-loop recursion (memory 5) in 64 bits, per parameter."""
    model = _model(case, seed)
    grads = _gradients(case, seed, model)
    m = [t.double() for t in model]
    below = torch.zeros(case["nz"], 1, dtype=torch.float64, device=DEV)
    below[16:] = 1.0
    first = (3e5, 2e5, 2.5e5)
    back_m, back_g, pairs = None, None, [[], [], []]
    for k in range(case["nt"]):
        g = [t.double() for t in grads[k]]
        if k == 0:
            step = [a * x / x.norm() for a, x in zip(first, g)]
            base = m
        else:
            step = []
            for p in range(3):
                pairs[p] = (pairs[p] + [(m[p] - back_m[p], g[p] - back_g[p])])[-5:]
                q, al = g[p].clone(), []
                for s, y in reversed(pairs[p]):
                    a = (s * q).sum() / (s * y).sum()
                    al.append(a)
                    q -= a * y
                s, y = pairs[p][-1]
                r = q * ((s * y).sum() / (y * y).sum())
                for (s, y), a in zip(pairs[p], reversed(al)):
                    r += s * (a - (y * r).sum() / (s * y).sum())
                step.append(r)
            base = m
        back_m, back_g = base, g
        m = [b - below * x for b, x in zip(base, step)]
        m[0] = torch.where(below > 0, torch.maximum(m[0], m[2]), m[0])
    return {"v_hor": m[0], "v_po": m[1], "v_nmo": m[2]}
