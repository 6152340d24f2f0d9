"""Contexts of one process on the resident path from several threads at once: their launches share the
device's SMs (other plans than alone) or wait for them, and each gets, bit for bit, what it gets alone.  Forward and adjoint resident, tile forward with a resident adjoint, checkpoints with a
recompute, and a context on the tile passes beside them; one context goes away while others run."""
import threading

import numpy as np
import pytest

from test_native_gpu import exact_problem, wavelet

pytestmark = pytest.mark.gpu

PROBLEMS = [  # nx, nz, cpml, shots, store, images
    (209, 90, 20, 1, "FULL", "NATIVE"),
    (501, 60, 12, 2, "FULL", "FP16"),
    (140, 77, 13, 3, "CHECKPOINT", "BF16"),
    (120, 90, 20, 2, "BOUNDARY", "FP16"),
    (72, 56, 12, 2, "FULL", "NATIVE"),
]


def test_contexts_in_threads_get_what_they_get_alone():
    import fwi_gb300 as f
    nt, calls = 160, 6
    work = []
    for nx, nz, cpml, n, store, images in PROBLEMS:
        p = exact_problem(seed=nx, nx=nx, nz=nz, nt=nt)
        ctx = f.Context(nx=nx, nz=nz, dh=p["dh"], dt=p["dt"], cpml=cpml, f_cpml=p["f"], nt_max=nt, max_shots=n,
                        store=getattr(f, "STORE_" + store), store_prec=getattr(f, "SPREC_" + images))
        ctx.set_wavelet(wavelet(p).astype(np.float32))
        ctx.set_model(*(np.ascontiguousarray(p[k], np.float32) for k in ("vh", "vp", "vn")))
        sh = f.make_shots([dict(sx=4 + (nx - 9) * (k + 1) // (n + 1), sz=6, rz=6, rx0=4, rx1=nx - 4, nt=nt, x0=0, nxw=0)
                           for k in range(n)])
        obs = np.random.default_rng(nx).standard_normal(n * nt * (nx - 8)).astype(np.float32)
        alone = (ctx.forward(sh), ctx.gradient(sh, obs))
        work.append((ctx, sh, obs, alone))
    failed, start = [], threading.Barrier(len(work))

    def run(k):
        ctx, sh, obs, (t0, g0) = work[k]
        try:
            start.wait(30)
            for c in range(calls if k else 2):
                t, g = ctx.forward(sh), ctx.gradient(sh, obs)
                if not (np.array_equal(t, t0) and g[0] == g0[0] and all(np.array_equal(a, b) for a, b in zip(g[1:], g0[1:]))):
                    failed.append((k, c))
            if k == 0:
                ctx.close()
        except Exception as e:  # noqa: BLE001
            failed.append((k, repr(e)))

    threads = [threading.Thread(target=run, args=(k,)) for k in range(len(work))]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not any(t.is_alive() for t in threads) and not failed, failed


def test_threads_share_the_device():
    """Four contexts, one shot each (a shot of this size fills a quarter of the device): four threads
    take less than 3 times as long as one (1.1 times where this was written, 4 times in turn)."""
    import time

    import fwi_gb300 as f
    p = exact_problem(seed=3, nx=209, nz=209, nt=1000)
    work = []
    for k in range(4):
        ctx = f.Context(nx=209, nz=209, dh=p["dh"], dt=p["dt"], cpml=20, f_cpml=p["f"], nt_max=1000, max_shots=1)
        ctx.set_wavelet(wavelet(p).astype(np.float32))
        ctx.set_model(*(np.ascontiguousarray(p[k], np.float32) for k in ("vh", "vp", "vn")))
        sh = f.make_shots([dict(sx=60 + 30 * k, sz=6, rz=6, rx0=100, rx1=104, nt=1000, x0=0, nxw=0)])
        work.append((ctx, sh, np.zeros(4000, np.float32)))

    def calls(w, barrier):
        barrier.wait(30)
        for _ in range(10):
            w[0].misfit(w[1], w[2])

    def seconds(ws):
        barrier = threading.Barrier(len(ws) + 1)
        threads = [threading.Thread(target=calls, args=(w, barrier)) for w in ws]
        for t in threads:
            t.start()
        barrier.wait(30)
        t0 = time.perf_counter()
        for t in threads:
            t.join(60)
        return time.perf_counter() - t0

    seconds(work)
    one = min(seconds(work[:1]) for _ in range(3))
    assert min(seconds(work) for _ in range(3)) < 3 * one


@pytest.mark.parametrize("polls", [1, 64, 4096])
def test_resident_waits_give_up(polls):
    """The wait for a neighbour's rows, on a word that nothing writes, ends after its polls, is reported,
    and leaves a context whose resident calls give what they gave."""
    import fwi_gb300 as f
    p = exact_problem(seed=2, nx=140, nz=100, nt=120)
    ctx = f.Context(nx=140, nz=100, dh=p["dh"], dt=p["dt"], cpml=12, f_cpml=p["f"], nt_max=120, max_shots=1)
    ctx.set_wavelet(wavelet(p).astype(np.float32))
    ctx.set_model(*(np.ascontiguousarray(p[k], np.float32) for k in ("vh", "vp", "vn")))
    sh = f.make_shots([dict(sx=70, sz=6, rz=6, rx0=4, rx1=136, nt=120, x0=0, nxw=0)])
    obs = np.zeros(120 * 132, np.float32)
    first = ctx.gradient(sh, obs)
    assert ctx.check_bounded_wait(polls) == -2  # FWI_ERR_CUDA
    again = ctx.gradient(sh, obs)
    assert again[0] == first[0] and all(np.array_equal(a, b) for a, b in zip(again[1:], first[1:]))
