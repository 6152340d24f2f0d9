"""The rows that the resident path's CTAs exchange, on the CPU: builds tests/resident_exchange_check.cpp against
fwi_gb300/csrc/resident_plan.h with g++ and runs it (copies kept, orders of the CTAs' steps, words taken);
and fwi_config_bytes counts them: they lie in state that is idle meanwhile, and only a context of one
shot needs more, 72 bytes a point at the kernels' row pitch against 56 idle, and 20 KB."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

from fwi_gb300 import native

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


def test_resident_exchange(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None or not os.path.exists(os.path.join(CUDA_INC, "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    exe = tmp_path / "resident_exchange_check"
    subprocess.run([gxx, "-std=c++17", "-O2", "-include", "cuda_runtime.h", f"-I{CUDA_INC}",
                    os.path.join(ROOT, "tests", "resident_exchange_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.startswith("OK"), out.stdout


@pytest.fixture(scope="module")
def lib():
    from fwi_gb300 import build
    build.build()
    return native.lib()


@pytest.mark.parametrize("store", [native.STORE_FULL, native.STORE_CHECKPOINT, native.STORE_BOUNDARY])
@pytest.mark.parametrize("nx,nz,window", [(209, 209, 0), (609, 309, 0), (72, 56, 0), (4009, 1209, 1603), (130, 400, 129)])
def test_config_bytes_count_the_exchange(lib, store, nx, nz, window):
    def extra(shots):
        cfg = native.Config()
        lib.fwi_config_default(C.byref(cfg))
        cfg.nx, cfg.nz, cfg.max_window, cfg.max_shots, cfg.store, cfg.nt_max = nx, nz, window, shots, store, 500
        cfg.store_prec = native.SPREC_FP16
        cfg.precision = native.PREC_FP32
        total = lib.fwi_config_bytes(C.byref(cfg))
        cfg.store_prec, cfg.precision = native.SPREC_NATIVE, native.PREC_FP64  # the same arrays, of 8 bytes, no exchange
        images = 2 * shots * 2 if store == native.STORE_BOUNDARY else 0
        if store == native.STORE_FULL:
            images = shots * 500 * 2
        if store == native.STORE_CHECKPOINT:
            return None, total
        slot = nz * ((window or nx) + 31 >> 5 << 5)
        return total - (lib.fwi_config_bytes(C.byref(cfg)) // 2 - images * slot * 2), slot

    one, slot = extra(1)
    if one is None:
        return
    four, _ = extra(4)
    assert 0 <= one <= 48 * slot + 20736 and 0 <= four <= 8 * 4 * slot + 20736
    if (nx, store) == (209, native.STORE_FULL):
        assert one == (72 * 224 - 56 * 224) * 209 + 20480 and four == 0
