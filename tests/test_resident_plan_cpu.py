"""The resident path's plan, checked on the CPU.

Builds tests/resident_plan_check.cpp against fwi_gb300/csrc/resident_plan.h with g++ and runs it:
over a sweep of windows, grid heights, layer widths, batches and device sizes, every launch fits
the SMs, threads, registers and shared memory, covers each row and column pair once, forms no index
outside its arrays, and every exchanged row is published by a CTA close enough that none of its
copies is overwritten unread.
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


def test_resident_plan(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None or not os.path.exists(os.path.join(CUDA_INC, "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    exe = tmp_path / "resident_plan_check"
    subprocess.run([gxx, "-std=c++17", "-O2", "-include", "cuda_runtime.h", f"-I{CUDA_INC}",
                    os.path.join(ROOT, "tests", "resident_plan_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.startswith("OK"), out.stdout
