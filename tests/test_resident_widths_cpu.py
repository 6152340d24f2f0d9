"""The search of the resident path's plan, on the CPU: builds tests/resident_widths_check.cpp against
fwi_gb300/csrc/resident_plan.h with g++ and runs it (the cheapest partitions against a search of all
splits, plans with kept widths against plans without, the time a plan takes)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


def test_resident_widths(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None or not os.path.exists(os.path.join(CUDA_INC, "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    exe = tmp_path / "resident_widths_check"
    subprocess.run([gxx, "-std=c++17", "-O2", "-include", "cuda_runtime.h", f"-I{CUDA_INC}",
                    os.path.join(ROOT, "tests", "resident_widths_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.startswith("OK"), out.stdout
