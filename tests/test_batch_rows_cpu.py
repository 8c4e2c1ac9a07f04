"""Segments and filter groups of a launch (plan_segments, filter_batch,
fft3dcl_gb300/csrc/f3d_batch_plan.hpp) on the CPU over the segments engines
ask for: compiles tests/batch_plan/rows.cpp with the host compiler against the
CUDA runtime headers (no GPU needed)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


def test_rows(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None or not os.path.exists(os.path.join(CUDA_INC, "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA runtime headers")
    exe = str(tmp_path / "rows")
    subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-I", os.path.join(ROOT, "fft3dcl_gb300", "csrc"),
                    "-I", os.path.join(ROOT, "include"), "-I", CUDA_INC,
                    os.path.join(ROOT, "tests", "batch_plan", "rows.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
