"""The shared-memory limits of the evaluation and tensor-core kernels are set on
every device that launches them (tests/host/device_limits_check.cpp: their host code
against a stand-in for the CUDA runtime, no GPU)."""
import os
import shutil
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "tensorcrossinterpolation.jl_gb300")


def test_kernel_limits_on_every_device(tmp_path):
    cxx = shutil.which(os.environ.get("CXX", "g++"))
    if cxx is None:
        pytest.skip("no C++ compiler")
    sys.path.insert(0, PKG)
    try:
        import build as B
    finally:
        sys.path.remove(PKG)
    B.build()
    exe = str(tmp_path / "device_limits_check")
    cmd = [cxx, "-std=c++20", "-O1", "-I", os.path.join(PKG, "csrc"), "-I", os.path.join(B.CUDA_HOME, "include"),
           os.path.join(HERE, "host", "device_limits_check.cpp")]
    cmd += [os.path.join(B.BUILD, name + ".cu.o") for name in ("tt_eval", "tc_gemm")] + ["-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
