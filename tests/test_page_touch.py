"""The page-touching thread of rrlu's results (tests/host/page_touch_check.cpp)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "tensorcrossinterpolation.jl_gb300", "csrc")


def test_page_touching_thread(tmp_path):
    cxx = shutil.which(os.environ.get("CXX", "g++"))
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "page_touch_check")
    r = subprocess.run([cxx, "-std=c++20", "-O1", "-I", CSRC, os.path.join(HERE, "host", "page_touch_check.cpp"),
                        "-o", exe, "-lpthread"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


def test_rrlu_has_no_bare_thread():
    """tci_rrlu starts its thread through that class only: a std::thread that is still
    joinable when the call ends by an exception ends the process."""
    with open(os.path.join(CSRC, "capi.cpp")) as fh:
        text = fh.read()
    body = text[text.index("int tci_rrlu(tci_ctx* ctx"):text.index("int tci_rrlu_batched(tci_ctx* ctx")]
    assert "std::thread" not in body and "PageToucher" in body
