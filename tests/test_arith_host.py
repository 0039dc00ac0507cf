"""The device's 64-bit arithmetic (erdos-strauss_gb300/csrc/es_arith.cuh) compiled for the host."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_montgomery_constants_without_signed_overflow(tmp_path):
    exe = str(tmp_path / "arith_host_check")
    src = os.path.join(os.path.dirname(__file__), "arith_host_check.cpp")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fsanitize=signed-integer-overflow", "-fsanitize-undefined-trap-on-error",
                    "-I", os.path.join(PKG, "csrc"), src, "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + str(out.returncode)
