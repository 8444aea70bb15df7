"""lean64's integer arithmetic (host builds of the device source) under the
undefined-behaviour sanitizer: its sums and products that wrap are unsigned."""
import os
import shutil
import subprocess

import pytest

from noa_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("source,args", [("lean64_host_check.cu", ["20000"]), ("fixed_point_check.cu", [])])
def test_no_undefined_arithmetic(tmp_path, source, args):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "check")
    built = subprocess.run([nvcc, "-std=c++17", "-O1", "-Xcompiler",
                            "-ffp-contract=off,-fsanitize=signed-integer-overflow,-fsanitize=shift", "-I",
                            os.path.join(build.ROOT, "include"), "-o", exe, os.path.join(HERE, source), "-lubsan"],
                           capture_output=True, text=True)
    if built.returncode and "ubsan" in built.stderr:
        pytest.skip("no sanitizer library")
    assert built.returncode == 0, built.stderr
    out = subprocess.run([exe, *args], check=True, capture_output=True, text=True, timeout=600)
    assert "runtime error" not in out.stderr, out.stderr
