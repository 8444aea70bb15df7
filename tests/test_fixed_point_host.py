"""lean64's fixed-point functions (host build of the device source) against
long double libm.  Bars: a logarithm's 2^e carries |e| <= 58 halves of a unit
(2^-57), one for the cut, and 8 where the argument is itself cut to 2^-54
relative; an exponential below 64 as an integer 2^-60 relative and one for the
cut; a result rounded to double half an ulp and 2^-60 relative before it."""
import os
import shutil
import subprocess

import pytest

from noa_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))
BARS = {"log": 31, "log3p": 39, "log_of": 39, "exp": 0.51, "exp_to": 10, "ratio": 0.51, "round_by_one": 0}


@pytest.fixture(scope="module")
def report(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path_factory.mktemp("fixed_point") / "check")
    subprocess.run([nvcc, "-std=c++17", "-O2", "-Xcompiler", "-ffp-contract=off", "-I",
                    os.path.join(build.ROOT, "include"), "-o", exe, os.path.join(HERE, "fixed_point_check.cu")],
                   check=True, capture_output=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=600).stdout
    return {k: float(v) for k, v in (line.split() for line in out.splitlines())}


@pytest.mark.parametrize("name", sorted(BARS))
def test_error(report, name):
    assert report[name] <= BARS[name]
