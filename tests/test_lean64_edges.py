"""lean_log and lean_exp (host build of the device source) at the edges of
their ranges: the exponents where the log's fixed-point scale changes (|e| = 0,
15, 16), the ends of its window around 1, every table bin's two ends, and the
exp's small arguments (2^-11, where x starts to be cut), the two halves of T_0
and the ends of its fast range."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from noa_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def evaluate(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    d = tmp_path_factory.mktemp("lean64_edges")
    exe = str(d / "lean64_host_check")
    subprocess.run([nvcc, "-std=c++17", "-O2", "-Xcompiler", "-ffp-contract=off", "-I",
                    os.path.join(build.ROOT, "include"), "-o", exe, os.path.join(HERE, "lean64_host_check.cu")],
                   check=True, capture_output=True)

    def run(x):
        x.tofile(d / "x.bin")
        subprocess.run([exe, "values", str(d / "x.bin"), str(d / "y.bin")], check=True, timeout=300)
        y = np.fromfile(d / "y.bin")
        return y[:x.size], y[x.size:]
    return run


def neighbours(x, k=40):
    """Each value and the k doubles on either side of it."""
    b = np.ascontiguousarray(x, dtype=np.float64).view(np.int64)
    return (b[:, None] + np.arange(-k, k + 1)).ravel().view(np.float64)


def ulps(got, ref):
    return np.abs(got - ref).astype(np.float64) / np.spacing(np.abs(ref.astype(np.float64)))


@pytest.mark.parametrize("exponent", [0, -1, 1, 14, 15, 16, -14, -15, -16, 17, -17, 1023, -1022])
def test_log(evaluate, exponent):
    t = 1 + np.arange(256) / 256.0
    x = neighbours(np.concatenate([t, [np.sqrt(0.5) * 2, 1 + 2.0 ** -9, 2 - 2.0 ** -8 + 2.0 ** -10]]))
    x = x[(x >= 1) & (x < 2)] * 2.0 ** exponent
    got, _ = evaluate(x)
    # half an ulp of rounding, and at the smallest |log| outside the window (2^-9, ulp 2^-62) units of
    # 2^-64 for the table, 2^-63 / 2 for the rounded correction and ~2^-64 for its float-float value
    assert ulps(got, np.log(x.astype(np.longdouble))).max() <= 1.0


@pytest.mark.parametrize("centre", [2.0 ** -11, 2.0 ** -10, 2.0 ** -52, 2.0 ** -64, 1e-40, np.log(2) / 256,
                                    np.log(2) / 2, 1.0, 37.0, 699.9])
def test_exp(evaluate, centre):
    x = neighbours([centre])
    x = np.concatenate([x, -x, np.log(2) * np.arange(-8, 9) / 128, np.log(2) * (np.arange(-8, 8) + 0.5) / 128])
    _, got = evaluate(x)
    # half an ulp, and a few units of 2^-61 (2^-8 ulp)
    assert ulps(got, np.exp(x.astype(np.longdouble))).max() <= 0.53
