"""The tile layout of the batched engine's plans on the host: the autotuner has to
time each shape at the tile at which the plan would run it, whatever prefix of the
segments it times."""
import os
import shutil
import subprocess

import pytest

from noa_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))


def test_sampled_layout_keeps_the_tile(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "batch_tiles_check")
    subprocess.run([nvcc, *build.ARCH, "-std=c++17", "-O1", "--expt-relaxed-constexpr", "-I",
                    os.path.join(build.ROOT, "include"), "-o", exe, os.path.join(HERE, "batch_tiles_check.cu")],
                   check=True, capture_output=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=60).stdout.split()
    assert out[0] == "shapes" and int(out[1]) == 1008
    assert int(out[3]) == 0
