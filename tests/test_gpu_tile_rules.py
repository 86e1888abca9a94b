"""The tile rules of the kernels themselves (test_split_rule.py restates them): the
division-free index split and the fixed-point scale, run on the device over every
input by a small program built with nvcc from tests/native/."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.gpu
@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not available")
def test_split_and_scale_on_the_device(tmp_path):
    exe = str(tmp_path / "tile_check")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O2", "--expt-relaxed-constexpr",
                    os.path.join(HERE, "native", "tile_check.cu"), "-o", exe], check=True, timeout=600)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "OK", (r.stdout, r.stderr)
