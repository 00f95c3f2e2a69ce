"""The kernels' reciprocal (qas_device.cuh: rcp_positive) equals the IEEE quotient on the device at the significands
where its derivation needs care, over every exponent of its range, and its seed is within what the derivation uses."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu
def test_reciprocal_points(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "reciprocal_points")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "--fmad=false", "-std=c++17",
                    "-I", os.path.join(ROOT, "qasmhd_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "reciprocal_points.cu"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
