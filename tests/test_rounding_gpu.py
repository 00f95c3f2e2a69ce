"""The kernels' short division forms give the IEEE quotients on the device (qas_device.cuh:
rcp_normal, div24), and cells beyond the range of the fast interpolation take the reference's
divisions."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from oracle import refcase as R
from qasmhd_b200 import problems as P
from tests.cases import assert_bitwise, run_gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu
def test_short_divisions_are_ieee(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "rounding_points")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "--fmad=false", "-std=c++17",
                    "-I", os.path.join(ROOT, "qasmhd_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "rounding_points.cu"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


def _scaled(prob, k):
    """The same flow in other units: velocities and fields times 2^k, pressures and energy times 4^k
    (exact, and the step scales with it as long as nothing leaves the number range)."""
    p = prob.copy()
    s = 2.0 ** k
    p.state[1:7] *= s
    p.state[7] *= s * s
    return p


@pytest.mark.gpu
@pytest.mark.parametrize("make", [lambda: P.orszag_tang(24, nym=17), lambda: P.kelvin_helmholtz(3, 12, nym=9, nzm=11, mach=0.3),
                                  lambda: P.kelvin_helmholtz(2, 33, nym=21, mach=0.3, rmn=0)],
                         ids=["ot2d_hlld", "kh3d_mlau", "kh2d_roe"])
@pytest.mark.parametrize("k", [60, 115, 127])
def test_large_magnitudes(make, k):
    """Pressures of 2^120 (within the fast interpolation), 2^230 and 2^254: the smoothness
    denominators pass 2^900 and, at the last, overflow.  Bit for bit the oracle's step."""
    p = _scaled(make(), k)
    dt = 1e-3 * 2.0 ** -k
    want = R.Restatement().run(p, 1, mode=R.MODE_STEP, dt=dt)["state"]
    assert np.isfinite(want).all()
    got = run_gpu(p, R.MODE_STEP, dt=dt)["state"]
    assert_bitwise(got, want.reshape(got.shape), f"{p.name} 2^{k}")
