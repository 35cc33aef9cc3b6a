"""div2, the FP64 update's two quotients from one reciprocal, against the division
operator: the same bits for every pair of special operands (zeros, subnormals,
infinities, NaN, the bounds of its range, divisors at and next to the guard below a
power of two) and for 2^30 random pairs of each of six classes (tests/native/div2.cu).
Both are correctly rounded, so nothing may differ."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "bsam_b200", "csrc")


def test_div2_is_the_operator(gpu_lib, tmp_path):
    from bsam_b200 import build as B
    exe = str(tmp_path / "div2")
    r = subprocess.run([B.nvcc(), "-O3", "-std=c++17", *B.ARCH, "--fmad=false", f"-I{CSRC}",
                        os.path.join(HERE, "native", "div2.cu"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
    compared, bad = (int(v) for v in r.stdout.split())
    assert compared > 1.2e10 and bad == 0
