"""The shared-memory addresses that the chain kernel's threads form, replayed on the
host with the kernel's own functions over all even extents up to 512 x 256 and
40 x 40 x 64 with every combination of periodic and physical faces in the first and
last dimension, clusters of 16 and 8, FP64 and mixed: all inside the level's own
field.  (A CTA that holds no rows of a level used to read a periodic neighbour a
whole level away: 110 x 28, periodic in y, has 14 pairs of rows for 16 CTAs.)
Compiles for the host and runs here: no GPU needed."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "bsam_b200", "csrc")


def nvcc():
    for c in (shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if c and os.path.exists(c):
            return c
    return None


@pytest.mark.skipif(nvcc() is None, reason="nvcc not found")
def test_every_address_lies_in_its_level(tmp_path):
    exe = str(tmp_path / "chain_reads")
    r = subprocess.run([nvcc(), "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a",
                        f"-I{CSRC}", os.path.join(HERE, "native", "chain_reads.cu"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    chains, idle, bad = (int(v) for v in r.stdout.split())
    assert chains > 50000
    assert idle > 500  # the case that went wrong is among them
    assert bad == 0, r.stderr
