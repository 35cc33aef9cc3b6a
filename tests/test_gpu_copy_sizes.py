"""put_field / get_field round trips at the edges of the copy paths (the bounce
buffer up to 128 KiB, the driver's pitched copies, pieces copied by several host
threads from 8 MiB), in 2D and 3D, and twice in a row from one array."""
import numpy as np
import pytest

import bsam_b200 as B
from bsam_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mx", [(2, 2), (34, 6), (88, 88), (88, 90), (256, 256), (720, 724), (722, 724),
                                (1022, 512),
                                (2, 2, 2), (62, 30, 14), (64, 64, 128), (100, 70, 76)])
def test_fields_come_back_as_put(gpu_lib, mx):
    nd = len(mx)
    rng = np.random.default_rng(sum(mx))
    h = 1.0 / mx[0]
    prob = W.Problem(ndims=nd, mx=tuple(mx) + (1,) * (3 - nd), eps=0.02, dt=1e-4, nsteps=1,
                     qerrortol=1e-8, xupper=tuple([n * h for n in mx] + [1.0] * (3 - nd)),
                     c0=np.full(int(np.prod(mx)), 0.5))
    shape = tuple(m + 2 for m in mx) + (2,)
    a = np.asfortranarray(rng.standard_normal(shape))
    b = np.asfortranarray(rng.standard_normal(shape))
    out = np.empty(shape, order="F")
    with B.Solver(prob) as s:
        s.put_q(a)
        s.get_q_into(out)
        assert np.array_equal(out, a)
        work = a.copy(order="F")
        s.put_q(work)
        work[...] = b  # the array is the caller's again once put returns
        s.get_q_into(out)
        assert np.array_equal(out, a)
        s.put_q(a)
        s.put_q(b)
        s.get_q_into(out)
        assert np.array_equal(out, b)


# Rows of several parts (a warp each), and pieces of either size: rows below 4 KB
# from 8 MiB (128 KB a piece, 256 from 24 MiB), longer rows from 32 MiB.
@pytest.mark.parametrize("mx", [(510, 8), (4094, 2), (400, 1280), (400, 1310), (508, 1100),
                                (30, 20000), (400, 4000), (1030, 1024), (2046, 1020),
                                (2046, 1030), (5000, 424), (62, 62, 130), (40, 200, 190)])
def test_long_rows_and_pieces(gpu_lib, mx):
    nd = len(mx)
    rng = np.random.default_rng(sum(mx))
    h = 1.0 / mx[0]
    prob = W.Problem(ndims=nd, mx=mx + (1,) * (3 - nd), eps=0.02, dt=1e-4, nsteps=1,
                     qerrortol=1e-8, xupper=tuple([n * h for n in mx] + [1.0] * (3 - nd)),
                     c0=np.full(int(np.prod(mx)), 0.5))
    a = np.asfortranarray(rng.standard_normal(tuple(m + 2 for m in mx) + (2,)))
    out = np.zeros_like(a, order="F")
    with B.Solver(prob) as s:
        s.put_q(a)
        s.get_q_into(out)
    assert np.array_equal(out, a)


STARVED = """
import ctypes, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
import bsam_b200 as B
from bsam_b200 import workloads as W

mx = (400, 2600)
prob = W.Problem(ndims=2, mx=mx + (1,), eps=0.02, dt=1e-4, nsteps=1, qerrortol=1e-8,
                 xupper=(1.0, mx[1] / mx[0], 1.0), c0=np.full(int(np.prod(mx)), 0.5))
shape = tuple(m + 2 for m in mx) + (2,)
a = np.asfortranarray(np.random.default_rng(1).standard_normal(shape))
out = np.zeros(shape, order="F")
s = B.Solver(prob)
# Every thread started from here on wants a 64 TiB stack, which is refused.
attr = ctypes.create_string_buffer(256)
libc = ctypes.CDLL(None)
assert libc.pthread_attr_init(attr) == 0
assert libc.pthread_attr_setstacksize(attr, ctypes.c_size_t(1 << 46)) == 0
assert libc.pthread_setattr_default_np(attr) == 0
s.put_q(a)
s.get_q_into(out)
print("equal" if np.array_equal(a, out) else "different")
"""


def test_large_copies_without_threads(gpu_lib):
    """Where no copy thread can be had, the calling thread does the work."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", STARVED, root], capture_output=True, text=True,
                       timeout=300)
    assert r.stdout.strip() == "equal", (r.returncode, r.stderr[-2000:])
