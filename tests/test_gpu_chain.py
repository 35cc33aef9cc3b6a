"""The coarse end of the V-cycle in one cluster's shared memory (k_chain) against
the same levels as grid launches (bottom_cells=-1), which the parity tests pin:
every value the same bit for bit, at the sizes where the chain can go wrong --
one CTA or a cluster, rows dealt out unevenly, levels two cells wide, odd
coarsest levels, one or several pairs of cells per thread, each face rule -- in
2D and 3D, FP64 (with the V-cycle loop in the kernel where the whole solve fits)
and mixed."""
import numpy as np
import pytest

import bsam_b200 as B
from bsam_b200 import workloads as W

pytestmark = pytest.mark.gpu

SIZES = [(2, 2), (4, 2), (16, 2), (2, 64), (32, 16), (16, 16), (34, 34), (50, 30), (24, 40),
         (128, 128), (192, 96), (200, 8), (2, 2, 2), (8, 8, 8), (12, 20, 4), (16, 16, 16),
         (24, 16, 40), (32, 32, 32), (6, 10, 64)]


def problem(mx, faces):
    nd = len(mx)
    rng = np.random.default_rng(int(np.prod(mx)))
    h = 1.0 / mx[0]
    return W.Problem(ndims=nd, mx=tuple(mx) + (1,) * (3 - nd), eps=0.02, dt=1e-4, nsteps=2,
                     qerrortol=1e-12, maxvcycles=4,
                     mthbc=tuple(faces) + (1,) * (6 - 2 * nd),
                     xupper=tuple([n * h for n in mx] + [1.0] * (3 - nd)),
                     c0=0.5 + 0.1 * rng.uniform(-1, 1, int(np.prod(mx))))


def solve(prob, precision, bottom_cells):
    with B.Solver(prob, precision=precision, bottom_cells=bottom_cells) as s:
        steps = [s.step() for _ in range(prob.nsteps)]
        return steps, s.trace(), s.get_q()


@pytest.mark.parametrize("precision", [B.PREC_FP64, B.PREC_MIXED])
@pytest.mark.parametrize("faces", ["neumann", "user", "periodic_x", "periodic_last"])
@pytest.mark.parametrize("mx", SIZES)
def test_chain_equals_the_levels_as_launches(gpu_lib, mx, faces, precision):
    nd = len(mx)
    codes = {"neumann": [1] * (2 * nd), "user": [10] * (2 * nd),
             "periodic_x": [2, 2] + [10] * (2 * nd - 2),
             "periodic_last": [1] * (2 * nd - 2) + [2, 2]}[faces]
    odd = list(mx)  # a periodic dimension is even or 1 on every level
    while all(n % 2 == 0 for n in odd):
        odd = [n // 2 for n in odd]
    d = {"periodic_x": 0, "periodic_last": nd - 1}.get(faces)
    if d is not None and odd[d] % 2 and odd[d] > 1:
        pytest.skip("not a periodic extent")
    prob = problem(mx, codes)
    want = solve(prob, precision, -1)
    got = solve(prob, precision, 0)
    assert got[0] == want[0]
    assert np.array_equal(got[1], want[1])
    assert np.array_equal(got[2], want[2])


def test_first_sweep_reads_the_ghosts_as_given(gpu_lib):
    """A solve started on a state whose ghost ring is not what SetGhost gives
    reads it as it stands, chain or launches."""
    prob = problem((64, 48), [1, 1, 10, 10])
    q0 = prob.q0()
    rng = np.random.default_rng(3)
    ring = np.ones(q0.shape[:2], dtype=bool)
    ring[1:-1, 1:-1] = False
    q0[ring] += 0.01 * rng.standard_normal((int(ring.sum()), 2))
    out = []
    for cells in (-1, 0):
        with B.Solver(prob, bottom_cells=cells) as s:
            s.put_q(q0)  # and no SetGhost
            L = B.lib()
            import ctypes
            nv, conv, res = ctypes.c_int(0), ctypes.c_int(0), ctypes.c_double(0.0)
            assert L.bsam_gpu_copy_q_to_qold(s.h) == 0
            assert L.bsam_gpu_multigrid_iterations(s.h, ctypes.byref(nv), ctypes.byref(res),
                                                   ctypes.byref(conv)) == 0
            out.append((nv.value, res.value, s.trace(), s.get_q()))
    assert out[0][:2] == out[1][:2]
    assert np.array_equal(out[0][2], out[1][2])
    assert np.array_equal(out[0][3], out[1][3])


def test_coarse_levels_are_readable(gpu_lib):
    """q and f of the levels below the root, as get_field returns them."""
    prob = problem((64, 48), [10, 10, 1, 1])
    out = []
    for cells in (-1, 0):
        with B.Solver(prob, bottom_cells=cells) as s:
            s.step()
            out.append([(s.get_q(p), s.get_f(p)) for p in range(s.npatch)])
    for (qa, fa), (qb, fb) in zip(*out):
        assert np.array_equal(qa, qb)
        assert np.array_equal(fa, fb)


# More CTAs in the cluster than the level has pairs of rows (planes), the last
# dimension periodic: the CTAs without rows take no part in the level.
@pytest.mark.parametrize("precision", [B.PREC_FP64, B.PREC_MIXED])
@pytest.mark.parametrize("mx", [(110, 28), (98, 24), (44, 56), (126, 12), (10, 18, 24),
                                (16, 24, 16), (22, 14, 12)])
def test_clusters_with_ctas_without_rows(gpu_lib, mx, precision):
    nd = len(mx)
    prob = problem(mx, [1] * (2 * nd - 2) + [2, 2])
    want = solve(prob, precision, -1)
    got = solve(prob, precision, 0)
    assert got[0] == want[0]
    assert np.array_equal(got[1], want[1])
    assert np.array_equal(got[2], want[2])


@pytest.mark.parametrize("precision", [B.PREC_FP64, B.PREC_MIXED])
@pytest.mark.parametrize("mx", [(256, 256), (40, 40, 48), (40, 48, 56), (48, 48, 48), (64, 32, 64)])
def test_chains_of_the_largest_tops(gpu_lib, mx, precision):
    """Levels just inside the size to which the chain reaches below other levels."""
    prob = problem(mx, [10] * (2 * len(mx)))
    want = solve(prob, precision, -1)
    got = solve(prob, precision, 0)
    assert got[0] == want[0]
    assert np.array_equal(got[1], want[1])
    assert np.array_equal(got[2], want[2])


RESET = """
import ctypes, glob, os, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
import bsam_b200 as B
from bsam_b200 import workloads as W
import torch

def solve(nd, precision):
    prob = W.config1(nsteps=1, n=128) if nd == 2 else W.config3(nsteps=1, n=32)
    with B.Solver(prob, precision=precision) as s:
        return s.step(), s.get_q()

forms = [(2, B.PREC_FP64), (2, B.PREC_MIXED), (3, B.PREC_FP64)]
want = [solve(*f) for f in forms]
names = glob.glob("/usr/local/cuda/lib64/libcudart.so*") + glob.glob(
    os.path.join(os.path.dirname(torch.__file__), "..", "nvidia", "*", "lib", "libcudart.so*"))
assert ctypes.CDLL(sorted(names)[0]).cudaDeviceReset() == 0
for f, w in zip(forms, want):
    got = solve(*f)
    assert got[0] == w[0] and np.array_equal(got[1], w[1]), f
print("equal after the reset")
"""


def test_handles_of_a_context_after_a_reset(gpu_lib):
    """The chain kernel's attributes go with the context: a new handle after
    cudaDeviceReset (of this process's own context) sets them anew."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", RESET, root], capture_output=True, text=True,
                       timeout=300)
    assert "equal after the reset" in r.stdout, r.stderr[-2000:]
