"""List kernels of a batch (colour passes, restriction, coarse load, correction by
blocks, defect and residual by warps, bottom chains) at extents where their tiles
can go wrong -- rows of one pair, of a few cells, just over 8, 16, 32 and 64, and
planes that end inside a tile -- against the single-problem library, whose coarse
levels are those of k_chain: every value the same bit for bit, 2D and 3D, FP64
and mixed, each face rule, with nearly every level in the lists (bottom chains of
64 cells at most) and with the default bottom chains."""
import numpy as np
import pytest

import bsam_b200 as B
from bsam_b200 import batch as BB
from bsam_b200 import workloads as W

pytestmark = pytest.mark.gpu

SIZES = {2: [(2, 2), (6, 10), (24, 40), (24, 72), (40, 24), (136, 4), (4, 132), (8, 200),
             (80, 144)],
         3: [(2, 2, 2), (6, 10, 4), (10, 6, 8), (20, 36, 4), (36, 20, 4), (68, 4, 4),
             (4, 4, 68), (24, 24, 24), (40, 24, 8)]}
FACES = {"neumann": 1, "user": 10}


def problem(mx, faces):
    nd = len(mx)
    h = 1.0 / max(mx)
    rng = np.random.default_rng(int(np.prod(mx)))
    code = [FACES[faces]] * (2 * nd)
    return W.Problem(ndims=nd, mx=tuple(mx) + (1,) * (3 - nd), eps=0.02, dt=1e-4, nsteps=2,
                     qerrortol=1e-12, maxvcycles=3, mthbc=tuple(code) + (1,) * (6 - 2 * nd),
                     xupper=tuple([n * h for n in mx] + [1.0] * (3 - nd)),
                     c0=0.5 + 0.1 * rng.uniform(-1, 1, int(np.prod(mx))))


def batch(probs, precision, bottom_cells, per_pass):
    with BB.Batch(probs[0].ndims, precision=precision, max_slots=len(probs),
                  qerrortol=probs[0].qerrortol, maxvcycles=probs[0].maxvcycles,
                  bottom_cells=bottom_cells) as b:
        if per_pass:
            b.set_tuning(per_pass=1)
        slots = [b.submit(p) for p in probs]
        b.run()
        return [b.collect(s) for s in slots]


@pytest.mark.parametrize("precision", [BB.PREC_FP64, BB.PREC_MIXED])
@pytest.mark.parametrize("faces", sorted(FACES))
@pytest.mark.parametrize("cells", [64, 0])
@pytest.mark.parametrize("nd", [2, 3])
def test_batch_equals_single_solves(gpu_lib, nd, cells, faces, precision):
    probs = [problem(mx, faces) for mx in SIZES[nd]]
    want = []
    for p in probs:
        with B.Solver(p, precision=precision, bottom_cells=cells or BB.BOTTOM_CELLS) as s:
            want.append(s.run(p.nsteps))
    for per_pass in ((0, 1) if nd == 2 else (0,)):
        for p, g, w in zip(probs, batch(probs, precision, cells, per_pass), want):
            assert np.array_equal(g["q"], w["q"][-1]), p.mx
            assert np.array_equal(g["nvcycles"], w["nvcycles"]), p.mx
            assert np.array_equal(g["residual"], w["residual"]), p.mx
