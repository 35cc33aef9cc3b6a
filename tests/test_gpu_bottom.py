"""A batch's bottom chains beyond the default size, against single solves of the same
levels (bit for bit): chains that do not fit a CTA's shared memory and run in global
memory (kb_bottom), chains just below that size, both kinds in one batch, and a larger
chain admitted while the batch's graph is already running."""
import dataclasses

import numpy as np
import pytest

import bsam_b200 as B
from bsam_b200 import batch as BB
from bsam_b200 import workloads as W

pytestmark = pytest.mark.gpu


def problem(mx, code, nsteps=2):
    nd = len(mx)
    h = 1.0 / max(mx)
    rng = np.random.default_rng(int(np.prod(mx)) + code)
    return W.Problem(ndims=nd, mx=tuple(mx) + (1,) * (3 - nd), eps=0.02, dt=1e-4, nsteps=nsteps,
                     qerrortol=1e-12, maxvcycles=4, mthbc=(code,) * (2 * nd) + (1,) * (6 - 2 * nd),
                     xupper=tuple([n * h for n in mx] + [1.0] * (3 - nd)),
                     c0=0.5 + 0.1 * rng.uniform(-1, 1, int(np.prod(mx))))


def singles(probs, precision, cells):
    out = []
    for p in probs:
        with B.Solver(p, precision=precision, bottom_cells=cells) as s:
            out.append(s.run(p.nsteps))
    return out


def same(got, want, prob):
    assert np.array_equal(got["q"], want["q"][-1]), prob.mx
    assert np.array_equal(got["nvcycles"], want["nvcycles"]), prob.mx
    assert np.array_equal(got["residual"], want["residual"]), prob.mx


# 64^2 FP64 takes 209 KB and its mixed form 259; 16^3 234 and 283.
SIZES = {2: [(64, 64), (128, 128), (192, 64), (32, 32), (4, 1024), (8, 8)],
         3: [(16, 16, 16), (32, 32, 32), (12, 20, 16), (8, 8, 8), (4, 4, 64)]}


@pytest.mark.parametrize("precision", [BB.PREC_FP64, BB.PREC_MIXED])
@pytest.mark.parametrize("code", [1, 10])
@pytest.mark.parametrize("cells", [2048, 4096])
@pytest.mark.parametrize("nd", [2, 3])
def test_large_bottom_chains(gpu_lib, nd, cells, code, precision):
    probs = [problem(mx, code) for mx in SIZES[nd]]
    want = singles(probs, precision, cells)
    with BB.Batch(nd, precision=precision, max_slots=len(probs), qerrortol=probs[0].qerrortol,
                  maxvcycles=probs[0].maxvcycles, bottom_cells=cells) as b:
        slots = [b.submit(p) for p in probs]
        b.run()
        for p, s, w in zip(probs, slots, want):
            same(b.collect(s), w, p)


@pytest.mark.parametrize("precision", [BB.PREC_FP64, BB.PREC_MIXED])
@pytest.mark.parametrize("nd", [2, 3])
def test_a_larger_chain_joins_a_running_batch(gpu_lib, nd, precision):
    sizes = {2: [(8, 8), (32, 32), (64, 48), (64, 64)],
             3: [(4, 4, 4), (8, 8, 8), (12, 20, 16), (16, 16, 16)]}[nd]
    probs = [problem(mx, 1, nsteps=6) for mx in sizes]
    want = singles(probs, precision, 4096)
    with BB.Batch(nd, precision=precision, max_slots=len(probs), qerrortol=probs[0].qerrortol,
                  maxvcycles=probs[0].maxvcycles, bottom_cells=4096) as b:
        slots = []
        for p in probs:
            slots.append(b.submit(p))
            b.advance(3)
        b.run()
        for p, s, w in zip(probs, slots, want):
            same(b.collect(s), w, p)


@pytest.mark.parametrize("precision", [B.PREC_FP64, B.PREC_MIXED])
@pytest.mark.parametrize("sweeps", [1, 3])
@pytest.mark.parametrize("mx", [(32, 32), (128, 128), (200, 40), (320, 200), (16, 16, 16),
                                (32, 32, 32)])
def test_other_sweep_counts(gpu_lib, mx, sweeps, precision):
    """The chain kernel and the mixed 2D stages at one and three sweeps, against one
    launch per pass."""
    prob = dataclasses.replace(problem(mx, 10), nsmoothingpasses=sweeps)
    out = []
    for cells in (-1, 0):
        with B.Solver(prob, precision=precision, bottom_cells=cells) as s:
            out.append(([s.step() for _ in range(2)], s.trace(), s.get_q()))
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1])
    assert np.array_equal(out[0][2], out[1][2])
