"""bsam_gpu_profile times every finest-level smoothing stage, two a V-cycle, also where
the finest level runs in the chain kernel when it is not timed; the solve is the same
bit for bit."""
import numpy as np
import pytest

import bsam_b200 as B
from bsam_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [B.PREC_FP64, B.PREC_MIXED])
@pytest.mark.parametrize("mx", [(32, 32), (128, 128), (160, 96), (256, 192), (16, 16, 16),
                                (32, 24, 40)])
def test_stages_are_timed(gpu_lib, mx, precision):
    nd = len(mx)
    h = 1.0 / mx[0]
    rng = np.random.default_rng(sum(mx))
    prob = W.Problem(ndims=nd, mx=tuple(mx) + (1,) * (3 - nd), eps=0.02, dt=1e-4, nsteps=2,
                     qerrortol=1e-9, xupper=tuple([n * h for n in mx] + [1.0] * (3 - nd)),
                     c0=0.5 + 0.1 * rng.uniform(-1, 1, int(np.prod(mx))))
    out = []
    for timed in (False, True):
        with B.Solver(prob, precision=precision) as s:
            if timed:
                s.profile(True)
            steps = [s.step() for _ in range(prob.nsteps)]
            if timed:
                st = s.stats()
                s.profile(False)
            steps.append(s.step())
            out.append((steps, s.get_q()))
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1])
    stages = 2 * sum(nv for nv, _, _ in out[1][0][:prob.nsteps])
    assert st["smooth_stages"] == stages
    assert st["smooth_cells"] == stages * int(np.prod(mx))
    assert st["smooth_ms"] > 0.0 and st["smooth_bytes"] > 0.0
