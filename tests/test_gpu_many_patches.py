"""SetBC of more root patches than a launch's grid has rows (65535)."""
import ctypes

import numpy as np
import pytest

import bsam_b200 as B

pytestmark = pytest.mark.gpu


def test_set_ghost_of_70000_roots(gpu_lib):
    npatch = 70000
    L = gpu_lib
    rp = B.RunParams(ndims=2, nrvars=2, mbc=1, maux=0, nsmoothingpasses=2, maxvcycles=2,
                     errortype=1, precision=B.PREC_FP64, dt=1e-4, qerrortol=1e-9, alpha=1.0,
                     eps=0.02)
    h = ctypes.c_void_p()
    assert L.bsam_gpu_create(ctypes.byref(h), 0, ctypes.byref(rp)) == 0
    try:
        arr = (B.PatchDesc * npatch)()
        for d in arr:
            d.level, d.parent, d.dx = 0, -1, 0.5
            for n in range(3):
                d.mx[n] = 2 if n < 2 else 1
                for k in range(2):
                    d.mbounds[n][k] = d.mglobal[n][k] = 1 + k * (d.mx[n] - 1)
            for f in range(6):
                d.mthbc[f] = 1
        assert L.bsam_gpu_set_hierarchy(h, npatch, arr, 0) == 0, L.bsam_gpu_last_error(h)
        rng = np.random.default_rng(1)
        dp = ctypes.POINTER(ctypes.c_double)
        for p in (0, 65534, 65535, npatch - 1):
            q = np.asfortranarray(rng.standard_normal((4, 4, 2)))
            out = np.zeros_like(q, order="F")
            assert L.bsam_gpu_put_field(h, p, B.FIELD_Q, q.ctypes.data_as(dp)) == 0
            assert L.bsam_gpu_set_ghost(h) == 0
            assert L.bsam_gpu_get_field(h, p, B.FIELD_Q, out.ctypes.data_as(dp)) == 0
            want = np.pad(q[1:-1, 1:-1], ((1, 1), (1, 1), (0, 0)), mode="edge")
            assert np.array_equal(out, want)
    finally:
        L.bsam_gpu_destroy(h)
