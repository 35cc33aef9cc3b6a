"""bsam_gpu_resid_norm_noalloc at the edges of a warp's piece (64 columns, 4 to 128
rows) and of the grid, against the oracle's Operator.  Tolerance: the sums have
at most 2e5 positive terms, each a few roundings off, added pairwise or in runs
of at most a few hundred: 1e-12 relative is far above what that can reach."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mx", [(1, 1), (31, 5), (32, 4), (33, 17), (2001, 37), (7, 4000),
                                (64, 1024), (1, 1, 1), (33, 5, 7), (19, 30, 120), (2, 17, 33)])
def test_norm_of_ragged_patches(gpu_lib, oracle, mx):
    import torch
    nd = len(mx)
    rng = np.random.default_rng(sum(mx))
    q = np.asfortranarray(0.5 + 0.1 * rng.standard_normal(tuple(m + 2 for m in mx) + (2,)))
    f = np.asfortranarray(0.01 * rng.standard_normal(tuple(mx) + (2,)))
    h, dt, eps, alpha = 1.0 / mx[0], 1e-4, 0.02, 1.0
    rf = f - oracle.operator(nd, mx, h, dt, alpha, eps, q)
    total = float(np.sum(rf * rf))
    qd = torch.from_numpy(q.ravel(order="F").copy()).cuda()
    fd = torch.from_numpy(f.ravel(order="F").copy()).cuda()
    m = (ctypes.c_int32 * 3)(*(list(mx) + [1] * (3 - nd)))
    stream = torch.cuda.current_stream()
    for _ in range(2):  # the second call finds the ticket the first one left
        out = torch.full((2,), -1.0, dtype=torch.float64, device="cuda")
        rc = gpu_lib.bsam_gpu_resid_norm_noalloc(
            torch.cuda.current_device(), nd, m, h, dt, eps, alpha,
            ctypes.c_void_p(qd.data_ptr()), ctypes.c_void_p(fd.data_ptr()),
            ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(stream.cuda_stream))
        assert rc == 0
        torch.cuda.synchronize()
        got = out.cpu().numpy()
        np.testing.assert_allclose(got[1], total, rtol=1e-12)
        np.testing.assert_allclose(got[0], np.sqrt(total / (2.0 * np.prod(mx))), rtol=1e-12)


def norm_call(lib, mx, q, f, out, stream):
    m = (ctypes.c_int32 * 3)(*(list(mx) + [1] * (3 - len(mx))))
    import torch
    return lib.bsam_gpu_resid_norm_noalloc(
        torch.cuda.current_device(), len(mx), m, 1.0 / mx[0], 1e-4, 0.02, 1.0,
        ctypes.c_void_p(q.data_ptr()), ctypes.c_void_p(f.data_ptr()),
        ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(stream.cuda_stream))


def fields(mx, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    ring = int(np.prod([m + 2 for m in mx]))
    q = 0.5 + 0.1 * torch.randn(2 * ring, generator=g, dtype=torch.float64, device="cuda")
    f = 0.01 * torch.randn(2 * int(np.prod(mx)), generator=g, dtype=torch.float64, device="cuda")
    return q, f


def test_overlapping_calls_spoil_no_later_one(gpu_lib):
    """Calls that overlap share the scratch and may be wrong themselves; what they
    leave in it must not reach a later call."""
    import torch
    sizes = [(64, 200), (500, 300)]
    data = [fields(mx, k) for k, mx in enumerate(sizes)]
    outs = [torch.zeros(2, dtype=torch.float64, device="cuda") for _ in sizes]
    main = torch.cuda.current_stream()
    want = []
    for mx, (q, f), out in zip(sizes, data, outs):
        assert norm_call(gpu_lib, mx, q, f, out, main) == 0
        torch.cuda.synchronize()
        want.append(out.cpu().numpy().copy())
    streams = [torch.cuda.Stream() for _ in sizes]
    for _ in range(50):
        for _ in range(4):
            for mx, (q, f), out, st in zip(sizes, data, outs, streams):
                assert norm_call(gpu_lib, mx, q, f, out, st) == 0
        torch.cuda.synchronize()
        for mx, (q, f), out, w in zip(sizes, data, outs, want):
            out.fill_(-1.0)
            assert norm_call(gpu_lib, mx, q, f, out, main) == 0
            torch.cuda.synchronize()
            assert np.array_equal(out.cpu().numpy(), w)


def test_captured_call_replays(gpu_lib):
    import torch
    mx = (500, 300)
    q, f = fields(mx, 5)
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    assert norm_call(gpu_lib, mx, q, f, out, torch.cuda.current_stream()) == 0
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        assert norm_call(gpu_lib, mx, q, f, out, torch.cuda.current_stream()) == 0
    for seed in (5, 6):
        a, b = fields(mx, seed)
        want = torch.zeros(2, dtype=torch.float64, device="cuda")
        assert norm_call(gpu_lib, mx, a, b, want, torch.cuda.current_stream()) == 0
        q.copy_(a)
        f.copy_(b)
        out.fill_(-1.0)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)


@pytest.mark.parametrize("mx", [(2, 2), (66, 6), (130, 34), (200, 72), (62, 1030), (512, 512),
                                (64, 512), (64, 514), (2048, 256), (2048, 258),
                                (2048, 1030), (6, 10, 4), (70, 10, 6), (128, 66, 34),
                                (200, 96, 64)])
def test_norm_is_the_solvers_bit_for_bit(gpu_lib, mx):
    """The same number as the final residual of a solve of these fields."""
    import torch

    import bsam_b200 as B
    from bsam_b200 import workloads as W
    nd = len(mx)
    rng = np.random.default_rng(sum(mx))
    h = 1.0 / mx[0]
    prob = W.Problem(ndims=nd, mx=tuple(mx) + (1,) * (3 - nd), eps=0.02, dt=1e-4, nsteps=1,
                     qerrortol=1e-12, maxvcycles=2,
                     xupper=tuple([n * h for n in mx] + [1.0] * (3 - nd)),
                     c0=0.5 + 0.1 * rng.uniform(-1, 1, int(np.prod(mx))))
    with B.Solver(prob) as s:
        _, res, _ = s.step()
        q, f, dx = s.get_q(), s.get_f(), s.patches[0].dx
    qd = torch.from_numpy(q.ravel(order="F").copy()).cuda()
    fd = torch.from_numpy(f.ravel(order="F").copy()).cuda()
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    m = (ctypes.c_int32 * 3)(*prob.mx)
    rc = gpu_lib.bsam_gpu_resid_norm_noalloc(
        torch.cuda.current_device(), nd, m, dx, prob.dt, prob.eps, prob.alpha,
        ctypes.c_void_p(qd.data_ptr()), ctypes.c_void_p(fd.data_ptr()),
        ctypes.c_void_p(out.data_ptr()),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    torch.cuda.synchronize()
    assert out.cpu().numpy()[0] == res
