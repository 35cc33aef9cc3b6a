"""What is timed: the solves, batches, refined hierarchies and residual norms
that a program asks of this library, each through the public entry points
(bsam_b200.Solver, bsam_b200.batch.Batch, bsam_b200.amr.AmrRun, the C ABI's
bsam_gpu_resid_norm_noalloc), from the smallest call to the largest.

Every solve starts from its own composition field c = mean + amp * U(-1, 1)
with the chemical potential that belongs to it, in host arrays as a program
holds them, and ends with the final fields back on the host.  `exact` is the same
scheme (FAS V-cycles with the red-black Newton smoother, to the same residual)
written with plain float64 tensor operations.
"""
import ctypes
import math

import numpy as np
import torch

import bsam_b200 as B
from bsam_b200 import amr
from bsam_b200 import batch as BB
from bsam_b200 import workloads as W

DT = 1e-4        # time step of the uniform workloads
ALPHA = 1.0
AMP = 0.025      # phi0 = 0.05 U(-1, 1), c = (1 + phi) / 2
MAXV = 20
# V-cycles that a time step needs at least in these workloads (the first step
# takes more); `work` counts no more than this.
VCYCLES = {"uniform": 4, "batch": 4, "amr": 7}
BATCH_SIDES = "64,96,128,192,256"


def listed():
    return [
        # The smallest solve: one time step of a 32^2 grid, as an interactive
        # program or a test issues it; launches and latency are all of it.
        {"name": "uniform2d_32_fp64", "kind": "uniform", "nx": 32, "ny": 32, "nz": 0,
         "faces": "neumann", "precision": "fp64", "eps": 0.02, "tol": 1e-9, "steps": 1},
        # The reference's example size: 128^2, V(2,2) to 1e-9.
        {"name": "uniform2d_128_fp64", "kind": "uniform", "nx": 128, "ny": 128, "nz": 0,
         "faces": "neumann", "precision": "fp64", "eps": 0.01, "tol": 1e-9, "steps": 10},
        # The shipped example's faces (periodic in x, user-coded in y) on a
        # domain that is not square and whose sides are no power of two.
        {"name": "uniform2d_320x200_periodic_fp64", "kind": "uniform", "nx": 320, "ny": 200,
         "nz": 0, "faces": "periodic_x", "precision": "fp64", "eps": 0.01, "tol": 1e-9,
         "steps": 5},
        # The largest served 2D side, alone, in the mixed form.
        {"name": "uniform2d_512_mixed", "kind": "uniform", "nx": 512, "ny": 512, "nz": 0,
         "faces": "neumann", "precision": "mixed", "eps": 0.01, "tol": 1e-8, "steps": 5},
        # The 3D configuration: 128^3 in FP64.
        {"name": "uniform3d_128_fp64", "kind": "uniform", "nx": 128, "ny": 128, "nz": 128,
         "faces": "neumann", "precision": "fp64", "eps": 0.02, "tol": 1e-8, "steps": 5},
        # A 3D channel, sides 96 x 64 x 80 (coarsest 6 x 4 x 5), every face
        # user-coded, mixed form.
        {"name": "uniform3d_96x64x80_user_mixed", "kind": "uniform", "nx": 96, "ny": 64,
         "nz": 80, "faces": "user", "precision": "mixed", "eps": 0.02, "tol": 1e-8, "steps": 5},
        # The batched workload of the benchmark: 512 problems of 64^2 .. 256^2,
        # ten steps each, mixed, host arrays in and out.
        {"name": "batch2d_512_mixed", "kind": "batch", "ndims": 2, "nprob": 512,
         "sides": BATCH_SIDES, "precision": "mixed", "tol": 1e-8, "steps": 10},
        # A parameter sweep in FP64: 96 of them.
        {"name": "batch2d_96_fp64", "kind": "batch", "ndims": 2, "nprob": 96,
         "sides": BATCH_SIDES, "precision": "fp64", "tol": 1e-8, "steps": 10},
        # Served 3D requests, 32^3 and 64^3, in one batch.
        {"name": "batch3d_24_mixed", "kind": "batch", "ndims": 3, "nprob": 24,
         "sides": "32,64", "precision": "mixed", "tol": 1e-8, "steps": 4},
        # The 2D AMR workload with sustained refinement as one request: a
        # 256^2 root, two refined levels regridded every step, statistics
        # every step, the state of every patch read back at the end.
        {"name": "amr2d_256", "kind": "amr", "root": 256, "nprob": 1, "steps": 8},
        # Eight such requests stepping in one batch.
        {"name": "amr2d_256_batch8", "kind": "amr", "root": 256, "nprob": 8, "steps": 6},
        # The residual norm of fields that a caller holds on the device, at
        # the largest patch the entry point takes.
        {"name": "residnorm_4096", "kind": "norm", "nx": 4096, "ny": 4096, "nz": 0},
    ]


def _log_even(rng, lo, hi):
    """An even size of [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, 2 * round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 2)))


def _log_multiple(rng, lo, hi, k):
    """A multiple of k in [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, k * round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / k)))


def draw(rng):
    kind = rng.choice(["uniform", "uniform", "uniform", "batch", "batch", "amr", "norm"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "uniform":
        # Sides that halve at least three times: the coarsest level of any
        # smaller multiple would be a grid of its own size.
        if rng.random() < 0.6:
            case = {"kind": kind, "nx": _log_multiple(rng, 32, 512, 8),
                    "ny": _log_multiple(rng, 32, 512, 8), "nz": 0, "tol": 1e-9}
            case["faces"] = rng.choice(["neumann", "user", "periodic_x"])
            n = case["nx"], case["ny"]
        else:
            case = {"kind": kind, "nx": _log_multiple(rng, 24, 128, 8),
                    "ny": _log_multiple(rng, 24, 128, 8), "nz": _log_multiple(rng, 24, 128, 8),
                    "tol": 1e-8}
            case["faces"] = rng.choice(["neumann", "user"])
            n = case["nx"], case["ny"], case["nz"]
        # Keep the coarsest level within what one CTA takes: the sides are
        # raised to multiples of 16 (2D: 32) where they are long.
        k = 32 if len(n) == 2 and max(n) > 256 else 16 if max(n) > 64 else 8
        for side in ("nx", "ny", "nz"):
            if case[side]:
                case[side] = k * max(1, round(case[side] / k))
        if case["faces"] == "periodic_x":  # even (or 1) on every level
            case["nx"] = 1 << max(5, min(9, round(math.log2(case["nx"]))))
        return {**case, "precision": precision, "eps": round(rng.uniform(0.008, 0.02), 4),
                "steps": rng.randint(1, 5)}
    if kind == "batch":
        if rng.random() < 0.7:
            sides = sorted({_log_multiple(rng, 48, 256, 16) for _ in range(4)})
            return {"kind": kind, "ndims": 2, "nprob": round(math.exp(rng.uniform(1.4, 5.0))),
                    "sides": ",".join(map(str, sides)), "precision": precision, "tol": 1e-8,
                    "steps": rng.randint(2, 8)}
        sides = sorted({_log_multiple(rng, 24, 64, 8) for _ in range(2)})
        return {"kind": kind, "ndims": 3, "nprob": rng.randint(3, 16),
                "sides": ",".join(map(str, sides)), "precision": precision, "tol": 1e-8,
                "steps": rng.randint(2, 4)}
    if kind == "amr":
        return {"kind": kind, "root": rng.choice([64, 96, 128, 160, 192, 256]),
                "nprob": rng.choice([1, 1, 2, 4]), "steps": rng.randint(2, 6)}
    if rng.random() < 0.5:
        return {"kind": kind, "nx": _log_even(rng, 32, 4000) + 1, "ny": _log_even(rng, 32, 4000),
                "nz": 0}
    return {"kind": kind, "nx": _log_even(rng, 16, 200) + 1, "ny": _log_even(rng, 16, 200),
            "nz": _log_even(rng, 16, 200)}


# ---- inputs --------------------------------------------------------------------
#
# Fields are tensors [problem, component, (z,) y, x] with a ghost ring, whose
# memory per problem is the library's q(0:mx+1, ..., 1:2) (x fastest).

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _generator(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed) % (1 << 62))
    return g


def _sizes(case):
    return [case["nx"], case["ny"]] + ([case["nz"]] if case["nz"] else [])


def _faces(case, nd):
    """Codes mthbc per face: 1 Neumann, 2 periodic, 10 the problem module's."""
    kind = case.get("faces", "neumann")
    if kind == "user":
        return [10] * (2 * nd)
    if kind == "periodic_x":
        return [2, 2] + [10] * (2 * nd - 2)
    return [1] * (2 * nd)


def _inner(a, d=None, shift=0):
    """The interior of a padded field, moved by `shift` along dimension d."""
    nd = a.dim() - 1
    ix = [slice(None)]
    for k in range(nd - 1, -1, -1):  # storage order z, y, x
        s = shift if k == d else 0
        ix.append(slice(1 + s, a.shape[nd - k] - 1 + s))
    return a[tuple(ix)]


def _fill(a, codes):
    """Ghosts of a padded field, face by face, x first."""
    nd = a.dim() - 1
    for d in range(nd):
        ax = nd - d
        n = a.shape[ax] - 2
        for side in (0, 1):
            code = codes[2 * d + side]
            ghost = a.select(ax, n + 1 if side else 0)
            if code == 2:
                ghost.copy_(a.select(ax, 1 if side else n))
                continue
            mirror = a.select(ax, n if side else 1)
            # The 2D module reflects about 1 on the x faces and copies on the
            # y faces; the 3D one reflects on every face.
            reflect = code != 1 and not (nd == 2 and d == 1)
            ghost.copy_(2.0 - mirror if reflect else mirror)
    return a


def _lap(a):
    nd = a.dim() - 1
    out = _inner(a, 0, 1) + _inner(a, 0, -1)
    for d in range(1, nd):
        out = out + _inner(a, d, 1)
        out = out + _inner(a, d, -1)
    return out - 2.0 * nd * _inner(a)


def _initial(sizes, nprob, mean, eps, h, gen):
    """[nprob, 2, (z,) y, x]: the composition and its chemical potential."""
    nd = len(sizes)
    shape = [nprob] + [n + 2 for n in reversed(sizes)]
    col = [nprob] + [1] * nd
    q = torch.zeros([nprob, 2] + shape[1:], dtype=torch.float64, device=_device())
    u = torch.rand([nprob] + list(reversed(sizes)), generator=gen, dtype=torch.float64,
                   device=_device())
    c, mu = q[:, 0], q[:, 1]
    _inner(c).copy_(mean.view(col) + AMP * (2.0 * u - 1.0))
    neumann = [1] * (2 * nd)
    _fill(c, neumann)
    ci = _inner(c)
    k = (eps * eps / (h * h)).view(col)
    _inner(mu).copy_(ALPHA * (ci - 0.5) ** 3 - ALPHA * (ci - 0.5) / 4.0 - k * _lap(c))
    _fill(mu, neumann)
    return q


def _uniform_fields(case, seed):
    sizes = _sizes(case)
    one = torch.ones(1, dtype=torch.float64, device=_device())
    h = 1.0 / case["nx"]
    return _initial(sizes, 1, 0.5 * one, case["eps"] * one, h, _generator(seed)), h


def _batch_plan(case, seed):
    """Per problem its side, eps and mean composition."""
    rng = np.random.default_rng(int(seed) + 77)
    sides = [int(s) for s in case["sides"].split(",")]
    n = case["nprob"]
    # Every side equally often, the largest first: batches of one case cost the
    # same whatever the seed.
    side = np.array([sides[-1 - i % len(sides)] for i in range(n)])
    rng.shuffle(side)
    return side, rng.uniform(0.005, 0.02, n), 0.5 + 0.5 * rng.uniform(-0.3, 0.3, n)


def _batch_groups(case, seed):
    """(problem indices, side, eps, initial fields) per side of a batch."""
    side, eps, mean = _batch_plan(case, seed)
    gen = _generator(seed)
    for s in sorted(set(side.tolist())):
        at = np.flatnonzero(side == s)
        e = torch.tensor(eps[at], dtype=torch.float64, device=_device())
        m = torch.tensor(mean[at], dtype=torch.float64, device=_device())
        yield at, s, e, _initial([s] * case["ndims"], len(at), m, e, 1.0 / s, gen)


def _precision(case):
    return B.PREC_MIXED if case["precision"] == "mixed" else B.PREC_FP64


class _State:
    """What a program keeps between passes; closes its handles when dropped."""

    def __init__(self, case):
        self.case = case
        self.handles = []

    def __del__(self):
        for h in reversed(self.handles):
            h.close()


def prepare(case, seed):
    s = _State(case)
    if case["kind"] == "uniform":
        sizes = _sizes(case)
        nd = len(sizes)
        q, h = _uniform_fields(case, seed)
        mx = tuple(sizes + [1] * (3 - nd))
        s.prob = W.Problem(ndims=nd, mx=mx, eps=case["eps"], dt=DT, nsteps=case["steps"],
                           qerrortol=case["tol"], alpha=ALPHA, maxvcycles=MAXV,
                           mthbc=tuple(_faces(case, nd) + [1] * (6 - 2 * nd)),
                           xupper=tuple([n * h for n in sizes] + [1.0] * (3 - nd)))
        s.q0 = q[0].cpu().numpy().transpose()
        s.q = np.empty_like(s.q0)
        s.solver = B.Solver(s.prob, precision=_precision(case), q0=s.q0)
        s.handles.append(s.solver)
    elif case["kind"] == "batch":
        nd, n = case["ndims"], case["nprob"]
        side, eps, _ = _batch_plan(case, seed)
        first = np.zeros(n + 1, dtype=np.int64)
        first[1:] = np.cumsum(2 * (side + 2) ** nd)
        q0, s.q = (torch.empty(int(first[-1]), dtype=torch.float64, pin_memory=True)
                   for _ in range(2))
        views = [[a.numpy()[first[k]:first[k + 1]].reshape((side[k] + 2,) * nd + (2,), order="F")
                  for k in range(n)] for a in (q0, s.q)]
        s.q0s, s.outs = views
        for at, _, _, q in _batch_groups(case, seed):
            for j, k in enumerate(at):
                q0[first[k]:first[k + 1]].copy_(q[j].reshape(-1))
        s.probs = [W.Problem(ndims=nd, mx=tuple([int(side[k])] * nd + [1] * (3 - nd)),
                             eps=float(eps[k]), dt=DT, nsteps=case["steps"],
                             qerrortol=case["tol"], alpha=ALPHA) for k in range(n)]
        cells = int(np.sum(side ** nd))
        s.batch = BB.Batch(nd, precision=_precision(case), max_slots=n, qerrortol=case["tol"],
                           maxvcycles=MAXV, pool_bytes=cells * 224 + n * (1 << 20) + (64 << 20))
        s.handles.append(s.batch)
    elif case["kind"] == "amr":
        n = case["root"]
        eps = 0.005 * 256 / n
        s.starts = []
        for k in range(case["nprob"]):
            hier = amr.build(n, [], eps=eps, dt=5e-5, qerrortol=1e-9, field="drop",
                             seed=int(seed) % 100003 + 31 * k)
            # The sustained tag threshold |grad phi| > 0.25 / eps.
            prm = amr.RegridParams(maxlevel=2, ibuffer=[1, 1], desfill=[0.9, 0.9], mgp=[8, 8],
                                   qtolerance=[0.25 / (n * eps), 0.25 / (2 * n * eps)])
            s.starts.append((hier, prm))
        # The program's frame: the patches' fields one after another and the
        # grids' index boxes, with room for any hierarchy of the workload
        # (zeros after the last patch).
        s.frame = np.zeros(12 * n * n * case["nprob"])
        s.grids = np.zeros((256 * case["nprob"], 6), dtype=np.int32)
        if case["nprob"] > 1:
            s.batch = BB.Batch(2, precision=B.PREC_FP64, max_slots=case["nprob"],
                               qerrortol=1e-9, maxvcycles=MAXV, pool_bytes=1 << 20)
            s.handles.append(s.batch)
    else:
        sizes = _sizes(case)
        q, f, h = _norm_fields(case, seed)
        s.q, s.f = q.reshape(-1).contiguous(), f.reshape(-1).contiguous()
        s.mx = (ctypes.c_int32 * 3)(*(sizes + [1] * (3 - len(sizes))))
        s.nd, s.h = len(sizes), h
        s.out = torch.empty(2, dtype=torch.float64, device="cuda")
    return s


def _norm_fields(case, seed):
    sizes = _sizes(case)
    gen = _generator(seed)
    one = torch.ones(1, dtype=torch.float64, device=_device())
    h = 1.0 / case["nx"]
    q = _initial(sizes, 1, 0.5 * one, 0.02 * one, h, gen)
    f = 0.01 * (2.0 * torch.rand([2] + list(reversed(sizes)), generator=gen, dtype=torch.float64,
                                 device=_device()) - 1.0)
    return q[0], f, h


# ---- one pass --------------------------------------------------------------------

def run(s):
    case = s.case
    if case["kind"] == "uniform":
        s.solver.put_q(s.q0)
        r = s.solver.run(case["steps"], keep_steps=False)
        s.solver.get_q_into(s.q)
        return {"q": s.q, "nvcycles": r["nvcycles"], "residual": r["residual"],
                "mass": r["mass"]}
    if case["kind"] == "batch":
        slots = s.batch.submit_many(s.probs, q0s=s.q0s)
        s.batch.run()
        got = s.batch.collect_many(slots, outs=s.outs)
        return {"q": s.q, "nvcycles": np.concatenate([g["nvcycles"] for g in got]),
                "residual": np.concatenate([g["residual"] for g in got])}
    if case["kind"] == "amr":
        return _run_amr(s)
    rc = B.lib().bsam_gpu_resid_norm_noalloc(
        torch.cuda.current_device(), s.nd, s.mx, s.h, DT, 0.02, ALPHA,
        ctypes.c_void_p(s.q.data_ptr()), ctypes.c_void_p(s.f.data_ptr()),
        ctypes.c_void_p(s.out.data_ptr()),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    if rc:
        raise RuntimeError(f"bsam_gpu_resid_norm_noalloc failed ({rc})")
    return s.out


def _run_amr(s):
    # A request's driver lives as long as the request (amr.solve_request).
    steps, runs = s.case["steps"], []
    try:
        for hier, prm in s.starts:
            runs.append(amr.AmrRun(hier, prm))
        if len(runs) == 1:
            nv, res, stats = [], [], []
            for _ in range(steps):
                a, r = runs[0].step()
                nv.append(a)
                res.append(r)
                stats.append(runs[0].stats())
        else:
            slots = [s.batch.submit_amr(r, steps) for r in runs]
            s.batch.run()
            got = [s.batch.collect_amr(k) for k in slots]
            nv = np.concatenate([g["nvcycles"] for g in got])
            res = np.concatenate([g["residual"] for g in got])
            stats = [r.stats() for r in runs]
        at = 0
        for r in runs:
            for _, a in r.state():
                s.frame[at:at + a.size] = a.ravel(order="F")
                at += a.size
        s.frame[at:] = 0.0
        boxes = np.concatenate([t["mglobal"].reshape(len(t), 6)
                                for t in (r.table_array() for r in runs)])
        s.grids[:len(boxes)] = boxes
        s.grids[len(boxes):] = 0
        return {"q": s.frame, "nvcycles": np.asarray(nv), "residual": np.asarray(res),
                "stats": np.asarray(stats, dtype=np.float64), "grids": s.grids}
    finally:
        for r in runs:
            r.close()


# ---- what a pass cannot do without -----------------------------------------------

def _vcycle_work(cells, nd, mixed):
    """Bytes and operations of one V-cycle whose finest level has `cells`: a
    level's state and right-hand side pass by twice (before and after the
    coarser levels), each time with the state written back; the mixed form
    keeps its coarser levels in 32 bits (state, right-hand side and base) and
    updates a 64-bit state against a 64-bit right-hand side once.  A cell is
    relaxed eight times (4 sweeps of 2 colours update it 4 times) and takes
    part in two residuals, a restriction and a correction."""
    levels = 1.0 / (1.0 - 0.5 ** nd)
    if mixed:
        nbytes = cells * ((2 * 4 * 5 + 2 * 8) * levels + 16 + 32 + 12)
    else:
        nbytes = cells * 2 * (32 + 16) * levels
    relax = 20 + 4 * 2 * nd
    return nbytes, cells * levels * (4 * relax + 2 * (12 + 8 * nd) + 30)


def work(case):
    if case["kind"] == "norm":
        nd, cells = len(_sizes(case)), math.prod(_sizes(case))
        ring = math.prod(n + 2 for n in _sizes(case))
        return {"bytes": 16 * ring + 16 * cells, "flops": cells * (14 + 8 * nd)}
    if case["kind"] == "uniform":
        nd, cells = len(_sizes(case)), math.prod(_sizes(case))
        ring = math.prod(n + 2 for n in _sizes(case))
        steps = case["steps"] * VCYCLES["uniform"]
        mixed = case["precision"] == "mixed"
    elif case["kind"] == "batch":
        nd = case["ndims"]
        side = _batch_plan(case, 0)[0]
        cells, ring = int(np.sum(side ** nd)), int(np.sum((side + 2) ** nd))
        steps = case["steps"] * VCYCLES["batch"]
        mixed = case["precision"] == "mixed"
    else:
        # The refined levels follow the interface: about 40 + 100 patches on a
        # 256^2 root, together about as many cells as the root.
        nd, mixed = 2, False
        cells = ring = case["nprob"] * 2 * case["root"] ** 2
        steps = case["steps"] * VCYCLES["amr"]
    nbytes, flops = _vcycle_work(cells, nd, mixed)
    return {"bytes": int(steps * nbytes + 2 * 16 * ring), "flops": int(steps * flops)}


# ---- the scheme in plain float64 ---------------------------------------------------

class _Level:
    def __init__(self, sizes, h, eps, codes, nprob):
        self.nd = nd = len(sizes)
        self.codes = codes
        col = [nprob] + [1] * nd
        self.t1 = DT / (h * h)
        self.t2 = (eps * eps / (h * h)).view(col)
        idx = torch.zeros([1] * nd, dtype=torch.int64, device=_device())
        for d, n in enumerate(sizes):
            v = [1] * nd
            v[nd - 1 - d] = n
            idx = idx + torch.arange(1, n + 1, device=_device()).view(v)
        self.red = (idx % 2 == 0).unsqueeze(0)

    def take(self, at):
        o = object.__new__(_Level)
        o.__dict__.update(self.__dict__)
        o.t2 = self.t2[at]
        return o

    def relax(self, q, f):
        nd = self.nd
        for sweep in range(4):
            mask = self.red if sweep % 2 == 0 else ~self.red
            p, m = q
            pc = _inner(p)
            sp = _lap(p) + 2.0 * nd * pc
            sm = _lap(m) + 2.0 * nd * _inner(m)
            d2 = 3.0 * ALPHA * (pc - 0.5) ** 2
            a12 = 2.0 * nd * self.t1
            a21 = -d2 - 2.0 * nd * self.t2
            b1 = f[0] + self.t1 * sm
            b2 = f[1] + ALPHA * (pc - 0.5) ** 3 - d2 * pc - self.t2 * sp
            det = 1.0 - a12 * a21
            new = (b1 - a12 * b2) / det, (b2 - a21 * b1) / det
            for a, v in zip(q, new):
                i = _inner(a)
                i.copy_(torch.where(mask, v, i))
                _fill(a, self.codes)

    def operator(self, q):
        p, m = q
        pc = _inner(p)
        return (pc - self.t1 * _lap(m),
                _inner(m) - ALPHA * (pc - 0.5) ** 3 + self.t2 * _lap(p))

    def residual(self, q, f):
        o = self.operator(q)
        return f[0] - o[0], f[1] - o[1]


def _restrict(a):
    nd = a.dim() - 1
    for ax in range(1, nd + 1):
        n = a.shape[ax] // 2
        a = 0.5 * (a.unflatten(ax, (n, 2)).select(ax + 1, 0) +
                   a.unflatten(ax, (n, 2)).select(ax + 1, 1))
    return a


def _prolong(e):
    """Linear prolongation of a padded coarse field to the fine interior."""
    nd = e.dim() - 1
    for ax in range(1, nd + 1):
        n = e.shape[ax]
        lo, hi = e.narrow(ax, 0, n - 1), e.narrow(ax, 1, n - 1)
        # fine 2m takes (3 e(m) + e(m+1)) / 4, fine 2m + 1 takes (e(m) + 3 e(m+1)) / 4
        both = torch.stack(((3.0 * lo + hi) / 4.0, (lo + 3.0 * hi) / 4.0), dim=ax + 1)
        e = both.flatten(ax, ax + 1).narrow(ax, 1, 2 * (n - 2))
    return e


def _vcycle(levels, l, q, f):
    lv = levels[l]
    lv.relax(q, f)
    if l + 1 == len(levels):
        return
    up = levels[l + 1]
    cq, snap, cf = [], [], []
    for a in q:
        r = _restrict(_inner(a))
        c = torch.zeros([r.shape[0]] + [n + 2 for n in r.shape[1:]], dtype=r.dtype,
                        device=r.device)
        _inner(c).copy_(r)
        cq.append(_fill(c, lv.codes))
        snap.append(c.clone())
    for r, o in zip(lv.residual(q, f), up.operator(snap)):
        cf.append(_restrict(r) + o)
    _vcycle(levels, l + 1, cq, cf)
    for a, c, s0 in zip(q, cq, snap):
        i = _inner(a)
        i.copy_(i + _prolong(c - s0))
        _fill(a, lv.codes)
    lv.relax(q, f)


def _solve(sizes, h, eps, codes, q, steps, tol):
    """`steps` time steps of every problem of q, in place; (V-cycles, residuals)."""
    nprob, nd = q.shape[0], len(sizes)
    levels, s, hl = [], list(sizes), h
    while True:
        levels.append(_Level(s, hl, eps, codes, nprob))
        if any(n % 2 for n in s) or len(levels) == 11:
            break
        s, hl = [n // 2 for n in s], 2.0 * hl
    nv = np.zeros((nprob, steps), dtype=np.int32)
    res = np.zeros((nprob, steps))
    denom = 2.0 * math.prod(sizes)
    fields = q[:, 0], q[:, 1]
    for step in range(steps):
        for a in fields:
            _fill(a, codes)
        old = _inner(fields[0]).clone()
        f = old, -(old - 0.5) * ALPHA / 4.0
        at = np.arange(nprob)
        for it in range(1, MAXV + 1):
            t = torch.as_tensor(at, device=q.device)
            lv = [l.take(t) for l in levels]
            sub = [a[t].clone() for a in fields]
            fs = [a[t] for a in f]
            _vcycle(lv, 0, sub, fs)
            for a, b in zip(fields, sub):
                a[t] = b
            r = lv[0].residual(sub, fs)
            dims = tuple(range(1, nd + 1))
            norm = ((r[0] ** 2).sum(dims) + (r[1] ** 2).sum(dims)).div(denom).sqrt()
            norm = norm.cpu().numpy()
            nv[at, step], res[at, step] = it, norm
            at = at[norm >= tol]
            if not len(at):
                break
    return nv, res


def exact(case, seed):
    if case["kind"] == "norm":
        q, f, h = _norm_fields(case, seed)
        nd = len(_sizes(case))
        lv = _Level(_sizes(case), h, 0.02 * torch.ones(1, dtype=torch.float64, device=_device()),
                    None, 1)
        r = lv.residual([q[0:1], q[1:2]], [f[0:1], f[1:2]])
        total = (r[0] ** 2).sum() + (r[1] ** 2).sum()
        return torch.stack((torch.sqrt(total / (2.0 * math.prod(_sizes(case)))), total))
    if case["kind"] == "uniform":
        sizes = _sizes(case)
        nd = len(sizes)
        q, h = _uniform_fields(case, seed)
        eps = case["eps"] * torch.ones(1, dtype=torch.float64, device=_device())
        codes = _faces(case, nd)
        masses = []
        nv, res = np.zeros(case["steps"], dtype=np.int32), np.zeros(case["steps"])
        for step in range(case["steps"]):
            a, b = _solve(sizes, h, eps, codes, q, 1, case["tol"])
            nv[step], res[step] = a[0, 0], b[0, 0]
            masses.append(float(_inner(q[:, 0]).sum()) * h ** nd)
        fp64 = case["precision"] == "fp64"
        return {"q": q[0].permute(*range(nd, -1, -1)), "nvcycles": nv if fp64 else None,
                "residual": res if fp64 else None, "mass": np.asarray(masses)}
    if case["kind"] == "batch":
        nd, n = case["ndims"], case["nprob"]
        side = _batch_plan(case, seed)[0]
        first = np.zeros(n + 1, dtype=np.int64)
        first[1:] = np.cumsum(2 * (side + 2) ** nd)
        out = torch.empty(int(first[-1]), dtype=torch.float64)
        nv = np.zeros((n, case["steps"]), dtype=np.int32)
        res = np.zeros((n, case["steps"]))
        for at, sd, eps, q in _batch_groups(case, seed):
            nv[at], res[at] = _solve([sd] * nd, 1.0 / sd, eps, [1] * (2 * nd), q,
                                     case["steps"], case["tol"])
            for j, k in enumerate(at):
                out[first[k]:first[k + 1]].copy_(q[j].reshape(-1))
        fp64 = case["precision"] == "fp64"
        return {"q": out, "nvcycles": nv.ravel() if fp64 else None,
                "residual": res.ravel() if fp64 else None}
    return None  # a refined hierarchy, regridded every step
