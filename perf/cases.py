"""Performance cases of the preconditioned-solve path, through its public entry points.

Each case is one call (or the short sequence of calls) that a program built on
the package makes again and again with its matrix, factors and workspace
resident: an SpMV, an application of the preconditioner, a refactorisation
with new values, a whole solve, a solve with its adjoint, a block solve, the
LACE-named calls on host buffers, a batch of small systems.  The matrices are
the package's own workloads (5-point Laplacians, the upwind convection-
diffusion operator, the 5x5 block stencil, the anisotropic batch), from a few
thousand rows, where launches and latency count, to two million, where
memory traffic does.

`exact` recomputes each result with torch in FP64 (stencil arithmetic,
hyperplane substitution, BiCGSTAB to FP64 accuracy, fast diagonalisation),
without the package.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import lace_gb300 as lg
from lace_gb300 import problems

DEV = "cuda"
VSIZE = {"fp64": 8, "fp32": 4, "bf16": 2}


# ------------------------------------------------------------------- cases

def listed():
    return [
        # the residual of a small system inside someone else's iteration: launch latency
        dict(name="residual_laplace64", kind="spmv", op="laplace", nx=64, ny=64, nz=1, residual=True),
        # the SpMV of the headline operator: memory traffic
        dict(name="spmv_conv128", kind="spmv", op="conv", nx=128, ny=128, nz=128, residual=False),
        # M^-1 q with FP32 factors, as a mixed-precision outer method applies it
        dict(name="precond_fp32_conv128", kind="precond", nx=128, ny=128, nz=128, prec="fp32", sweeps=3),
        # M^-1 q in FP64 (the default precision) on a grid with odd sides
        dict(name="precond_fp64_93x70x51", kind="precond", nx=93, ny=70, nz=51, prec="fp64", sweeps=3),
        # a time step or Newton step: new values on the same pattern, factors again, first application
        dict(name="refactor_fp32_conv96", kind="refactor", nx=96, ny=96, nz=96, prec="fp32", sweeps=3),
        # the headline solve, factorisation included
        dict(name="solve_fp32_conv128", kind="solve", op="conv", nx=128, ny=128, nz=128, prec="fp32", sweeps=3,
             orth="householder", m=50, rtol=1e-10, order="natural"),
        # a small elliptic solve with LACE's default Gram-Schmidt method: launch and barrier latency
        dict(name="solve_mgs_laplace64", kind="solve", op="laplace", nx=64, ny=64, nz=1, prec="fp32", sweeps=5,
             orth="mgs", m=30, rtol=1e-12, order="natural"),
        # a system numbered by a Cuthill-McKee level ordering instead of grid lines
        dict(name="solve_fp32_levels48", kind="solve", op="conv", nx=48, ny=48, nz=48, prec="fp32", sweeps=3,
             orth="householder", m=30, rtol=1e-10, order="levels"),
        # a training step through the solver: forward solve, loss gradient, adjoint solve, dL/db and dL/dA
        dict(name="adjoint_fp32_conv64", kind="adjoint", nx=64, ny=64, nz=64, prec="fp32", sweeps=3, m=50,
             rtol=1e-10),
        # a coupled (block) system: block ParILU and solve
        dict(name="block_fp32_32", kind="block", nx=32, ny=32, nz=32, prec="fp32", sweeps=3, m=30, rtol=1e-10),
        # a LACE program's calls on host buffers, all FP64 (the library's default precision)
        dict(name="dropin_fp64_99x83x41", kind="dropin", nx=99, ny=83, nz=41, prec="fp64", sweeps=3, m=30,
             rtol=1e-10),
        # many small independent systems, several right-hand sides each, in one call
        dict(name="batch_fp32_24", kind="batch", count=24, lo=32, hi=96, nrhs=4, shape=11, prec="fp32", sweeps=3,
             m=30, rtol=1e-12),
    ]


def _sides(rng, lo, hi):
    """Three grid sides whose product is log-uniform in [lo, hi] rows, none the others' multiple on purpose."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    ax, ay = rng.uniform(0.75, 1.3), rng.uniform(0.75, 1.3)
    s = n ** (1.0 / 3.0)
    nx, ny = max(4, round(s * ax)), max(4, round(s * ay))
    return nx, ny, max(3, round(n / (nx * ny)))


def draw(rng):
    kind = rng.choice(["spmv", "precond", "refactor", "solve", "adjoint", "block", "dropin", "batch"])
    prec = rng.choice(["fp32", "fp32", "fp64", "bf16"])
    if kind == "spmv":
        if rng.random() < 0.5:
            s = round(math.exp(rng.uniform(math.log(48), math.log(1024))))
            return dict(kind=kind, op="laplace", nx=s, ny=s + rng.randint(0, 9), nz=1, residual=rng.random() < 0.5)
        nx, ny, nz = _sides(rng, 6000, 1.8e6)
        return dict(kind=kind, op="conv", nx=nx, ny=ny, nz=nz, residual=rng.random() < 0.5)
    if kind in ("precond", "refactor"):
        nx, ny, nz = _sides(rng, 15000, 1.6e6)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, prec=prec, sweeps=rng.choice([1, 3, 5]))
    if kind == "solve":
        order, orth = rng.choice(["natural", "natural", "levels"]), rng.choice(["householder", "mgs"])
        if rng.random() < 0.3:
            s = rng.randint(40, 110)
            return dict(kind=kind, op="laplace", nx=s, ny=s + rng.randint(0, 9), nz=1, prec=prec, sweeps=5,
                        orth=orth, m=30, rtol=1e-12, order=order)
        nx, ny, nz = _sides(rng, 12000, 3e5)
        if order == "natural" and rng.random() < 0.4:  # grids as people choose them, to the largest
            nx, ny, nz = rng.choice([32, 64, 96, 128]), rng.choice([32, 64, 96, 128]), rng.choice([32, 48, 64, 100])
        return dict(kind=kind, op="conv", nx=nx, ny=ny, nz=nz, prec=prec, sweeps=3, orth=orth,
                    m=rng.choice([20, 30, 50]), rtol=1e-10, order=order)
    if kind in ("adjoint", "dropin"):
        nx, ny, nz = _sides(rng, 12000, 1.2e5 if kind == "adjoint" else 3e5)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, prec=prec, sweeps=3, m=rng.choice([30, 50]), rtol=1e-10)
    if kind == "block":
        nx, ny, nz = _sides(rng, 1000, 60000)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, prec=prec, sweeps=3, m=30, rtol=1e-10)
    return dict(kind=kind, count=rng.randint(5, 40), lo=rng.randint(9, 32), hi=rng.randint(48, 90),
                nrhs=rng.randint(1, 5), shape=rng.randint(0, 1 << 20), prec=rng.choice(["fp32", "fp64"]), sweeps=3,
                m=30, rtol=1e-12)


# ---------------------------------------------------------------- matrices

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(1000003 * (seed + 1))
    return g


def _peclet(seed):
    """The cell Peclet number of the case's operator: around 10, another for each seed."""
    return 8.0 + 4.0 * ((seed * 0.6180339887498949) % 1.0)


def _coefs(case, seed):
    """[(dx, dy, dz, value)] of the stencil, ascending row-major offset."""
    if case.get("op") == "laplace":
        return [(0, -1, 0, -1.0), (-1, 0, 0, -1.0), (0, 0, 0, 4.0), (1, 0, 0, -1.0), (0, 1, 0, -1.0)]
    px, py, pz = (_peclet(seed) * f for f in (1.0, 0.5, 0.25))
    return [(0, 0, -1, -1.0 - pz), (0, -1, 0, -1.0 - py), (-1, 0, 0, -1.0 - px), (0, 0, 0, 6.0 + px + py + pz),
            (1, 0, 0, -1.0), (0, 1, 0, -1.0), (0, 0, 1, -1.0)]


def _coords(nx, ny, nz):
    i = torch.arange(nx * ny * nz, device=DEV)
    return i % nx, (i // nx) % ny, i // (nx * ny)


def _stencil(case, seed):
    """(row, col, val) of the operator as CUDA tensors: zero-based CSR, sorted columns."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    x, y, z = _coords(nx, ny, nz)
    i = torch.arange(n, device=DEV)
    co = _coefs(case, seed)
    mask = torch.stack([(x + a >= 0) & (x + a < nx) & (y + b >= 0) & (y + b < ny) & (z + c >= 0) & (z + c < nz)
                        for a, b, c, _ in co], 1)
    cols = torch.stack([i + a + nx * (b + ny * c) for a, b, c, _ in co], 1)[mask]
    vals = torch.tensor([v for *_, v in co], dtype=torch.float64, device=DEV).expand(n, -1)[mask]
    row = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    row[1:] = mask.sum(1).cumsum(0)
    return row.int(), cols.int(), vals.contiguous()


def _level_order(case):
    """new -> old numbering by the level sets from a corner, as Cuthill-McKee numbers a box grid."""
    x, y, z = _coords(case["nx"], case["ny"], case["nz"])
    return torch.argsort(x + y + z, stable=True)


def _permute(row, col, val, new2old):
    n = new2old.numel()
    old2new = torch.empty_like(new2old)
    old2new[new2old] = torch.arange(n, device=DEV)
    rid = torch.repeat_interleave(torch.arange(n, device=DEV), (row[1:] - row[:-1]).long())
    r, c = old2new[rid], old2new[col.long()]
    o = torch.argsort(r * n + c)
    ptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    ptr[1:] = torch.bincount(r, minlength=n).cumsum(0)
    return ptr.int(), c[o].int(), val[o]


def _block_stencil(case, seed):
    """(row, col, val) of the 5x5 block stencil, diagonally dominant (the package's block workload on the GPU)."""
    bs = 5
    row, col, _ = _stencil(dict(case, op="conv"), 0)
    nb, nblk = row.numel() - 1, col.numel()
    val = torch.randn((nblk, bs, bs), generator=_gen(seed), dtype=torch.float64, device=DEV) * 0.1
    rid = torch.repeat_interleave(torch.arange(nb, device=DEV), (row[1:] - row[:-1]).long())
    dg = rid == col
    val[dg] += 5.0 * torch.eye(bs, dtype=torch.float64, device=DEV)
    tot = torch.zeros((nb, bs), dtype=torch.float64, device=DEV).index_add_(0, rid, val.abs().sum(2))
    blk = val[dg]
    d = torch.diagonal(blk, dim1=1, dim2=2)
    need = 1.05 * (tot - d.abs())
    d.copy_(torch.where(d.abs() < need, torch.where(d < 0, -need, need), d))
    val[dg] = blk
    return row, col, val


def _batch_shapes(case):
    """[(side, eps)] of the batch: the structure is the case's, the right-hand sides the seed's."""
    rng = np.random.default_rng(case["shape"])
    sides = rng.integers(case["lo"], case["hi"] + 1, size=case["count"])
    eps = np.exp(rng.uniform(math.log(0.05), 0.0, size=case["count"]))
    return [(int(s), float(e)) for s, e in zip(sides, eps)]


def _host(row, col, val):
    return problems.CSR(row.numel() - 1, row.cpu().numpy(), col.cpu().numpy(), val.cpu().numpy())


def _normal(n, seed, k=0):
    g = _gen(seed)
    out = torch.randn(n, generator=g, dtype=torch.float64, device=DEV)
    for _ in range(k):
        out = torch.randn(n, generator=g, dtype=torch.float64, device=DEV)
    return out


# ----------------------------------------------------------------- prepare

class State:
    """What a program holds between calls: context, buffers, options."""

    def __init__(self, **kw):
        self.__dict__.update(kw)


_stream = None


def _context(prec):
    """A context on the program's one compute stream, which all its contexts share."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    ctx = lg.Context(0, stream=_stream)
    ctx.set_options(precision=prec, trsv="syncfree")
    return ctx, _stream


def prepare(case, seed):
    s = globals()["_prepare_" + case["kind"]](case, seed)
    s.kind, s.case = case["kind"], case
    torch.cuda.synchronize()
    return s


def _prepare_spmv(case, seed):
    A = _host(*_stencil(case, seed))
    ctx, stream = _context("fp64")
    ctx.upload(A)
    b, x, y = _normal(A.n, seed, 1), _normal(A.n, seed), torch.zeros(A.n, dtype=torch.float64, device=DEV)
    torch.cuda.synchronize()
    ctx.spmv(x, y)
    return State(ctx=ctx, stream=stream, b=b, x=x, y=y)


def _prepare_precond(case, seed):
    A = _host(*_stencil(case, seed))
    ctx, _ = _context(case["prec"])
    ctx.upload(A)
    ctx.parilu0(case["sweeps"], residual=False)
    q = _normal(A.n, seed)
    if case["prec"] != "fp64":
        q = q.float()
    z, q64 = torch.empty_like(q), q.double()
    z64 = torch.empty_like(q64)
    torch.cuda.synchronize()
    ctx.apply_precond(q64, z64)  # plans and schedules, as the first call makes them
    return State(ctx=ctx, q=q, z=z)


def _prepare_refactor(case, seed):
    # the context was set up with the previous step's values; this step's are in device memory
    s = _prepare_precond(case, 0)
    s.val = _stencil(case, seed)[2]
    s.q = _normal(s.q.numel(), seed).to(s.q.dtype)
    return s


def _prepare_solve(case, seed):
    M = _stencil(case, seed)
    if case["order"] == "levels":
        M = _permute(*M, _level_order(case))
    A = _host(*M)
    ctx, stream = _context(case["prec"])
    ctx.upload(A)
    b, x = _normal(A.n, seed), torch.zeros(A.n, dtype=torch.float64, device=DEV)
    return State(ctx=ctx, stream=stream, b=b, x=x)


def _prepare_adjoint(case, seed):
    s = _prepare_solve(dict(case, op="conv", order="natural"), seed)
    n, nnz = s.x.numel(), _nnz(case)
    s.target = _normal(n, seed, 1)
    s.gb = torch.empty(n, dtype=torch.float64, device=DEV)
    s.gA = torch.empty(nnz, dtype=torch.float64, device=DEV)
    return s


def _prepare_block(case, seed):
    row, col, val = _block_stencil(case, seed)
    A = problems.BCSR(row.numel() - 1, 5, row.cpu().numpy(), col.cpu().numpy(), val.cpu().numpy())
    ctx, stream = _context(case["prec"])
    ctx.upload(A)
    return State(ctx=ctx, stream=stream, b=_normal(A.n, seed), x=torch.zeros(A.n, dtype=torch.float64, device=DEV))


def _prepare_dropin(case, seed):
    from lace_gb300 import dropin
    A = _host(*_stencil(case, seed))
    return State(A=dropin.csr(A.row, A.col, A.val, A.n), b=_normal(A.n, seed).cpu().numpy(), x=np.zeros(A.n))


class _Batch:
    """A lace_gpu_batch handle, destroyed before its context."""

    def __init__(self, ctx, n, row_off, nnz_off, row, col, val, nrhs):
        self.ctx, self.h = ctx, C.c_void_p()
        rc = lg.lib().lace_gpu_batch_create(C.byref(self.h), ctx.h, len(n), n.ctypes.data, row_off.ctypes.data,
                                            nnz_off.ctypes.data, row.ctypes.data, col.ctypes.data, val.ctypes.data,
                                            nrhs)
        if rc:
            raise lg.LaceError(rc, "batch_create")

    def __del__(self):
        if self.h:
            lg.lib().lace_gpu_batch_destroy(self.h)
            self.h = C.c_void_p()


def _prepare_batch(case, seed):
    mats = [problems.aniso2d(s, e) for s, e in _batch_shapes(case)]
    n = np.array([m.n for m in mats], dtype=np.int32)
    cum = lambda v: np.concatenate([[0], np.cumsum(v)[:-1]]).astype(np.int32)  # noqa: E731
    cat = lambda k: np.concatenate([getattr(m, k) for m in mats])  # noqa: E731
    ctx, stream = _context(case["prec"])
    batch = _Batch(ctx, n, cum(n), cum([m.nnz for m in mats]), cat("row").astype(np.int32),
                   cat("col").astype(np.int32), cat("val"), case["nrhs"])
    N = int(n.sum())
    return State(ctx=ctx, stream=stream, batch=batch, b=_normal(N * case["nrhs"], seed),
                 x=torch.zeros(N * case["nrhs"], dtype=torch.float64, device=DEV))


# --------------------------------------------------------------------- run

def run(s):
    return globals()["_run_" + s.kind](s)


def _run_spmv(s):
    if s.case["residual"]:  # r = b - A x
        with torch.cuda.stream(s.stream):
            s.y.copy_(s.b)
        s.ctx.spmv(s.x, s.y, alpha=-1.0, beta=1.0)
    else:
        s.ctx.spmv(s.x, s.y)
    return s.y


def _run_precond(s):
    # FP32 and BF16 factors: the FP32 vectors of the outer method's own arrays; FP64: the plain call
    if s.case["prec"] == "fp64":
        s.ctx.apply_precond(s.q, s.z)
    else:
        s.ctx.precond_enqueue(s.q, s.z)
    return s.z


def _run_refactor(s):
    s.ctx.update_values(s.val)
    step, _ = s.ctx.parilu0(s.case["sweeps"], residual=False)
    _run_precond(s)
    return [s.z, step]


def _solve(s):
    c = s.case
    with torch.cuda.stream(s.stream):
        s.x.zero_()
    s.ctx.parilu0(c["sweeps"], residual=False)
    s.ctx.fgmres(s.b, s.x, search_max=c["m"], restart_max=60, rtol=c["rtol"],
                 orthogonalization=c.get("orth", "householder"))
    return s.x


def _run_solve(s):
    return _solve(s)


def _run_block(s):
    return _solve(s)


def _run_adjoint(s):
    c = s.case
    _solve(s)
    with torch.cuda.stream(s.stream):
        g = (s.x - s.target).mul_(2.0)  # d/dx ||x - target||^2
    s.ctx.backward(s.x, g, s.gb, s.gA, search_max=c["m"], restart_max=60, rtol=c["rtol"])
    return [s.x, s.gb, s.gA]


class _Held(np.ndarray):
    """An array in memory that the library allocated, which its owner releases."""


def _values(M):
    v = np.ctypeslib.as_array(C.cast(M.m.val, C.POINTER(C.c_double)), shape=(M.m.nnz,)).view(_Held)
    v.owner = M
    return v


def _run_dropin(s):
    from lace_gb300 import dropin
    c = s.case
    dropin.set_options(precision=c["prec"])
    L, U, _ = dropin.parilu_mats(s.A, max_sweeps=c["sweeps"])
    s.x[:] = 0.0
    x, rc, log = dropin.fgmres_householder_restart(s.A, s.b, s.x, L, U, search_max=c["m"], restart_max=60,
                                                   rtol=c["rtol"], tol_type=1, x0_inplace=True)
    vals = [_values(M) for M in (L, U)]
    return [x, *vals]


def _run_batch(s):
    c = s.case
    with torch.cuda.stream(s.stream):
        s.x.zero_()
    rc = lg.lib().lace_gpu_batch_solve(s.batch.h, c["sweeps"], c["m"], 60, c["rtol"], s.b.data_ptr(),
                                       s.x.data_ptr(), None)
    if rc not in (lg.DEV_SUCCESS, lg.DEV_NOTCONVERGED):
        raise lg.LaceError(rc, "batch_solve")
    return s.x


# -------------------------------------------------------------------- work

def _nnz(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    return n + 2 * ((nx - 1) * ny * nz + nx * (ny - 1) * nz + nx * ny * (nz - 1))


def work(case):
    """Bytes and operations of one pass: matrices as CSR with int32 indices, every array once per operation that
    needs it; a solve counts its operator, factors and basis once per search direction (at the number of directions
    such a system takes)."""
    kind = case["kind"]
    if kind == "batch":
        n = sum(s * s for s, _ in _batch_shapes(case))
        pairs, dirs = case["nrhs"], 60.0
        nnz, vs, ld = 5 * n, VSIZE[case["prec"]], 1
    else:
        n, nnz = case["nx"] * case["ny"] * case["nz"], _nnz(case)
        ld = 25 if kind == "block" else 1
        vs = VSIZE[case.get("prec", "fp64")]
        pairs, dirs = 1, {"block": 5.0}.get(kind, 80.0 if case.get("op") == "laplace" else 25.0)
    rows = n * (5 if kind == "block" else 1)
    qs = 8 if case.get("prec", "fp64") == "fp64" else 4
    a_bytes = nnz * (8 * ld + 4) + 4 * n
    f_bytes = (nnz + n) * (vs * ld + 4) + 8 * n
    spmv = dict(bytes=a_bytes + (24 if case.get("residual") else 16) * rows, flops=2.0 * nnz * ld)
    apply_ = dict(bytes=f_bytes + 2 * qs * rows, flops=2.0 * nnz * ld)
    if kind == "spmv":
        return spmv
    if kind == "precond":
        return apply_
    sweep = dict(bytes=a_bytes + 2 * vs * nnz * ld, flops=6.0 * nnz * ld)
    facto = {k: case["sweeps"] * sweep[k] for k in sweep}
    if kind == "refactor":
        return {k: facto[k] + apply_[k] + (8 * nnz if k == "bytes" else 0) for k in facto}
    # a direction: the operator, the factors, the basis so far once
    m = min(case["m"], dirs)
    per = dict(bytes=a_bytes + f_bytes + 8 * rows * (m / 2 + 3), flops=4.0 * nnz * ld + 6.0 * rows * m / 2)
    solves = 2 if kind == "adjoint" else 1
    out = {k: facto[k] + pairs * solves * dirs * per[k] for k in per}
    if kind == "dropin":
        out["bytes"] += 8 * (2 * nnz + n) + 16 * rows
    return out


# ------------------------------------------------------------------- exact

class _Grid:
    """The stencil operator on a grid as FP64 torch arrays (nz, ny, nx) per offset, zero outside."""

    def __init__(self, case, seed):
        self.shape = (case["nz"], case["ny"], case["nx"])
        self.co = [(o, self._coef(*o)) for o in _coefs(case, seed)]

    def _coef(self, a, b, c, v):
        t = torch.full(self.shape, v, dtype=torch.float64, device=DEV)
        for d, o in ((2, a), (1, b), (0, c)):
            if o:
                t.select(d, 0 if o < 0 else self.shape[d] - 1).zero_()
        return t

    @staticmethod
    def shift(t, a, b, c):
        """t at (x + a, y + b, z + c), zero outside."""
        out = torch.zeros_like(t)
        src, dst = [], []
        for o, n in ((c, t.shape[0]), (b, t.shape[1]), (a, t.shape[2])):
            dst.append(slice(max(0, -o), n - max(0, o)))
            src.append(slice(max(0, o), n + min(0, o)))
        out[tuple(dst)] = t[tuple(src)]
        return out

    def matvec(self, v, transpose=False):
        t = v.view(self.shape)
        out = torch.zeros_like(t)
        for (a, b, c, _), k in self.co:
            out += self.shift(k * t, -a, -b, -c) if transpose else k * self.shift(t, a, b, c)
        return out.view(-1)

    def factors(self, sweeps):
        """The synchronous ParILU(0) sweeps from the A-initial guess: (L offsets, U diagonal, U offsets)."""
        lower = [(o[:3], k) for o, k in self.co if sum(o[:3]) < 0]
        upper = [(o[:3], k) for o, k in self.co if sum(o[:3]) > 0]
        adiag = next(k for o, k in self.co if not any(o[:3]))
        L, d, U = [(o, k.clone()) for o, k in lower], adiag.clone(), [(o, k.clone()) for o, k in upper]
        up = {o: k for o, k in U}
        for _ in range(sweeps):
            nd = adiag.clone()
            for o, k in L:  # l_ik u_ki: k = i + o, u at k towards i
                nd -= k * self.shift(up[tuple(-v for v in o)], *o)
            L = [(o, torch.where(k != 0, k / self.shift(d, *o), k)) for o, k in lower]
            d = nd
        return L, d, U

    def substitute(self, tri, diag, rhs, lower):
        """Hyperplane substitution: (diag + sum of tri offsets) x = rhs."""
        nz, ny, nx = self.shape
        n = nx * ny * nz
        x_, y_, z_ = _coords(nx, ny, nz)
        lev = x_ + y_ + z_
        order = torch.argsort(lev, stable=True)
        cnt = torch.bincount(lev).tolist()
        sets = torch.split(order, cnt)
        out = torch.zeros(n + 1, dtype=torch.float64, device=DEV)
        rhs, flat = rhs.reshape(-1).double(), [(o[0] + nx * (o[1] + ny * o[2]), k.reshape(-1)) for o, k in tri]
        dg = None if diag is None else diag.reshape(-1)
        for idx in (sets if lower else reversed(sets)):
            acc = rhs[idx]
            for off, k in flat:
                acc = acc - k[idx] * out[(idx + off).clamp(0, n)]  # a zero coefficient where the neighbour is outside
            out[idx] = acc if dg is None else acc / dg[idx]
        return out[:n]

    def precond(self, sweeps, q):
        L, d, U = self.factors(sweeps)
        return self.substitute(U, d, self.substitute(L, None, q, True), False)


def _bicgstab(mv, b, tol=1e-15, most=6000):
    """x = A^-1 b in FP64 with restarts from the true residual; mv acts on vectors like b."""
    x, best, still = torch.zeros_like(b), math.inf, 0
    bn = float(b.norm())
    xbest = x
    for _ in range(40):
        r = b - mv(x)
        rn = float(r.norm())
        if rn < 0.7 * best:
            best, xbest, still = rn, x.clone(), 0
        else:
            still += 1
        if rn <= tol * bn or still >= 2:
            break
        r0, p, rho = r.clone(), r.clone(), float(r @ r)
        target = max(tol * bn * 0.5, rn * 1e-9)
        for k in range(most):
            v = mv(p)
            den = float(r0 @ v)
            if den == 0.0:
                break
            a = rho / den
            sv = r - a * v
            t = mv(sv)
            tt = float(t @ t)
            if tt == 0.0:
                x = x + a * p
                break
            w = float(t @ sv) / tt
            x = x + a * p + w * sv
            r = sv - w * t
            rn = float(r.norm())
            if not math.isfinite(rn):
                x = xbest.clone()
                break
            if rn <= target:
                break
            rho1 = float(r0 @ r)
            if rho1 == 0.0 or w == 0.0:
                break
            p = r + (rho1 / rho) * (a / w) * (p - w * v)
            rho = rho1
    return xbest


def exact(case, seed):
    return globals()["_exact_" + case["kind"]](case, seed)


def _exact_spmv(case, seed):
    n = case["nx"] * case["ny"] * case["nz"]
    y = _Grid(case, seed).matvec(_normal(n, seed))
    return _normal(n, seed, 1) - y if case["residual"] else y


def _rounded_q(case, seed):
    q = _normal(case["nx"] * case["ny"] * case["nz"], seed)
    return q if case["prec"] == "fp64" else q.float().double()


def _exact_precond(case, seed):
    return _Grid(case, seed).precond(case["sweeps"], _rounded_q(case, seed))


def _exact_refactor(case, seed):
    return [_exact_precond(case, seed), None]


def _exact_solve(case, seed):
    g = _Grid(case, seed)
    b = _normal(case["nx"] * case["ny"] * case["nz"], seed)
    if case["order"] == "natural":
        return _bicgstab(g.matvec, b)
    p = _level_order(case)
    nat = torch.empty_like(b)
    nat[p] = b
    return _bicgstab(g.matvec, nat)[p]


def _exact_adjoint(case, seed):
    g = _Grid(case, seed)
    n = case["nx"] * case["ny"] * case["nz"]
    x = _bicgstab(g.matvec, _normal(n, seed))
    lam = _bicgstab(lambda v: g.matvec(v, True), 2.0 * (x - _normal(n, seed, 1)))
    row, col, _ = _stencil(case, seed)
    rid = torch.repeat_interleave(torch.arange(n, device=DEV), (row[1:] - row[:-1]).long())
    return [x, lam, -lam[rid] * x[col.long()]]


def _exact_block(case, seed):
    row, col, val = _block_stencil(case, seed)
    nb = row.numel() - 1
    rid = torch.repeat_interleave(torch.arange(nb, device=DEV), (row[1:] - row[:-1]).long())

    def mv(v):
        prod = torch.einsum("krc,kc->kr", val, v.view(nb, 5)[col.long()])
        return torch.zeros((nb, 5), dtype=torch.float64, device=DEV).index_add_(0, rid, prod).view(-1)

    return _bicgstab(mv, _normal(nb * 5, seed))


def _exact_dropin(case, seed):
    g = _Grid(case, seed)
    n = case["nx"] * case["ny"] * case["nz"]
    L, d, U = g.factors(case["sweeps"])
    # L by rows: ascending columns, the unit diagonal last; U by columns: ascending rows, the diagonal last
    lk = torch.stack([k.reshape(-1) for o, k in L] + [torch.ones(n, dtype=torch.float64, device=DEV)], 1)
    lm = torch.stack([k.reshape(-1) != 0 for o, k in L] + [torch.ones(n, dtype=torch.bool, device=DEV)], 1)
    uk = torch.stack([g.shift(k, *(-v for v in o)).reshape(-1) for o, k in reversed(U)] + [d.reshape(-1)], 1)
    um = torch.cat([uk[:, :-1] != 0, torch.ones((n, 1), dtype=torch.bool, device=DEV)], 1)
    x = _bicgstab(g.matvec, _normal(n, seed))
    return [x, lk[lm], uk[um]]


def _exact_batch(case, seed):
    """Fast diagonalisation: the operator is a sum of two 1D Laplacians, diagonal in the sine basis."""
    shapes = _batch_shapes(case)
    N = sum(s * s for s, _ in shapes)
    b = _normal(N * case["nrhs"], seed).view(case["nrhs"], N)
    out, at = torch.empty_like(b), 0
    for s, eps in shapes:
        k = torch.arange(1, s + 1, device=DEV, dtype=torch.float64)
        S = torch.sin(math.pi / (s + 1) * k[:, None] * k[None, :]) * math.sqrt(2.0 / (s + 1))
        lam = 2.0 - 2.0 * torch.cos(math.pi * k / (s + 1))
        rhs = b[:, at:at + s * s].reshape(-1, s, s)  # (y, x): x fastest
        out[:, at:at + s * s] = (S @ ((S @ rhs @ S) / (lam[:, None] + eps * lam[None, :])) @ S).reshape(-1, s * s)
        at += s * s
    return out.view(-1)
