"""The solves whose rows push their values to the rows that wait for them
(sptrsv_push.cu): reordered grids (up to three and up to six entries a row),
groups that end inside a level, one CTA and clusters, blocks of every size,
against the oracle's sequential substitution."""
import numpy as np
import pytest

from lace_gb300 import problems as P
from oracle import oracle as orc
from tests.test_gpu_grid import _args, grid_matrix

pytestmark = pytest.mark.gpu


def reordered(shape, how, seed=3):
    A = grid_matrix(*shape, seed=seed)
    nx, ny, nz = shape
    i = np.arange(A.n)
    level = i % nx + i // nx % ny + i // (nx * ny)
    order = np.argsort(level, kind="stable") if how == "levels" else np.random.default_rng(seed).permutation(A.n)
    at = np.empty(A.n, dtype=np.int64)
    at[order] = i
    return P._assemble(A.n, [at[A.rowidx()]], [at[A.col]], [A.val])


# the bounds of the other solves' tests: thousands of roundings of the largest value
@pytest.mark.parametrize("prec,tol", [("fp64", 1e-12), ("fp32", 1e-4), ("bf16", 5e-2)])
@pytest.mark.parametrize("how", ["levels", "random"])
@pytest.mark.parametrize("shape", [(2, 2, 1), (31, 33, 1), (64, 65, 1), (5, 9, 5), (21, 20, 19), (40, 39, 41)],
                         ids=lambda s: "%dx%dx%d" % s)
def test_pushed_solves_match_oracle(torch_cuda, shape, how, prec, tol):
    import lace_gb300 as lg
    torch = torch_cuda
    A = reordered(shape, how)
    F = orc.parilu(A.row, A.col, A.val, 2, mode="sync")
    b = np.random.default_rng(7).standard_normal(A.n)
    bd = torch.tensor(b, device="cuda")
    with lg.Context(0) as ctx:
        ctx.set_options(precision=prec)
        ctx.upload(A)
        ctx.parilu0(2)
        sol = {}
        for which in range(4):
            x = bd.clone()
            ctx.sptrsv(which, x, x)
            sol[which] = orc.trsv(*_args(F, which, b))
            assert np.abs(x.cpu().numpy() - sol[which]).max() <= tol * np.abs(sol[which]).max(), which
        if how == "levels" and A.n > 1000:
            assert ctx.trsv_schedule()[:2] == (1, 0)
        ref = orc.trsv(*_args(F, 1, sol[0]))
        z = torch.zeros(A.n, dtype=torch.float64, device="cuda")
        for sweeps in (2, 2, 3):  # the plans take the current factor values
            ctx.parilu0(sweeps)
            ctx.apply_precond(bd, z)
        F = orc.parilu(A.row, A.col, A.val, 3, mode="sync")
        ref = orc.trsv(*_args(F, 1, orc.trsv(*_args(F, 0, b))))
        assert np.abs(z.cpu().numpy() - ref).max() <= 2 * tol * np.abs(ref).max()


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-12), ("fp32", 1e-4)])
@pytest.mark.parametrize("bs", range(1, 9))
def test_pushed_block_solves_match_oracle(torch_cuda, bs, prec, tol):
    import lace_gb300 as lg
    torch = torch_cuda
    B = P.bcsr3d(7, 6, 11, bs=bs, seed=4)
    F = orc.bcsr_parilu(B, 2, mode="sync")
    Ur = F.U_rows()
    q = np.random.default_rng(2).standard_normal(B.n)
    t, ref = np.zeros(B.n), np.zeros(B.n)
    lib = orc.lib()
    lib.orc_bcsr_trsv_lower_unit(B.nb, B.bs, F.L.ptr, F.L.idx, np.ascontiguousarray(F.L.val.ravel()), q, t)
    lib.orc_bcsr_trsv_upper(B.nb, B.bs, Ur.ptr, Ur.idx, np.ascontiguousarray(Ur.val.ravel()),
                            np.ascontiguousarray(F.dinv().ravel()), t, ref)
    with lg.Context(0) as ctx:
        ctx.set_options(precision=prec)
        ctx.upload(B)
        ctx.parilu0(2)
        z = torch.zeros(B.n, dtype=torch.float64, device="cuda")
        ctx.apply_precond(torch.tensor(q, device="cuda"), z)
    assert np.abs(z.cpu().numpy() - ref).max() <= tol * np.abs(ref).max()


def test_pushed_solve_keeps_infinities_apart(torch_cuda):
    """An infinite right-hand side entry reaches the rows that depend on it and no others."""
    import lace_gb300 as lg
    torch = torch_cuda
    A = reordered((9, 20, 11), "levels")
    b = np.random.default_rng(7).standard_normal(A.n)
    b[700] = np.inf
    with lg.Context(0) as ctx:
        ctx.upload(A)
        ctx.parilu0(2)
        x = torch.zeros(A.n, dtype=torch.float64, device="cuda")
        for which in (0, 1):
            ctx.sptrsv(which, torch.tensor(b, device="cuda"), x)
            dep = np.zeros(A.n, dtype=bool)
            dep[700] = True
            for i in range(701, A.n) if which == 0 else range(699, -1, -1):
                c = A.col[A.row[i]:A.row[i + 1]]
                dep[i] = dep[c[c < i] if which == 0 else c[c > i]].any()
            assert np.array_equal(~np.isfinite(x.cpu().numpy()), dep)
