"""The grid solves (sptrsv_grid.cu): the triangular solves of factors whose
pattern is a lexicographic 5- or 7-point grid, at the edges of their tiles,
against the oracle's sequential substitution; patterns that only almost are
such a grid go the general way."""
import numpy as np
import pytest

from lace_gb300 import problems as P
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

# sides around the tile sizes (32 lines of 8 x 4, 4 x 8 or 32 x 1, four tiles a
# CTA), the four-step blocks, one line, thin boxes and more CTAs than one wave
SHAPES = [(2, 2, 1), (3, 5, 1), (64, 64, 1), (5, 33, 1), (9, 129, 1), (33, 300, 1), (2, 2, 2), (4, 8, 4), (5, 9, 5),
          (31, 17, 9), (32, 16, 8), (7, 40, 2), (3, 2, 45), (65, 33, 18), (130, 10, 11), (6, 130, 90), (1000, 9, 6)]


def grid_matrix(nx, ny, nz, seed):
    """Random diagonally dominant values on the grid's pattern."""
    A = P.laplace2d(nx, ny) if nz == 1 else P.convdiff3d(nx, ny, nz)
    rng = np.random.default_rng(seed)
    rid = A.rowidx()
    A.val = rng.uniform(-1.0, 1.0, A.nnz)
    off = np.bincount(rid, weights=np.abs(A.val) * (rid != A.col), minlength=A.n)
    d = rid == A.col
    A.val[d] = np.sign(A.val[d]) * (1.05 * off[rid[d]] + 0.1)
    return A


# an FP64 row is four roundings of terms below the row's size, and a dominant
# matrix damps them along the wavefront: 1e-12 of the largest value is
# thousands of roundings (the bound of the other solves' tests); FP32 the same
# with 6e-8 roundings and factors rounded once more
@pytest.mark.parametrize("prec,tol", [("fp64", 1e-12), ("fp32", 1e-4), ("bf16", 5e-2)])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "%dx%dx%d" % s)
def test_grid_solves_match_oracle(torch_cuda, shape, prec, tol):
    import lace_gb300 as lg
    torch = torch_cuda
    A = grid_matrix(*shape, seed=3)
    F = orc.parilu(A.row, A.col, A.val, 2, mode="sync")
    b = np.random.default_rng(7).standard_normal(A.n)
    bd = torch.tensor(b, device="cuda")
    with lg.Context(0) as ctx:
        ctx.set_options(precision=prec)
        ctx.upload(A)
        ctx.parilu0(2)
        z = torch.zeros(A.n, dtype=torch.float64, device="cuda")
        sol = {}
        for which in range(4):
            xd = torch.zeros(A.n, dtype=torch.float64, device="cuda")
            ctx.sptrsv(which, bd, xd)
            again = bd.clone()
            ctx.sptrsv(which, again, again)  # in place
            assert torch.equal(xd, again)
            ref = orc.trsv(*_args(F, which, b))
            sol[which] = ref
            err = np.abs(xd.cpu().numpy() - ref).max() / np.abs(ref).max()
            assert err <= tol, (which, err)
        # the grid solve ran (a lane per line) where it is meant to: FP64 lines of 1000 do not fit its
        # shared memory, the shortest chains are faster by chunks
        if A.n > 2000:
            assert (ctx.trsv_schedule()[0] == shape[0]) == (prec != "fp64" or shape[0] < 600)
        ref = orc.trsv(*_args(F, 1, sol[0]))
        for _ in range(3):  # the faces are ready for the next solve
            ctx.apply_precond(bd, z)
            err = np.abs(z.cpu().numpy() - ref).max() / np.abs(ref).max()
            assert err <= 2 * tol, err


def _args(F, which, b):
    from tests.test_gpu_parity import _oracle_tri
    T, lower, unit = _oracle_tri(F, which)
    return T.ptr, T.idx, T.val, b, lower, unit


@pytest.mark.parametrize("what", ["hole", "extra", "wrap"])
def test_almost_grids_go_the_general_way(torch_cuda, what):
    """One neighbour missing, one more, or lines joined end to start."""
    import lace_gb300 as lg
    torch = torch_cuda
    A = grid_matrix(12, 9, 7, seed=5)
    D = A.to_dense()
    if what == "hole":
        D[301, 300] = 0.0  # x = 1: it has a left neighbour
    elif what == "extra":
        D[500, 480] = 0.25
    else:
        D[12, 11] = D[11, 12] = 0.25
    i, j = np.nonzero(D)
    B = P._assemble(A.n, [i], [j], [D[i, j]])
    F = orc.parilu(B.row, B.col, B.val, 2, mode="sync")
    b = np.random.default_rng(7).standard_normal(B.n)
    with lg.Context(0) as ctx:
        ctx.upload(B)
        ctx.parilu0(2)
        x = torch.zeros(B.n, dtype=torch.float64, device="cuda")
        for which in range(4):
            ctx.sptrsv(which, torch.tensor(b, device="cuda"), x)
            ref = orc.trsv(*_args(F, which, b))
            assert np.abs(x.cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max()
        assert ctx.trsv_schedule()[0] in (1, 2, 4)


def test_grid_solve_keeps_infinities_apart(torch_cuda):
    """An infinite right-hand side entry reaches the rows that depend on it
    and no others, as in the sequential substitution."""
    import lace_gb300 as lg
    torch = torch_cuda
    nx, ny, nz = 9, 20, 11
    A = grid_matrix(nx, ny, nz, seed=5)
    b = np.random.default_rng(7).standard_normal(A.n)
    cx, cy, cz = 4, 9, 5
    b[cx + nx * (cy + ny * cz)] = np.inf
    with lg.Context(0) as ctx:
        ctx.upload(A)
        ctx.parilu0(2)
        x = torch.zeros(A.n, dtype=torch.float64, device="cuda")
        for which in (0, 1):
            ctx.sptrsv(which, torch.tensor(b, device="cuda"), x)
            v = x.cpu().numpy().reshape(nz, ny, nx)
            z, y, xx = np.indices(v.shape)
            dep = (z >= cz) & (y >= cy) & (xx >= cx) if which == 0 else (z <= cz) & (y <= cy) & (xx <= cx)
            assert np.array_equal(~np.isfinite(v), dep)
