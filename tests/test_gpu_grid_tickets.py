"""The grid solves (sptrsv_grid.cu) where clusters of CTAs take more than one
group of tiles: the tiles of a second round reuse the shared-memory faces of the
first at another start offset, so every entry the first one left there has to
be marked unsolved again, those past a line's end among them.  Against the
oracle's sequential substitution, all four triangles, again and again."""
import numpy as np
import pytest

from lace_gb300 import problems as P
from oracle import oracle as orc
from tests.test_gpu_grid import _args, grid_matrix

pytestmark = pytest.mark.gpu

# groups of tiles for the clusters that 152 SMs hold at most: FP64 35 for 19, 28
# for 19, 70 for 38 (L) and 19 (U), FP32 70 for 57 and 38; with the tiles' offsets
# of 0 to 3, lines of 13, 61, 127 and 128 rows end on every entry of a block of four
SHAPES = [("fp64", (127, 130, 97)), ("fp64", (128, 128, 100)), ("fp64", (61, 200, 150)), ("fp32", (13, 200, 300))]


# the bounds of the other solves' tests: thousands of roundings of the largest value
@pytest.mark.parametrize("prec,shape", SHAPES, ids=lambda v: v if isinstance(v, str) else "%dx%dx%d" % v)
def test_second_round_of_tiles(torch_cuda, prec, shape):
    import lace_gb300 as lg
    torch = torch_cuda
    tol = {"fp64": 1e-12, "fp32": 1e-4}[prec]
    A = grid_matrix(*shape, seed=3)
    F = orc.parilu(A.row, A.col, A.val, 2, mode="sync")
    b = np.random.default_rng(7).standard_normal(A.n)
    bd = torch.tensor(b, device="cuda")
    with lg.Context(0) as ctx:
        ctx.set_options(precision=prec)
        ctx.upload(A)
        ctx.parilu0(2)
        sol = {}
        for which in range(4):
            x = torch.zeros(A.n, dtype=torch.float64, device="cuda")
            ctx.sptrsv(which, bd, x)
            sol[which] = orc.trsv(*_args(F, which, b))
            err = np.abs(x.cpu().numpy() - sol[which]).max() / np.abs(sol[which]).max()
            assert err <= tol, (which, err)
            for _ in range(5):
                y = torch.zeros_like(x)
                ctx.sptrsv(which, bd, y)
                assert torch.equal(x, y)
        assert ctx.trsv_schedule()[0] == shape[0]
        ref = torch.tensor(orc.trsv(*_args(F, 1, sol[0])), device="cuda")
        z = torch.zeros(A.n, dtype=torch.float64, device="cuda")
        for _ in range(20):
            ctx.apply_precond(bd, z)
            err = float((z - ref).abs().max() / ref.abs().max())
            assert err <= 2 * tol, err
