"""Which triangular solves a context takes: a pinned schedule keeps the
block-scheduled ones."""
import numpy as np
import pytest

from lace_gb300 import problems as P
from oracle import oracle as orc
from tests.test_gpu_grid import _args, grid_matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pin", [dict(schedule=(0, 8, 0)), dict(schedule=(0, 0, 2)),
                                 dict(schedule=(64, 0, 0)), dict(rows_per_lane=4)],
                         ids=["warps", "cluster", "chunks", "rows"])
def test_pinned_schedules_keep_the_block_solves(torch_cuda, pin):
    import lace_gb300 as lg
    torch = torch_cuda
    A = grid_matrix(70, 65, 1, seed=3)
    F = orc.parilu(A.row, A.col, A.val, 2, mode="sync")
    b = np.random.default_rng(7).standard_normal(A.n)
    bd, x = torch.tensor(b, device="cuda"), torch.zeros(A.n, dtype=torch.float64, device="cuda")
    with lg.Context(0) as ctx:
        ctx.upload(A)
        ctx.parilu0(2)
        ctx.sptrsv(0, bd, x)
        assert ctx.trsv_schedule()[0] == 70  # a lane per line of the grid
        ctx.set_options(**pin)
        for which in range(4):
            ctx.sptrsv(which, bd, x)
            assert ctx.trsv_schedule()[0] in (1, 2, 4)
            ref = orc.trsv(*_args(F, which, b))
            assert np.abs(x.cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max()
