"""Which solves a context takes and when their plans are made: a pinned schedule
keeps the block-scheduled solves, and a schedule that is chosen has the plans
of L and U, so that the preconditioner can be enqueued into a stream capture."""
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


@pytest.mark.parametrize("order", ["grid", "random"])
def test_capture_after_a_transposed_solve(torch_cuda, order):
    """The first solve is one with U^T; then M^-1 q goes into a graph."""
    import lace_gb300 as lg
    torch = torch_cuda
    A = grid_matrix(33, 20, 9, seed=3)
    if order == "random":
        at = np.random.default_rng(3).permutation(A.n)
        A = P._assemble(A.n, [at[A.rowidx()]], [at[A.col]], [A.val])
    F = orc.parilu(A.row, A.col, A.val, 2, mode="sync")
    b = np.random.default_rng(7).standard_normal(A.n)
    st = torch.cuda.Stream()
    q = torch.tensor(b, device="cuda")
    z = torch.zeros_like(q)
    torch.cuda.synchronize()
    with lg.Context(0, stream=st) as ctx:
        ctx.upload(A)
        ctx.parilu0(2)
        ctx.sptrsv(2, q, z)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            ctx.precond_enqueue(q, z)
        z.zero_()
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        ref = orc.trsv(*_args(F, 1, orc.trsv(*_args(F, 0, b))))
        assert np.abs(z.cpu().numpy() - ref).max() <= 2e-12 * np.abs(ref).max()
        del g
