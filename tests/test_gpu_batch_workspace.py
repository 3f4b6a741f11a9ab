"""A batched solve whose workspace could not be allocated leaves the batch
usable: the next call at the old number of directions (more than the failed
one's, so more memory) has a plan and a workspace of that size again."""
import ctypes as C

import numpy as np
import pytest

from lace_gb300 import problems as P
from tests.test_gpu_batch import make_batch
from tests.test_gpu_batch_cluster import System, arrow

pytestmark = pytest.mark.gpu

DEV_ERR_DEVICE_ALLOC = -113


# the form with a cluster per pair, and (too many dependants a row) the one with a CTA per system
@pytest.mark.parametrize("form", ["cluster", "cta"])
def test_failed_workspace_is_made_again(torch_cuda, form):
    import lace_gb300 as lg
    torch = torch_cuda
    systems = [System(A) for A in (P.aniso2d(25, 0.4), arrow(300, 1) if form == "cta" else P.aniso2d(31, 0.3))]
    n, row_off, nnz_off, row, col, val = make_batch(systems)
    N, nrhs = int(n.sum()), 2
    bd = torch.tensor(np.random.default_rng(1).standard_normal(nrhs * N), device="cuda")
    L = lg.lib()

    def solve(bh, m):
        x = torch.zeros(nrhs * N, dtype=torch.float64, device="cuda")
        rc = L.lace_gpu_batch_solve(bh, 3, m, 60, 1e-10, bd.data_ptr(), x.data_ptr(), None)
        return rc, x

    failures = 0
    try:
        for k in range(40):
            with lg.Context(0) as ctx:
                bh = C.c_void_p()
                assert L.lace_gpu_batch_create(C.byref(bh), ctx.h, len(systems), n.ctypes.data, row_off.ctypes.data,
                                               nnz_off.ctypes.data, row.ctypes.data, col.ctypes.data,
                                               val.ctypes.data, nrhs) == 0
                rc, ref = solve(bh, 10)
                assert rc == 0
                L.lace_gpu_inject_alloc_failure(k)
                rc, _ = solve(bh, 40)
                L.lace_gpu_inject_alloc_failure(-1)
                done = rc == 0
                if not done:
                    assert rc == DEV_ERR_DEVICE_ALLOC
                    failures += 1
                rc, x = solve(bh, 10)  # back to what it had
                assert rc == 0 and torch.equal(x, ref)
                rc, large = solve(bh, 40)
                assert rc == 0
                L.lace_gpu_inject_alloc_failure(k)
                rc, _ = solve(bh, 5)
                L.lace_gpu_inject_alloc_failure(-1)
                assert rc in (0, DEV_ERR_DEVICE_ALLOC)
                rc, x = solve(bh, 40)
                assert rc == 0 and torch.equal(x, large)
                L.lace_gpu_batch_destroy(bh)
                if done:
                    break
    finally:
        L.lace_gpu_inject_alloc_failure(-1)
    assert failures >= 1
