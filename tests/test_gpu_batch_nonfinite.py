"""Batched solves of pairs that have nothing to solve or cannot be solved: a zero
right-hand side (converged at once, x as it came), a zero pivot and a NaN or an
infinity in the right-hand side (not converged, x as it came), beside pairs that
must solve as on their own; in the form with a cluster per pair and in the
one with a CTA per system."""
import ctypes as C

import numpy as np
import pytest

from lace_gb300 import problems as P
from tests.test_gpu_batch import make_batch
from tests.test_gpu_batch_cluster import System, arrow

pytestmark = pytest.mark.gpu


def solve(torch, systems, b, x0, prec, restart_max=20):
    import lace_gb300 as lg
    L = lg.lib()
    n, row_off, nnz_off, row, col, val = make_batch(systems)
    nrhs = b.shape[0]
    with lg.Context(0) as ctx:
        ctx.set_options(precision=prec)
        bh = C.c_void_p()
        assert L.lace_gpu_batch_create(C.byref(bh), ctx.h, len(systems), n.ctypes.data, row_off.ctypes.data,
                                       nnz_off.ctypes.data, row.ctypes.data, col.ctypes.data, val.ctypes.data,
                                       nrhs) == 0
        bd = torch.tensor(b.ravel(), device="cuda")
        xd = torch.tensor(x0.ravel(), device="cuda")
        iters = np.zeros(len(systems) * nrhs, dtype=np.int32)
        rc = L.lace_gpu_batch_solve(bh, 3, 30, restart_max, 1e-10, bd.data_ptr(), xd.data_ptr(), iters.ctypes.data)
        L.lace_gpu_batch_destroy(bh)
    return rc, iters.reshape(len(systems), nrhs), xd.cpu().numpy().reshape(b.shape)


def parts(systems):
    n = [s.A.n for s in systems]
    return [slice(int(sum(n[:k])), int(sum(n[:k + 1]))) for k in range(len(n))]


# a system whose rows have more than four dependants takes the whole batch to the form with a CTA per system
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("form", ["cluster", "cta"])
def test_pairs_without_a_solution(torch_cuda, form, prec):
    import lace_gb300 as lg
    good = [P.aniso2d(17, 0.5), P.aniso2d(30, 0.25), arrow(200, 1) if form == "cta" else P.aniso2d(25, 0.4)]
    bad = P.aniso2d(12, 0.5)
    bad.val = bad.val.copy()
    bad.val[bad.row[0] + np.flatnonzero(bad.col[bad.row[0]:bad.row[1]] == 0)[0]] = 0.0
    one = P.CSR(1, np.array([0, 1], np.int32), np.array([0], np.int32), np.array([0.0]))
    rng = np.random.default_rng(1)
    systems = [System(A) for A in good]
    at = parts(systems)
    N = at[-1].stop
    b = rng.standard_normal((4, N))
    x0 = np.zeros((4, N))
    b[0, at[0]] = 0.0                       # nothing to solve
    b[1, at[1]] = good[1].matvec(np.ones(good[1].n))
    x0[1, at[1]] = 1.0                      # nothing left to solve
    rc, iters, x = solve(torch_cuda, systems, b, x0, prec)
    assert rc == 0
    assert iters[0, 0] == 0 and not x[0, at[0]].any()
    assert iters[1, 1] == 0 and np.array_equal(x[1, at[1]], np.ones(good[1].n))
    for k, A in enumerate(good):
        for r in range(4):
            res = np.linalg.norm(b[r, at[k]] - A.matvec(x[r, at[k]]))
            assert res <= 2e-10 * np.linalg.norm(b[r, at[k]]), (k, r)
    # the same batch with pairs that cannot be solved: the others' results stay
    systems = [System(A) for A in good + [bad, one]]
    at = parts(systems)
    N2 = at[-1].stop
    b2, x2 = np.zeros((4, N2)), np.zeros((4, N2))
    b2[:, :N], x2[:, :N] = b, x0
    b2[:, N:], x2[:, N:] = rng.standard_normal((4, N2 - N)), 0.5
    b2[2, at[0].start + 7] = np.nan
    b2[3, at[1].start + 7] = np.inf
    rc, iters2, y = solve(torch_cuda, systems, b2, x2, prec)
    assert rc == lg.DEV_NOTCONVERGED
    for k in range(len(systems)):
        for r in range(4):
            if k >= len(good) or (k, r) in ((0, 2), (1, 3)):
                assert np.array_equal(y[r, at[k]], x2[r, at[k]]), (k, r)
                assert iters2[k, r] == 0, (k, r)
            else:
                res = np.linalg.norm(b2[r, at[k]] - good[k].matvec(y[r, at[k]]))
                assert res <= 2e-10 * np.linalg.norm(b2[r, at[k]]), (k, r)
