"""The batched solve with a cluster per (system, right-hand side) at its edges:
systems of one row, fewer rows than search directions, rows that do not divide
over the CTAs, three and four entries a row of a triangle, and a batch whose
rows have too many dependants for it, each pair against the oracle's
FGMRES-Householder."""
import ctypes as C

import numpy as np
import pytest

from lace_gb300 import problems as P
from oracle import oracle as orc
from tests.test_gpu_batch import make_batch

pytestmark = pytest.mark.gpu


class System:
    def __init__(self, A):
        self.A = A


def banded(n, offsets, seed):
    """Dominant, with the given off-diagonals of both triangles."""
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    rows, cols = [i], [i]
    for d in offsets:
        rows += [i[d:], i[:-d]]
        cols += [i[d:] - d, i[:-d] + d]
    vals = [2.0 * len(offsets) + 0.3 + rng.random(n)] + [rng.uniform(-1, 1, len(r)) for r in rows[1:]]
    return P._assemble(n, rows, cols, vals)


def arrow(n, seed):
    """Row 0 has a dependant in every eighth row (of L; the upper triangle is a band)."""
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    k = i[8::8]
    return P._assemble(n, [i, i[1:], i[:-1], k], [i, i[1:] - 1, i[:-1] + 1, 0 * k],
                       [4.0 + rng.random(n), rng.uniform(-1, 1, n - 1), rng.uniform(-1, 1, n - 1),
                        rng.uniform(-1, 1, len(k))])


BATCHES = {
    "tiny": lambda: [P.aniso2d(s, 0.5) for s in (1, 2, 3, 5, 17)],
    "ragged": lambda: [P.aniso2d(s, 0.3) for s in (33, 7, 47, 31, 50)],
    "one_large": lambda: [P.aniso2d(90, 0.2)],
    "three": lambda: [banded(n, (1, 9, 40), n) for n in (300, 1001, 77)],
    "four": lambda: [banded(n, (1, 5, 30, 200), n) for n in (700, 2047)],
    "arrow": lambda: [arrow(n, n) for n in (100, 555)],
}


# both solve to 1e-10 of the right-hand side: 2e-10 in the residual, two directions
# apart, as in the tests of the single-CTA form
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("m", [7, 30, 64])
@pytest.mark.parametrize("name", list(BATCHES))
def test_cluster_batch_matches_oracle(torch_cuda, name, m, prec):
    import lace_gb300 as lg
    torch = torch_cuda
    systems = [System(A) for A in BATCHES[name]()]
    nrhs = 2
    n, row_off, nnz_off, row, col, val = make_batch(systems)
    N = int(n.sum())
    b = np.random.default_rng(1).standard_normal((nrhs, N))
    L = lg.lib()
    with lg.Context(0) as ctx:
        ctx.set_options(precision=prec)
        bh = C.c_void_p()
        assert L.lace_gpu_batch_create(C.byref(bh), ctx.h, len(systems), n.ctypes.data, row_off.ctypes.data,
                                       nnz_off.ctypes.data, row.ctypes.data, col.ctypes.data, val.ctypes.data,
                                       nrhs) == 0
        bd = torch.tensor(b.ravel(), device="cuda")
        its, sols = [], []
        for _ in range(2):  # a second solve finds the workspace as the first left it
            xd = torch.zeros(nrhs * N, dtype=torch.float64, device="cuda")
            iters = np.zeros(len(systems) * nrhs, dtype=np.int32)
            assert L.lace_gpu_batch_solve(bh, 3, m, 60, 1e-10, bd.data_ptr(), xd.data_ptr(), iters.ctypes.data) == 0
            its.append(iters)
            sols.append(xd.cpu().numpy())
        L.lace_gpu_batch_destroy(bh)
    assert np.array_equal(its[0], its[1]) and np.array_equal(sols[0], sols[1])
    X = sols[0].reshape(nrhs, N)
    for s, sy in enumerate(systems):
        A = sy.A
        F = orc.parilu(A.row, A.col, A.val, 3, mode="sync")
        for r in range(nrhs):
            br = b[r, row_off[s]:row_off[s] + n[s]]
            x = X[r, row_off[s]:row_off[s] + n[s]]
            assert np.linalg.norm(br - A.matvec(x)) <= 2e-10 * np.linalg.norm(br), (s, r)
            ref = orc.fgmres({"kind": "csr", "row": A.row, "col": A.col, "val": A.val},
                             orc.ilu_precond(F, "trsv_f32" if prec == "fp32" else "trsv"), br,
                             search_max=m, restart_max=60, rtol=1e-10)
            assert abs(int(its[0][s * nrhs + r]) - ref.total_iterations) <= 2, (s, r)
