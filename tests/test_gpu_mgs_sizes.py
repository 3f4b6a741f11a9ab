"""The one-kernel Gram-Schmidt steps at the edges of their splits: fewer rows
than a block takes, a block more, odd counts, one row a block more than the
chip has, more than 32 basis vectors, and a system whose blocks' rows do not
fit shared memory twice (the step with a sum for every coefficient), against the
oracle's modified Gram-Schmidt."""
import numpy as np
import pytest

from lace_gb300 import problems as P
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def shifted(n, off=0.45):
    """Tridiagonal, unsymmetric, well conditioned but not solved by its ILU (one sweep)."""
    i = np.arange(n)
    rng = np.random.default_rng(n)
    return P._assemble(n, [i, i[1:], i[:-1]], [i, i[1:] - 1, i[:-1] + 1],
                       [2.0 + 0.1 * rng.random(n), -1.0 - off * rng.random(n - 1), -0.6 + 0.1 * rng.random(n - 1)])


# both reach 1e-10 on a condition number of about 100: 1e-8 of x apart at most,
# times ten for the norms in between
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("reorth", [0, 2])
@pytest.mark.parametrize("n", [2, 7, 255, 256, 257, 513, 4095, 256 * 152 - 1, 256 * 152 + 33, 2000003])
def test_mgs_one_kernel_sizes(torch_cuda, n, reorth, prec):
    import lace_gb300 as lg
    torch = torch_cuda
    if n > 1000000 and (reorth or prec == "fp64"):
        pytest.skip("one run of the large system")
    A = shifted(n)
    b = P.rhs_normal(n, 0)
    F = orc.parilu(A.row, A.col, A.val, 1, mode="sync")
    m = 45
    r = orc.fgmres_mgs({"kind": "csr", "row": A.row, "col": A.col, "val": A.val},
                       orc.ilu_precond(F, "trsv_f32" if prec == "fp32" else "trsv"), b,
                       search_max=m, restart_max=50, rtol=1e-10, reorth=reorth)
    with lg.Context(0) as ctx:
        ctx.set_options(precision=prec)
        ctx.upload(A)
        ctx.parilu0(1)
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        res = ctx.fgmres(torch.tensor(b, device="cuda"), x, search_max=m, restart_max=50, rtol=1e-10,
                         orthogonalization="mgs", reorth=reorth)
        assert ctx.solve_stats()["one_kernel_step"]
        x = x.cpu().numpy()
    assert res.converged and r.converged
    assert abs(res.total_iterations - r.total_iterations) <= 2
    assert np.linalg.norm(b - A.matvec(x)) <= 2e-10 * np.linalg.norm(b)
    assert np.linalg.norm(x - r.x) <= 1e-7 * np.linalg.norm(r.x)
