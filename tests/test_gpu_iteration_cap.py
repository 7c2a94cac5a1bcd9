"""The persistent solvers under the largest cap on the iterations: their sums
go round a few slots, whatever the cap."""
import numpy as np
import pytest

from statfem_b200 import api
from statfem_b200 import meshgen as mg
from tests.problems import QPS, statfem_problem

pytestmark = pytest.mark.gpu


# one cluster, the grid (1e5 nonzeros divide them), the learned CG with a restart from the true residual
@pytest.mark.parametrize("kind,n,method,precond", [
    (mg.TRI3_POISSON, 20, api.SFC_SOLVER_PCG_FP64, api.SFC_PRECOND_JACOBI),
    (mg.TRI3_POISSON, 130, api.SFC_SOLVER_PCG_FP64, api.SFC_PRECOND_JACOBI),
    (mg.TRI3_POISSON, 130, api.SFC_SOLVER_PCG_FP64, api.SFC_PRECOND_TWO_LEVEL),
    (mg.HEX8_POISSON, 15, api.SFC_SOLVER_FCG_MPNN, api.SFC_PRECOND_JACOBI),
    (mg.TRI3_POISSON, 40, api.SFC_SOLVER_FCG_MPNN, api.SFC_PRECOND_JACOBI)])
def test_largest_cap(ctx, kind, n, method, precond):
    pr = statfem_problem(kind, n, 1, seed=n)
    mesh = pr["mesh"]
    gm = api.Mesh(ctx, kind, QPS[kind], mesh.coords, mesh.conn)
    gm.set_coefficients(pr["coeff"])
    s = api.SystemSolveCuda(ctx, mesh.num_dofs)
    net = api.LearnedPreconditioner(ctx, seed=1)
    net.attach(s)
    s.assemble(gm)
    s.assemble_load(gm, 1.0)
    s.applyConstraints((pr["bc"], np.zeros(len(pr["bc"]))))
    u, st = [], []
    for cap in (20000, 2 ** 31 - 1):
        s.set_options(method=method, precond=precond, tol=1e-12, max_iter=cap)
        s.solveSystem()
        u.append(s.giveSolution())
        st.append(s.last_stats())
    assert st[0]["converged"] == st[1]["converged"] == 1 and st[1]["iterations"] > 8
    # sums in another order: a step or two of a hundred, the solution to the residual times the condition number
    assert abs(st[0]["iterations"] - st[1]["iterations"]) <= 2 + st[0]["iterations"] // 20
    assert np.abs(u[0] - u[1]).max() <= 1e-8 * np.abs(u[0]).max()
    s.close()
    net.close()
    gm.close()
