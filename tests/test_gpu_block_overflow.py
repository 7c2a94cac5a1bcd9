"""Columns that the mixed solver's FP32 iteration blows up (tiny systems, tight
tolerances: a stalled recurrence goes on for hundreds of iterations) end with
the tolerance met, not with what they blew up to."""
import numpy as np
import pytest
import scipy.sparse as sp

from oracle import oracle as O
from statfem_b200 import api
from statfem_b200 import meshgen as mg
from tests.problems import statfem_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 6, 7])
def test_inverse_of_small_squares(ctx, n):
    for seed in range(12):
        prob = statfem_problem(mg.TRI3_POISSON, n, 1, seed=seed)
        mesh, bc = prob["mesh"], prob["bc"]
        gm = api.Mesh(ctx, mesh.kind, 3, mesh.coords, mesh.conn)
        gm.set_coefficients(prob["coeff"])
        s = api.SystemSolveCuda(ctx, mesh.num_dofs)
        s.set_options(method=api.SFC_SOLVER_PCG_MIXED, tol=1e-11, max_iter=30000)
        s.assemble(gm)
        s.applyConstraints((bc, np.zeros(len(bc))))
        U = s.solveSystemTranspose(np.eye(mesh.num_dofs))
        rp, col, v, _ = O.fem(mesh, 3, 1.0, bc, coeff=prob["coeff"])
        A = sp.csr_matrix((v, col, rp)).toarray()
        # A^T U^T = I: residual 1e-11 of a unit vector, and its rounding (entries below 50, columns of a few tens)
        assert np.abs(A.T @ U.T - np.eye(len(A))).max() <= 1e-10, seed
        assert s.last_stats()["max_rel_residual"] <= 1e-10
        s.close()
        gm.close()
