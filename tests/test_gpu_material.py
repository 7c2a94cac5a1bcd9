"""The material factor's kernel at its edges, through ForwardPerturbation
against the dense oracle: fewer elements than a warp, one warp per element
group and several, a rank beyond the factor's first allocation (256)."""
import numpy as np
import pytest

from oracle import oracle as O
from statfem_b200 import api
from statfem_b200 import meshgen as mg
from tests.problems import statfem_problem
from tests.test_gpu_perturbation import HP

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,length,rank_over", [(2, 0.3, 0), (4, 0.3, 0), (9, 0.1, 0), (16, 0.04, 256)])
def test_material_factor_matches_oracle(ctx, n, length, rank_over):
    hp = dict(HP, **{"material.length": length})
    pr = statfem_problem(mg.TRI3_POISSON, n, 3, seed=40 + n)
    mesh = pr["mesh"]
    gm = api.Mesh(ctx, mesh.kind, 3, mesh.coords, mesh.conn)
    gm.set_coefficients(pr["coeff"])
    s = api.SystemSolveCuda(ctx, mesh.num_dofs)
    s.set_options(method=api.SFC_SOLVER_PCG_MIXED, tol=1e-12)
    s.assemble(gm)
    s.assemble_load(gm, 1.0)
    s.applyConstraints((pr["bc"], np.zeros(len(pr["bc"]))))
    cf = api.CovarianceForcing(ctx, gm)
    cf.applyConstraints(pr["bc"])
    fg = api.ForwardGaussRHS(s, cf, 1e-3)
    fg.setProjectionMatrix(pr["P"])
    pt = api.ForwardPerturbation(fg, reg=1e-4)
    pt.updateSolution(hp, factor_tol=1e-15)
    assert rank_over < pt.rank <= mesh.num_elems
    C = pt.giveProjectedCovarU()
    pt.updateSolution(hp, factor_tol=1e-15, max_rank=max(1, pt.rank // 2))  # a cap on the rank is kept
    assert pt.rank <= mesh.num_elems // 2 + 1
    rp, col, val, F = O.fem(mesh, 3, 1.0, pr["bc"], coeff=pr["coeff"])
    phibar = O.unit_load(mesh, 3, pr["bc"])
    _, C_ref = O.forward_perturbation(mesh, 3, F, rp, col, val, pr["bc"], mg.projection_dense(mesh, *pr["P"]), phibar,
                                      hp["forcing.sigma"], hp["forcing.length"], hp["material.sigma"], length, 1e-4)
    # the factor drops 1e-15 of the covariance's diagonal; the solves are direct
    assert np.abs(C - C_ref).max() <= 1e-9 * np.abs(C_ref).max()
    for o in (pt, fg, cf, s, gm):
        o.close()
