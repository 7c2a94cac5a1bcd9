"""The material factor's cap on the rank, through ForwardPerturbation against
the dense oracle with the material covariance of NumPy's pivoted Cholesky
stopped at the same rank: one column, several, beyond the first 256."""
import numpy as np
import pytest

from oracle import oracle as O
from statfem_b200 import api
from statfem_b200 import meshgen as mg
from tests.problems import statfem_problem
from tests.test_gpu_perturbation import HP

pytestmark = pytest.mark.gpu


def truncated(C, rank):
    """L L^T after `rank` steps of the greedy pivoted Cholesky (the lowest
    index among equal pivots), and the last pivot."""
    d, L, last = C.diagonal().copy(), np.zeros((len(C), rank)), 0.0
    for k in range(rank):
        j = int(d.argmax())
        last = d[j]
        L[:, k] = (C[:, j] - L @ L[j]) / np.sqrt(last)
        d = np.maximum(d - L[:, k] ** 2, 0.0)
        d[j] = 0.0
    return L @ L.T, last


def oracle_covariance(monkeypatch, pr, hp, rank):
    """The oracle's covariance with the material covariance cut off at `rank`."""
    mesh, msig, mlen = pr["mesh"], hp["material.sigma"], hp["material.length"]
    se = O.se_matrix

    def cut(a, b, sigma, length):
        if len(a) != mesh.num_elems or length != mlen:
            return se(a, b, sigma, length)
        Cm, last = truncated(se(a, b, sigma, length), rank)
        assert last > 1e-6 * msig ** 2  # far from rounding: the order of the pivots is defined
        return Cm

    rp, col, val, F = O.fem(mesh, 3, 1.0, pr["bc"], coeff=pr["coeff"])
    phibar = O.unit_load(mesh, 3, pr["bc"])
    with monkeypatch.context() as mp:
        mp.setattr(O, "se_matrix", cut)
        return O.forward_perturbation(mesh, 3, F, rp, col, val, pr["bc"], mg.projection_dense(mesh, *pr["P"]),
                                      phibar, hp["forcing.sigma"], hp["forcing.length"], msig, mlen, 1e-4)[1]


@pytest.mark.parametrize("n,length,caps", [(4, 0.3, (1, 9)), (9, 0.25, (2, 33)), (13, 0.07, (255, 256, 257))])
def test_rank_cap_is_kept(ctx, monkeypatch, n, length, caps):
    hp = dict(HP, **{"material.length": length})
    pr = statfem_problem(mg.TRI3_POISSON, n, 3, seed=60 + n, amount=0.4)
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
    for cap in caps:
        pt.updateSolution(hp, factor_tol=1e-15, max_rank=cap)
        assert pt.rank == cap
        C, C_ref = pt.giveProjectedCovarU(), oracle_covariance(monkeypatch, pr, hp, cap)
        # solves to 1e-12; the factor's rounding (1e-16) over its last pivot (1e-6)
        assert np.abs(C - C_ref).max() <= 1e-9 * np.abs(C_ref).max()
    for o in (pt, fg, cf, s, gm):
        o.close()
