"""Direct block-tridiagonal solve behind the batched instances, against the
oracle's direct solver, where its tiles and chains have edges: a line of one
to a few row groups, a panel cut at every width, the two chains of equal and
unequal length, lines that need several CTAs per chain."""
import numpy as np
import pytest

from oracle import oracle as O
from statfem_b200 import api
from statfem_b200 import meshgen as mg
from tests.problems import statfem_problem
from tests.test_gpu_batch import make_batch, oracle_instance, rel, run_gpu
from tests.test_gpu_statfem import HP, gpu_prior, oracle_prior

pytestmark = pytest.mark.gpu


# lines of side + 1 dofs: 2, 8, 9, 32, 33, 40, 41, 64, 65, 100
@pytest.mark.parametrize("sides", [[1, 7, 8], [31, 32], [39, 40, 3], [63], [64, 2], [99]])
def test_direct_batch_matches_oracle(ctx, sides):
    """Every instance is solved without an iteration, to rounding: the prior
    within 1e-11 of SuperLU (condition number below 1e5 times 1e-16)."""
    pb = make_batch(sides, [min(32, 1 + s // 2) for s in sides], 11)
    b, gm = run_gpu(ctx, pb, 1e-3, tol=1e-11)
    res = b.results()
    assert (res["status"] == 0).all() and (res["iterations"] == 0).all()
    for k in range(len(sides)):
        m = len(pb["sensors"][k][0][0]) - 1
        mean, C, ll, pm, pc = oracle_instance(pb, k, 1e-3)
        assert rel(res["mean_s"][k, :m], mean) < 1e-11
        assert rel(res["cov_s"][k, :m, :m], C) < 1e-11
    b.close()
    gm.close()


def test_iteration_cap_keeps_its_meaning(ctx):
    """A cap that stops the iterative solve still stops the batch."""
    pb = make_batch([20], [4], 5)
    gm = api.Mesh(ctx, mg.TRI3_POISSON, 3, pb["union"].coords, pb["union"].conn)
    b = api.BatchStatFEM(ctx, gm, pb["off"], pb["sides"], pb["bc"], pb["sensors"], 1.0, 0)
    b.set_coefficients(np.concatenate(pb["coeffs"]))
    b.set_hparams(pb["hps"], 1e-3)
    b.set_readings(pb["Ys"])
    b.set_solver(tol=1e-11, max_iter=5)
    b.run()
    assert b.results()["status"][0] == api.SFC_ERR_NOT_CONVERGED
    b.set_solver(tol=1e-11)
    b.run()
    r = b.results()
    assert r["status"][0] == 0 and r["iterations"][0] == 0
    b.close()
    gm.close()


# the whole system as one line, 32-dof lines cut in the last one, grid lines
# of one to four CTAs per chain; more sensors than a column tile
@pytest.mark.parametrize("kind,n,ns,amount", [(mg.LINE2_POISSON, 1, 1, 0.0), (mg.LINE2_POISSON, 31, 5, 0.0),
                                              (mg.LINE2_POISSON, 63, 33, 0.0), (mg.LINE2_POISSON, 64, 3, 0.0),
                                              (mg.LINE2_POISSON, 150, 40, 0.0), (mg.TRI3_POISSON, 2, 2, 0.0),
                                              (mg.TRI3_POISSON, 30, 33, 0.2), (mg.TRI3_POISSON, 37, 70, 0.0),
                                              (mg.TRI3_POISSON, 66, 9, 0.0)])
def test_direct_adjoint_matches_oracle(ctx, kind, n, ns, amount):
    """Solves of ForwardGaussRHS by elimination: no iterations, the prior to
    the rounding of a direct solve (condition number below 1e5 times 1e-16)."""
    prob = statfem_problem(kind, n, ns, seed=3 + n, amount=amount, faces="x" if kind == mg.LINE2_POISSON else "all")
    g = gpu_prior(ctx, prob, HP, 1e-3, 1.0, api.SFC_SOLVER_PCG_MIXED, tol=1e-11)
    st = g["s"].last_stats()
    assert st["iterations"] == 0 and st["converged"] == 1 and st["num_rhs"] == ns
    o = oracle_prior(prob, HP, 1e-3, 1.0)
    assert rel(g["mean"], o["mean_s"]) < 1e-11
    assert rel(g["cov"], o["C_s"]) < 1e-11


def test_plain_method_keeps_its_iterations(ctx):
    prob = statfem_problem(mg.TRI3_POISSON, 32, 3, seed=2)
    g = gpu_prior(ctx, prob, HP, 1e-3, 1.0, api.SFC_SOLVER_PCG_FP64, tol=1e-11)
    assert g["s"].last_stats()["iterations"] > 0  # 1,089 dofs
