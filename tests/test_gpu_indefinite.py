"""Operators that are not positive definite behind the block elimination: it
solves them without a large residual, but the calls report them as the
iteration does."""
import numpy as np
import pytest

from oracle import oracle as O
from statfem_b200 import api
from statfem_b200 import meshgen as mg
from tests.problems import QPS, statfem_problem
from tests.test_gpu_batch import make_batch, oracle_instance, rel, run_gpu
from tests.test_gpu_statfem import HP, gpu_prior

pytestmark = pytest.mark.gpu


# lines of one and several panels
@pytest.mark.parametrize("side", [6, 20, 45])
def test_batch_instances_fail_alone(ctx, side):
    """A negative definite and an indefinite instance get SFC_ERR_NOT_SPD, the
    others their oracle's values."""
    sides = [9, side, 14, side, 11]
    ns = [5, 4, 7, 6, 3]
    pb = make_batch(sides, ns, 8)
    pb["coeffs"][1] = -pb["coeffs"][1]
    pb["coeffs"][3] = pb["coeffs"][3].copy()
    pb["coeffs"][3][::3] *= -0.9
    b, gm = run_gpu(ctx, pb, 1e-3, tol=1e-11)
    for _ in range(2):  # again from the captured graph
        res = b.results()
        assert res["status"][1] == res["status"][3] == api.SFC_ERR_NOT_SPD
        for k in (0, 2, 4):
            assert res["status"][k] == 0 and res["iterations"][k] == 0
            mean, C, ll, pm, pc = oracle_instance(pb, k, 1e-3)
            assert rel(res["mean_s"][k, :ns[k]], mean) < 1e-11
            assert rel(res["cov_s"][k, :ns[k], :ns[k]], C) < 1e-11
        b.run()
    b.set_coefficients(np.abs(np.concatenate(pb["coeffs"])))  # and positive again
    b.run()
    assert (b.results()["status"] == 0).all()
    b.close()
    gm.close()


@pytest.mark.parametrize("kind,n", [(mg.LINE2_POISSON, 30), (mg.LINE2_POISSON, 150), (mg.TRI3_POISSON, 20),
                                    (mg.TRI3_POISSON, 36)])
@pytest.mark.parametrize("method", [api.SFC_SOLVER_PCG_FP64, api.SFC_SOLVER_PCG_MIXED])
def test_prior_of_an_indefinite_operator(ctx, kind, n, method):
    """Positive diagonal, a negative eigenvalue: the solves inside the statX
    objects fail with SFC_ERR_NOT_SPD, once and again, and work on the
    positive definite operator that follows."""
    prob = statfem_problem(kind, n, 4, seed=n, faces="x" if kind == mg.LINE2_POISSON else "all")
    coeff = np.ones(prob["mesh"].num_elems)
    bad = coeff.copy()
    if kind == mg.LINE2_POISSON:
        bad[n // 2] = -0.4
    else:  # every other column of cells
        bad.reshape(n, n, 2)[:, ::2] = -0.4
    rp, col, v, F = O.fem(prob["mesh"], QPS[kind], 1.0, prob["bc"], coeff=bad)
    A = np.zeros((len(F), len(F)))
    for i in range(len(F)):
        A[i, col[rp[i]:rp[i + 1]]] = v[rp[i]:rp[i + 1]]
    free = np.setdiff1d(np.arange(len(F)), prob["bc"])
    S = A[np.ix_(free, free)]
    assert S.diagonal().min() > 0 and np.linalg.eigvalsh(S).min() < 0
    prob["coeff"] = coeff
    g = gpu_prior(ctx, prob, HP, 1e-3, 1.0, method, tol=1e-10)
    good = g["fg"].giveProjectedCovarU()

    def update(c):
        g["gm"].set_coefficients(c)
        g["s"].assemble(g["gm"])
        g["s"].applyConstraints((prob["bc"], np.zeros(len(prob["bc"]))))
        g["fg"].updateSolution(HP)

    for _ in range(2):
        with pytest.raises(api.SfcError) as e:
            update(bad)
        assert e.value.code == api.SFC_ERR_NOT_SPD
    with pytest.raises(api.SfcError) as e:
        g["fg"].updateSolution(HP)  # the same operator
    assert e.value.code == api.SFC_ERR_NOT_SPD
    update(coeff)
    assert rel(g["fg"].giveProjectedCovarU(), good) < 1e-12
    for k in ("fg", "cf", "s", "gm"):
        g[k].close()
