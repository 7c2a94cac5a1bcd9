"""Block elimination against the tolerance: the mixed method's solves keep the
true residual below it on operators of high contrast, and what rounding swamps
is left to the iteration."""
import numpy as np
import pytest

from statfem_b200 import api
from statfem_b200 import meshgen as mg
from tests.problems import statfem_problem
from tests.test_gpu_statfem import HP, gpu_prior, oracle_prior, rel_err

pytestmark = pytest.mark.gpu


# In NumPy the elimination leaves 2.7e-14 and 5.1e-14 here and one step of
# refinement 4e-15 and 1.4e-14: tolerances between the two, and one that the
# first solution meets.
@pytest.mark.parametrize("n,tol", [(20, 1.2e-14), (36, 2.7e-14), (36, 1e-11)])
def test_mixed_solves_meet_the_tolerance(ctx, n, tol):
    prob = statfem_problem(mg.TRI3_POISSON, n, 6, seed=n)
    prob["coeff"] = np.exp(2.0 * np.random.default_rng(n).standard_normal(prob["mesh"].num_elems))
    g = gpu_prior(ctx, prob, HP, 1e-3, 1.0, api.SFC_SOLVER_PCG_MIXED, tol=tol)
    st = g["s"].last_stats()
    assert st["converged"] == 1 and st["iterations"] == 0
    assert 0 < st["max_rel_residual"] <= tol
    o = oracle_prior(prob, HP, 1e-3, 1.0)
    # condition number below 1e5 times 1e-15 (no sensor sits at a field of zero)
    assert rel_err(g["mean"], o["mean_s"]) < 1e-9
    assert rel_err(g["cov"], o["C_s"]) < 1e-9
    for k in ("fg", "cf", "s", "gm"):
        g[k].close()


@pytest.mark.parametrize("method", [api.SFC_SOLVER_PCG_FP64, api.SFC_SOLVER_PCG_MIXED])
def test_singular_operator_is_refused(ctx, method):
    """No constraint: constants are in the null space, point loads are not in
    the range."""
    prob = statfem_problem(mg.TRI3_POISSON, 12, 3, seed=5)
    prob["bc"] = np.zeros(0, dtype=np.uint32)
    with pytest.raises(api.SfcError) as e:
        gpu_prior(ctx, prob, HP, 1e-3, 1.0, method, tol=1e-10)
    assert e.value.code in (api.SFC_ERR_NOT_SPD, api.SFC_ERR_NOT_CONVERGED)
