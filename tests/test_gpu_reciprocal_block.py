"""Blocks of the dense elimination whose pivots are outside the reciprocal's
range, through the log-likelihood: C = eps^2 I, readings two eps off."""
import numpy as np
import pytest

from statfem_b200 import api
from statfem_b200 import meshgen as mg
from tests.problems import statfem_problem
from tests.test_gpu_statfem import HP, gpu_prior

pytestmark = pytest.mark.gpu


# a part of a block, a whole one and one pivot, several
@pytest.mark.parametrize("ns", [5, 33, 70])
def test_every_pivot_at_the_ends_of_the_range(ctx, ns):
    prob = statfem_problem(mg.LINE2_POISSON, 12, ns, seed=ns, faces="x")
    g = gpu_prior(ctx, prob, HP, 1e-3, 1.0, api.SFC_SOLVER_PCG_FP64)
    koh = api.LikelihoodKOH(g["fg"], prob["pts"])
    # 1 / eps^2 overflows the approximation, is in range, is subnormal
    for eps in (1.0e-154, 1.45e-154, 1.55e-154, 1.37, 5e153, 7e153, 1.2e154):
        hp = dict(HP, **{"rho": 1e-200, "mismatch.sigma": 0.0, "mismatch.sensorEps": eps})
        koh.setSensorValues(np.full((ns, 3), 2 * eps))
        want = 3 * ns * (-0.5 * np.log(2 * np.pi) - np.log(eps) - 2.0)
        # ns terms, each to 1e-14; subnormal numbers have 50 bits here
        assert abs(koh.giveLogLikelihood(hp) - want) <= 1e-13 * abs(want), eps
    koh.close()
    for k in ("fg", "cf", "s", "gm"):
        g[k].close()
