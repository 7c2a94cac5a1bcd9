"""The reciprocal of the dense elimination over the exponents, through the
log-likelihood of one sensor: C = eps^2, readings two eps off."""
import numpy as np
import pytest

from statfem_b200 import api
from statfem_b200 import meshgen as mg
from tests.problems import statfem_problem
from tests.test_gpu_statfem import HP, gpu_prior

pytestmark = pytest.mark.gpu


def test_one_sensor_over_the_exponents(ctx):
    prob = statfem_problem(mg.LINE2_POISSON, 8, 1, seed=2, faces="x")
    g = gpu_prior(ctx, prob, HP, 1e-3, 1.0, api.SFC_SOLVER_PCG_FP64)
    koh = api.LikelihoodKOH(g["fg"], prob["pts"])
    # eps^2 from a subnormal number whose reciprocal is finite to the largest
    # numbers, whose reciprocals are subnormal
    for eps in np.concatenate([[1.0e-154, 1.45e-154, 1.55e-154], 10.0 ** np.arange(-150, 151, 6) * 1.37,
                               [5e153, 7e153, 1.2e154]]):
        hp = dict(HP, **{"rho": 1e-200, "mismatch.sigma": 0.0, "mismatch.sensorEps": eps})
        koh.setSensorValues(np.full((1, 3), 2 * eps))
        want = 3 * (-0.5 * np.log(2 * np.pi) - np.log(eps) - 2.0)
        # 1e-14 of the terms; subnormal numbers have 50 bits here
        assert abs(koh.giveLogLikelihood(hp) - want) <= 1e-13 * abs(want), eps
        assert abs(koh.giveLogLikelihoodBatch([hp])[0] - want) <= 1e-13 * abs(want), eps
