"""The dense inverse behind the log-likelihood at the edges of its panels
(32) and tiles (64), against NumPy on the same covariance."""
import numpy as np
import pytest

from oracle import oracle as O
from statfem_b200 import api
from statfem_b200 import meshgen as mg
from tests.problems import statfem_problem
from tests.test_gpu_statfem import gpu_prior

pytestmark = pytest.mark.gpu

HP = {"forcing.sigma": 0.1, "forcing.length": 0.2, "rho": 1.1, "mismatch.sigma": 0.02, "mismatch.length": 0.1,
      "mismatch.sensorEps": 1e-2}


def test_sizes(ctx):
    """Ascending and descending sizes on fresh and used scratch, twice each (the
    second from the captured graph)."""
    for ns in [1, 2, 31, 32, 33, 63, 64, 65, 96, 97, 128, 129, 191, 260, 64, 1]:
        prob = statfem_problem(mg.TRI3_POISSON, 20, ns, seed=ns)
        g = gpu_prior(ctx, prob, HP, 1e-3, 1.0, api.SFC_SOLVER_PCG_MIXED)
        mean, C = g["mean"], g["cov"]
        Y = (1.1 * mean)[:, None] + 0.02 * np.random.default_rng(ns).standard_normal((ns, 2))
        koh = api.LikelihoodKOH(g["fg"], prob["pts"])
        koh.setSensorValues(Y)
        Ks = O.mismatch_covariance(prob["pts"], HP["mismatch.sigma"], HP["mismatch.length"], HP["mismatch.sensorEps"])
        # condition number of K_s + rho^2 C_s below 1e5 (sigma^2 ns / eps^2): 1e-16 of it, hundredfold
        ll = O.koh_log_likelihood(mean, C, Ks, Y, HP["rho"])
        for _ in range(2):
            assert abs(koh.giveLogLikelihood(HP) - ll) <= 1e-9 * max(1.0, abs(ll)), ns
        koh.close()
        for k in ("fg", "cf", "s", "gm"):
            g[k].close()
