"""Batched log-likelihoods against numpy at the sizes where the kernel's shape
changes: one sensor, the edges of a warp, more rows than warps, the last size
whose system fits shared memory and the first that does not."""
import numpy as np
import pytest

from statfem_b200 import api
from statfem_b200 import meshgen as mg
from tests.problems import statfem_problem
from tests.test_gpu_statfem import gpu_prior

pytestmark = pytest.mark.gpu

HP = {"forcing.sigma": 0.3, "forcing.length": 0.3, "rho": 1.0, "mismatch.sigma": 0.05, "mismatch.length": 0.2,
      "mismatch.sensorEps": 0.05}


@pytest.mark.parametrize("ns,n_o", [(1, 1), (2, 5), (31, 1), (32, 4), (33, 70), (64, 8), (159, 1), (160, 1)])
def test_batch_matches_numpy(ctx, ns, n_o):
    prob = statfem_problem(mg.TRI3_POISSON, 14, ns, seed=ns)
    g = gpu_prior(ctx, prob, HP, 1e-3, 1.0, api.SFC_SOLVER_PCG_FP64, tol=1e-12)
    rng = np.random.default_rng(n_o)
    Y = g["mean"][:, None] + 0.1 * rng.standard_normal((ns, n_o))
    koh = api.LikelihoodKOH(g["fg"], prob["pts"])
    koh.setSensorValues(Y)
    hps = [dict(HP, **{"rho": rng.uniform(0.5, 2), "mismatch.sigma": rng.uniform(0.01, 0.1),
                       "mismatch.length": rng.uniform(0.05, 0.5)}) for _ in range(150 if ns < 40 else 5)]
    hps[-1]["mismatch.sigma"] = np.nan  # not positive definite
    got = koh.giveLogLikelihoodBatch(hps)
    d2 = ((prob["pts"][:, None, :] - prob["pts"][None, :, :]) ** 2)[..., :2].sum(-1)
    for h, v in zip(hps[:-1], got):
        K = h["mismatch.sigma"] ** 2 * np.exp(-d2 / (2 * h["mismatch.length"] ** 2)) + h["mismatch.sensorEps"] ** 2 * np.eye(ns)
        C = K + h["rho"] ** 2 * g["cov"]
        D = Y - h["rho"] * g["mean"][:, None]
        quad = np.einsum("ir,ir->", D, np.linalg.solve(C, D))
        logdet = np.linalg.slogdet(C)[1]
        ref = n_o * (-0.5 * ns * np.log(2 * np.pi) - 0.5 * logdet) - 0.5 * quad
        # backward stable factorisations on both sides: ns u cond(C) relative in each term
        tol = 8 * ns * 2.3e-16 * np.linalg.cond(C) * (quad + n_o * (abs(logdet) + ns))
        assert abs(v - ref) <= tol
    assert np.isnan(got[-1])


@pytest.mark.parametrize("ns", [1, 8, 31, 32, 33, 63, 64, 65, 96, 97, 130, 200])
def test_single_matches_numpy(ctx, ns):
    """The log-likelihood and the posterior through the block Gauss-Jordan
    inverse, at the edges of its 32-wide panels and 64 x 64 tiles (an odd and
    an even number of panels: the result lies in either copy)."""
    prob = statfem_problem(mg.TRI3_POISSON, 16, ns, seed=ns)
    g = gpu_prior(ctx, prob, HP, 1e-3, 1.0, api.SFC_SOLVER_PCG_FP64, tol=1e-12)
    Y = g["mean"][:, None] + 0.1 * np.random.default_rng(ns).standard_normal((ns, 3))
    koh = api.LikelihoodKOH(g["fg"], prob["pts"])
    koh.setSensorValues(Y)
    d2 = ((prob["pts"][:, None, :] - prob["pts"][None, :, :]) ** 2)[..., :2].sum(-1)
    C = 0.05 ** 2 * np.exp(-d2 / (2 * 0.2 ** 2)) + 0.05 ** 2 * np.eye(ns) + g["cov"]
    D = Y - g["mean"][:, None]
    quad = np.einsum("ir,ir->", D, np.linalg.solve(C, D))
    logdet = np.linalg.slogdet(C)[1]
    ref = 3 * (-0.5 * ns * np.log(2 * np.pi) - 0.5 * logdet) - 0.5 * quad
    # ns u cond(C) relative in each term
    tol = 8 * ns * 2.3e-16 * np.linalg.cond(C) * (quad + 3 * (abs(logdet) + ns))
    for _ in range(2):  # a replay of the captured launches too
        assert abs(koh.giveLogLikelihood(HP) - ref) <= tol
    with pytest.raises(api.SfcError):
        koh.giveLogLikelihood(dict(HP, **{"mismatch.sigma": np.nan}))
