"""Two host threads with a context each, as the header allows: calls of unequal
size on the same kernels do not get into each other's way."""
import threading

import numpy as np
import pytest

from statfem_b200 import api
from statfem_b200 import meshgen as mg
from tests.problems import statfem_problem
from tests.test_gpu_statfem import HP, gpu_prior

pytestmark = pytest.mark.gpu


def together(works):
    """Runs the calls in threads, each some hundred times; their errors."""
    errors, start = [], threading.Barrier(len(works))

    def loop(call, check):
        start.wait()
        try:
            for _ in range(400):
                call()
            check()
        except Exception as e:  # noqa: BLE001
            errors.append(repr(e))

    threads = [threading.Thread(target=loop, args=w) for w in works]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return errors


def works_of(make, sizes):
    """Per size a context, its call, and a check against the first result."""
    works = []
    for size in sizes:
        ctx = api.Context(0)
        call, result = make(ctx, size)
        call()
        first = result()
        works.append((call, lambda result=result, first=first: np.testing.assert_allclose(result(), first, rtol=1e-9)))
    return works


def test_likelihood_batches(ctx):
    """Systems of 150, 120, 90 and 80 sensors (more than 48 KB each)."""
    def make(c, ns):
        prob = statfem_problem(mg.TRI3_POISSON, 12, ns, seed=ns)
        g = gpu_prior(c, prob, HP, 1e-3, 1.0, api.SFC_SOLVER_PCG_MIXED, tol=1e-10)
        koh = api.LikelihoodKOH(g["fg"], prob["pts"])
        koh.setSensorValues(0.05 + 0.01 * np.random.default_rng(ns).standard_normal((ns, 2)))
        keep = [g, koh]
        out = {}
        return (lambda: out.update(ll=keep[1].giveLogLikelihoodBatch([HP]))), (lambda: out["ll"])
    assert together(works_of(make, [150, 120, 90, 80])) == []


def test_priors_by_elimination(ctx):
    """Lines of 66, 40 and 21 dofs."""
    def make(c, n):
        prob = statfem_problem(mg.TRI3_POISSON, n, 5, seed=n)
        g = gpu_prior(c, prob, HP, 1e-3, 1.0, api.SFC_SOLVER_PCG_MIXED, tol=1e-10)
        return (lambda: g["fg"].updateSolution(HP)), g["fg"].giveProjectedCovarU
    assert together(works_of(make, [65, 39, 20])) == []


def test_material_factors(ctx):
    """Ranks of unequal caps."""
    def make(c, n):
        prob = statfem_problem(mg.TRI3_POISSON, n, 3, seed=n)
        g = gpu_prior(c, prob, HP, 1e-3, 1.0, api.SFC_SOLVER_PCG_MIXED, tol=1e-10)
        pt = api.ForwardPerturbation(g["fg"])
        hp = dict(HP, **{"material.sigma": 0.3, "material.length": 0.4})
        return (lambda: pt.updateSolution(hp, factor_tol=1e-6)), pt.giveProjectedCovarU
    assert together(works_of(make, [14, 5])) == []


@pytest.mark.parametrize("kind,n", [(mg.HEX8_POISSON, 12), (mg.HEX8_ELASTIC, 7)])
def test_loads_from_one_mesh(ctx, kind, n):
    """Systems of several contexts take their loads from the same mesh, the
    first calls among them: each allocates for itself."""
    prob = statfem_problem(kind, n, 1, seed=n)
    mesh = prob["mesh"]
    f = np.arange(1.0, 1.0 + mesh.dof)
    gm = api.Mesh(ctx, kind, 8, mesh.coords, mesh.conn)
    s = api.SystemSolveCuda(ctx, mesh.num_dofs)
    s.assemble_load(gm, f)
    want = s.giveForce()
    shared = api.Mesh(ctx, kind, 8, mesh.coords, mesh.conn)
    works = []
    for _ in range(4):
        t = api.SystemSolveCuda(api.Context(0), mesh.num_dofs)

        def call(t=t):
            t.clearRhs()
            t.assemble_load(shared, f)

        works.append((call, lambda t=t: np.testing.assert_array_equal(t.giveForce(), want)))
    assert together(works) == []
