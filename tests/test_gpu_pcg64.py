"""The persistent FP64 PCG kernel against the direct oracle over its operator
forms (diagonals, node blocks, rows), preconditioners and launch forms (one
cluster, cooperative grid), at sizes on both sides of each choice."""
import numpy as np
import pytest
import scipy.sparse as sp

from oracle import oracle as O
from statfem_b200 import api
from statfem_b200 import meshgen as mg
from tests.problems import QPS, statfem_problem

pytestmark = pytest.mark.gpu


def shuffled(mesh, seed):
    """The mesh with its nodes renumbered at random: no diagonals."""
    perm = np.random.default_rng(seed).permutation(mesh.num_nodes)
    inv = np.empty_like(perm)
    inv[perm] = np.arange(len(perm))
    return mg.Mesh(mesh.kind, mesh.coords[perm], inv[mesh.conn.astype(np.int64)], grid=None)


# 1e5 nonzeros divide the launch forms: 118/120 squares, 14/15 cubes, 5/8 elastic cubes
@pytest.mark.parametrize("kind,n", [(mg.LINE2_POISSON, 2), (mg.LINE2_POISSON, 700), (mg.TRI3_POISSON, 3),
                                    (mg.TRI3_POISSON, 118), (mg.TRI3_POISSON, 120), (mg.HEX8_POISSON, 14),
                                    (mg.HEX8_POISSON, 15), (mg.HEX8_ELASTIC, 5), (mg.HEX8_ELASTIC, 8)])
@pytest.mark.parametrize("precond", [api.SFC_PRECOND_JACOBI, api.SFC_PRECOND_TWO_LEVEL])
@pytest.mark.parametrize("renumber", [False, True])
def test_pcg64_matches_direct_solver(ctx, kind, n, precond, renumber):
    pr = statfem_problem(kind, n, 1, seed=n, faces="x" if kind == mg.LINE2_POISSON else "x0" if kind == mg.HEX8_ELASTIC
                         else "all")
    mesh = shuffled(pr["mesh"], n) if renumber else pr["mesh"]
    f = np.array([1.0, -0.5, 0.25])[: mesh.dof]
    bc = mg.dirichlet_dofs(mesh, "x" if kind == mg.LINE2_POISSON else "x0" if kind == mg.HEX8_ELASTIC else "all")
    val = 0.1 * np.cos(np.arange(len(bc)))  # inhomogeneous values are lifted
    gm = api.Mesh(ctx, kind, QPS[kind], mesh.coords, mesh.conn)
    gm.set_coefficients(pr["coeff"])
    s = api.SystemSolveCuda(ctx, mesh.num_dofs)
    s.set_options(method=api.SFC_SOLVER_PCG_FP64, tol=1e-12, precond=precond, max_iter=50000)
    s.assemble(gm)
    s.assemble_load(gm, f)
    s.applyConstraints((bc, val))
    s.solveSystem()
    st = s.last_stats()
    assert st["converged"] == 1 and st["iterations"] > 0
    rp, col, v, F = O.fem(mesh, QPS[kind], f, bc, coeff=pr["coeff"], bc_values=val)
    u = O.DirectSolver(rp, col, v).solve(F)
    # relative residual 1e-12 times a condition number below 1e6
    assert np.abs(s.giveSolution() - u).max() <= 1e-6 * np.abs(u).max()
    r = F - sp.csr_matrix((v, col, rp)) @ s.giveSolution()
    free = np.ones(len(F), dtype=bool)
    free[bc] = False
    # the lifted right-hand side is at most the load and the boundary couplings
    scale = np.linalg.norm(F) + np.abs(v).max() * np.linalg.norm(val) * 8
    assert np.linalg.norm(r[free]) <= 1e-11 * scale
    for o in (s, gm):
        o.close()


def test_rows_of_no_pattern(ctx):
    """A random sparse SPD matrix inserted as triplets: the row form; a zero
    right-hand side; a cap on the iterations."""
    rng = np.random.default_rng(3)
    n = 3000
    A = sp.random(n, n, density=2e-3, random_state=4)
    A = sp.csr_matrix(A @ A.T + sp.diags(1.0 + rng.random(n)))
    s = api.SystemSolveCuda(ctx, n)
    s.set_options(method=api.SFC_SOLVER_PCG_FP64, tol=1e-13)
    for i in range(n):
        c = A.indices[A.indptr[i]:A.indptr[i + 1]]
        s.insertToMatrix(A.data[A.indptr[i]:A.indptr[i + 1]].reshape(1, -1), [i], c)
    b = rng.standard_normal(n)
    s.insertToRhs(b, np.arange(n))
    s.finishAssembly()
    s.solveSystem()
    assert np.linalg.norm(A @ s.giveSolution() - b) <= 1e-12 * np.linalg.norm(b)
    s.set_options(method=api.SFC_SOLVER_PCG_FP64, tol=1e-13, max_iter=2)
    with pytest.raises(api.SfcError) as e:
        s.solveSystem()
    assert e.value.code == api.SFC_ERR_NOT_CONVERGED
    s.set_options(method=api.SFC_SOLVER_PCG_FP64, tol=1e-13)
    s.clearRhs()
    s.solveSystem()
    assert not s.giveSolution().any()
    s.close()


def test_breakdown_is_reported(ctx):
    """An indefinite matrix with a positive diagonal: p^T A p <= 0."""
    s = api.SystemSolveCuda(ctx, 2)
    s.set_options(method=api.SFC_SOLVER_PCG_FP64, tol=1e-12)
    s.insertToMatrix(np.array([[1.0, 3.0], [3.0, 1.0]]), [0, 1], [0, 1])
    s.insertToRhs(np.array([1.0, -1.0]), [0, 1])
    with pytest.raises(api.SfcError) as e:
        s.solveSystem()
    assert e.value.code == api.SFC_ERR_NOT_SPD
    s.close()
