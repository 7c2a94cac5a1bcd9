"""Forms of the FP64 PCG that its sizes choose between (a cluster, the grid or
launches for rows of indices; one or eight lanes to a node of block diagonals;
the restriction by numbering or by lists): a mesh and the same mesh renumbered
at random take different ones and agree."""
import numpy as np
import pytest
import scipy.sparse as sp

from statfem_b200 import api
from statfem_b200 import meshgen as mg
from tests.problems import QPS, small_mesh

pytestmark = pytest.mark.gpu


def solve(ctx, mesh, coeff, f, bc, precond, **opt):
    gm = api.Mesh(ctx, mesh.kind, QPS[mesh.kind], mesh.coords, mesh.conn)
    gm.set_coefficients(coeff)
    s = api.SystemSolveCuda(ctx, mesh.num_dofs)
    s.set_options(method=api.SFC_SOLVER_PCG_FP64, precond=precond, **dict(dict(tol=1e-12, max_iter=50000), **opt))
    s.assemble(gm)
    s.assemble_load(gm, f)
    s.applyConstraints((bc, np.zeros(len(bc))))
    try:
        s.solveSystem()
        return s.giveSolution(), s.last_stats()
    finally:
        s.close()
        gm.close()


# renumbered rows: 40 thousand nonzeros (74, 77 squares), 2 million (42, 43 cubes);
# eight lanes to a node up to 18,944 (25, 26 elastic cubes)
@pytest.mark.parametrize("kind,n", [(mg.TRI3_POISSON, 74), (mg.TRI3_POISSON, 77), (mg.HEX8_POISSON, 42),
                                    (mg.HEX8_POISSON, 43), (mg.HEX8_ELASTIC, 1), (mg.HEX8_ELASTIC, 6),
                                    (mg.HEX8_ELASTIC, 25), (mg.HEX8_ELASTIC, 26)])
@pytest.mark.parametrize("precond", [api.SFC_PRECOND_JACOBI, api.SFC_PRECOND_TWO_LEVEL])
def test_renumbered_mesh_agrees(ctx, kind, n, precond):
    rng = np.random.default_rng(n)
    mesh = small_mesh(kind, n)
    coeff = np.exp(0.3 * rng.standard_normal(mesh.num_elems))
    faces = "x0" if kind == mg.HEX8_ELASTIC else "all"
    f = np.array([1.0, -0.5, 0.25])[: mesh.dof]
    perm = rng.permutation(mesh.num_nodes)
    inv = np.empty_like(perm)
    inv[perm] = np.arange(len(perm))
    other = mg.Mesh(kind, mesh.coords[perm], inv[mesh.conn.astype(np.int64)], grid=None)
    u, st = solve(ctx, mesh, coeff, f, mg.dirichlet_dofs(mesh, faces), precond)
    v, st2 = solve(ctx, other, coeff, f, mg.dirichlet_dofs(other, faces), precond)
    assert st["converged"] == st2["converged"] == 1
    v = v.reshape(-1, mesh.dof)[inv].ravel()
    # relative residual 1e-12 times a condition number below 1e6
    assert np.abs(u - v).max() <= 1e-6 * np.abs(u).max()


def test_launches_report_as_the_kernel_does(ctx):
    """A random sparse matrix of 2.2 million entries: solved, stopped by a cap, not
    positive definite, and with a right-hand side of zero."""
    n, rng = 90000, np.random.default_rng(3)
    rows = np.repeat(np.arange(n), 12)
    A = sp.csr_matrix((0.03 * rng.standard_normal(12 * n), (rows, rng.integers(0, n, 12 * n))), shape=(n, n))
    A = (A + A.T + sp.diags(np.full(n, 1.0))).tocsr()
    assert A.nnz > 2.1e6
    for shift, cap, code in ((0.0, 20000, 0), (0.0, 5, api.SFC_ERR_NOT_CONVERGED), (-0.9, 20000, api.SFC_ERR_NOT_SPD)):
        M = (A + sp.diags(np.full(n, shift))).tocsr()
        M.sort_indices()
        s = api.SystemSolveCuda(ctx, n)
        s.set_options(method=api.SFC_SOLVER_PCG_FP64, tol=1e-11, max_iter=cap)
        for i in range(n):
            at = slice(M.indptr[i], M.indptr[i + 1])
            s.insertToMatrix(M.data[at].reshape(1, -1), [i], M.indices[at])
        b = rng.standard_normal(n)
        s.insertToRhs(b, np.arange(n))
        s.finishAssembly()
        if code:
            with pytest.raises(api.SfcError) as e:
                s.solveSystem()
            assert e.value.code == code
        else:
            s.solveSystem()
            assert np.linalg.norm(M @ s.giveSolution() - b) <= 1.1e-11 * np.linalg.norm(b)
            assert s.last_stats()["converged"] == 1
            s.clearRhs()
            s.solveSystem()
            assert not s.giveSolution().any()
        s.close()
