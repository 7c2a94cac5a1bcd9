"""The mixed block solver with blocks that are not full: right-hand sides that
end anywhere in a block, a zero one, the streamed product with fewer columns
than a row holds, and meshes that are numbered like a lattice with moved nodes
(lattice view from 8,192 nodes on) or renumbered (node blocks)."""
import numpy as np
import pytest

from oracle import oracle as O
from statfem_b200 import api
from statfem_b200 import meshgen as mg
from tests.problems import QPS, distort, small_mesh
from tests.test_gpu_pcg64 import shuffled

pytestmark = pytest.mark.gpu


def solve(ctx, mesh, Rhs, bw, precond):
    bc = mg.dirichlet_dofs(mesh, "x0" if mesh.dof == 3 else "all")
    gm = api.Mesh(ctx, mesh.kind, QPS[mesh.kind], mesh.coords, mesh.conn)
    coeff = np.exp(0.3 * np.random.default_rng(3).standard_normal(mesh.num_elems))
    gm.set_coefficients(coeff)
    s = api.SystemSolveCuda(ctx, mesh.num_dofs)
    s.assemble(gm)
    s.assemble_load(gm, np.ones(mesh.dof))
    s.applyConstraints((bc, np.zeros(len(bc))))
    s.set_options(method=api.SFC_SOLVER_PCG_MIXED, tol=1e-10, block_width=bw, precond=precond)
    U = s.solveSystemTranspose(Rhs)
    U2 = s.solveSystemTranspose(Rhs[::-1])  # another block on the workspaces of the first
    st = s.last_stats()
    np.testing.assert_allclose(U2[::-1], U, rtol=0, atol=1e-7 * np.abs(U).max())
    rp, col, val, F = O.fem(mesh, QPS[mesh.kind], np.ones(mesh.dof), bc, coeff=coeff)
    ds = O.DirectSolver(rp, col, val)
    ref = np.stack([ds.solve_transpose(r) for r in Rhs])
    assert st["converged"] == 1 and st["max_rel_residual"] <= 1e-10
    # relative residual 1e-10, condition number below 1e3 of these operators' scaled form
    assert np.abs(U - ref).max() <= 1e-7 * np.abs(ref).max()
    s.close()
    gm.close()
    return st["spmm_kernel"]


@pytest.mark.parametrize("nrhs,bw", [(1, 32), (33, 64), (40, 64), (20, 64), (66, 64), (2, 128), (61, 128), (72, 128),
                                     (100, 128), (130, 128)])
@pytest.mark.parametrize("precond", [api.SFC_PRECOND_BLOCK_JACOBI, api.SFC_PRECOND_TWO_LEVEL])
def test_lattice_block(ctx, nrhs, bw, precond):
    mesh = small_mesh(mg.HEX8_ELASTIC, 7)
    Rhs = np.random.default_rng(nrhs).standard_normal((nrhs, mesh.num_dofs))
    if nrhs > 2:
        Rhs[nrhs // 2] = 0.0
    assert solve(ctx, mesh, Rhs, bw, precond) == 4


@pytest.mark.parametrize("kind,nrhs,bw", [(mg.HEX8_POISSON, 40, 64), (mg.HEX8_POISSON, 5, 32), (mg.TRI3_POISSON, 72, 128)])
@pytest.mark.parametrize("precond", [api.SFC_PRECOND_JACOBI, api.SFC_PRECOND_TWO_LEVEL])
def test_scalar_block(ctx, kind, nrhs, bw, precond):
    mesh = small_mesh(kind, 9)
    Rhs = np.random.default_rng(nrhs).standard_normal((nrhs, mesh.num_dofs))
    Rhs[1] = 0.0
    assert solve(ctx, mesh, Rhs, bw, precond) == 1


@pytest.mark.parametrize("n,numbered,kernel", [(20, True, 4), (11, True, 2), (11, False, 2)])
@pytest.mark.parametrize("precond", [api.SFC_PRECOND_BLOCK_JACOBI, api.SFC_PRECOND_TWO_LEVEL])
def test_moved_nodes(ctx, n, numbered, kernel, precond):
    mesh = distort(small_mesh(mg.HEX8_ELASTIC, n), np.random.default_rng(n), 0.3)
    if not numbered:
        mesh = shuffled(mesh, n)
    Rhs = np.random.default_rng(n).standard_normal((40, mesh.num_dofs))
    assert solve(ctx, mesh, Rhs, 64, precond) == kernel
