"""Which solves inside the statX objects the block elimination takes, and their
results on long lines and long chains of lines."""
import numpy as np
import pytest

from oracle import oracle as O
from statfem_b200 import api
from statfem_b200 import meshgen as mg
from tests.test_gpu_statfem import HP

pytestmark = pytest.mark.gpu


def prior(ctx, nx, ny, ns, precond, tol=1e-12, oracle=False, held="all"):
    """Prior at ns sensors of an nx x ny grid of square cells, held on its
    boundary or at its short ends; solver stats, and the mean by the oracle."""
    mesh = mg.unit_square_tri(nx, ny)
    rng = np.random.default_rng(nx + ny)
    P = mg.projection_matrix(mesh, mg.interior_points(rng, ns, 2, margin=0.05))
    bc = mg.dirichlet_dofs(mesh, "all")
    if held == "ends":
        bc = bc[mesh.coords[bc, 1] * (1 - mesh.coords[bc, 1]) < 1e-9]
    X = mesh.coords.copy()
    X[:, 1] *= ny / nx
    mesh = mg.Mesh(mesh.kind, X, mesh.conn, grid=mesh.grid)
    coeff = np.exp(0.5 * rng.standard_normal(mesh.num_elems))
    gm = api.Mesh(ctx, mesh.kind, 3, mesh.coords, mesh.conn)
    gm.set_coefficients(coeff)
    s = api.SystemSolveCuda(ctx, mesh.num_dofs)
    s.set_options(method=api.SFC_SOLVER_PCG_MIXED, tol=tol, precond=precond, max_iter=30000)
    s.assemble(gm)
    s.assemble_load(gm, 1.0)
    s.applyConstraints((bc, np.zeros(len(bc))))
    cf = api.CovarianceForcing(ctx, gm)
    cf.applyConstraints(bc)
    fg = api.ForwardGaussRHS(s, cf, 1e-3)
    fg.setProjectionMatrix(P)
    fg.updateSolution(HP)
    st, mean, cov = s.last_stats(), fg.giveProjectedMeanU(), fg.giveProjectedCovarU()
    for o in (fg, cf, s, gm):
        o.close()
    want = None
    if oracle:
        rp, col, v, F = O.fem(mesh, 3, 1.0, bc, coeff=coeff)
        u = O.DirectSolver(rp, col, v).solve(F)
        want = np.array([np.dot(P[2][a:b], u[P[1][a:b]]) for a, b in zip(P[0][:-1], P[0][1:])])
    return st, mean, cov, want


# lines of 258 to 320 dofs, one more than fits, and hundreds of short ones
@pytest.mark.parametrize("nx,ny,direct", [(257, 9, True), (288, 4, True), (318, 12, True), (319, 5, True),
                                          (320, 5, False), (30, 300, True), (33, 250, True), (12, 700, True)])
def test_lines_and_chains(ctx, nx, ny, direct):
    """Against the oracle's direct solver (condition number below 1e5 times
    1e-12), and the covariance against the two-level iteration."""
    st, mean, cov, want = prior(ctx, nx, ny, 9, api.SFC_PRECOND_JACOBI, oracle=True)
    assert (st["iterations"] == 0) == direct and st["max_rel_residual"] <= 1e-12
    assert np.abs(mean - want).max() <= 1e-7 * np.abs(want).max()
    _, mean2, cov2, _ = prior(ctx, nx, ny, 40, api.SFC_PRECOND_TWO_LEVEL)
    _, mean1, cov1, _ = prior(ctx, nx, ny, 40, api.SFC_PRECOND_JACOBI)
    assert np.abs(mean1 - mean2).max() <= 1e-7 * np.abs(mean1).max()
    assert np.abs(cov1 - cov2).max() <= 1e-7 * np.abs(cov1).max()


# the faster of the two as measured, on both sides of the line; a strip that
# is held along its edges and one that is held at its ends only
@pytest.mark.parametrize("nx,ny,ns,precond,held,direct", [
    (64, 64, 1, "two-level", "all", True), (128, 128, 8, "two-level", "all", True),
    (230, 230, 8, "two-level", "all", False), (230, 230, 200, "two-level", "all", True),
    (300, 300, 1, "two-level", "all", False), (20, 2000, 8, "two-level", "all", False),
    (20, 2000, 200, "two-level", "all", True), (60, 2000, 8, "two-level", "all", False),
    (60, 2000, 75, "two-level", "all", True), (230, 230, 8, "jacobi", "all", True),
    (60, 2000, 8, "jacobi", "all", True), (8, 3000, 8, "jacobi", "all", False), (8, 300, 8, "jacobi", "ends", True)])
def test_faster_route(ctx, nx, ny, ns, precond, held, direct):
    pre = {"jacobi": api.SFC_PRECOND_JACOBI, "two-level": api.SFC_PRECOND_TWO_LEVEL}[precond]
    st, _, _, _ = prior(ctx, nx, ny, ns, pre, tol=1e-11, held=held)
    assert (st["iterations"] == 0) == direct
    assert st["converged"] == 1 and st["max_rel_residual"] <= 1e-11
