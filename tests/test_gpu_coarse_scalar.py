"""The coarse matrix of scalar meshes: rows of 3 to 41 entries (more than a
warp), aggregates smaller and larger than the rows that a cluster takes at
once.  A wrong entry would show in the iteration count, which a numpy PCG with
the coarse matrix formed from the same boxes predicts."""
import numpy as np
import pytest
import scipy.sparse as sp

from oracle import mpnn_ref as R
from oracle import oracle as O
from statfem_b200 import api
from statfem_b200 import meshgen as mg
from tests.problems import QPS

pytestmark = pytest.mark.gpu


def fan(sectors, rings):
    """A disk of triangles whose centre couples to every node of the first ring."""
    ang = 2 * np.pi * np.arange(sectors) / sectors
    X = [[0.0, 0.0, 0.0]] + [[r / rings * np.cos(a), r / rings * np.sin(a), 0.0] for r in range(1, rings + 1) for a in ang]
    node = lambda r, s: 0 if r == 0 else 1 + (r - 1) * sectors + s % sectors  # noqa: E731
    T = [[0, node(1, s), node(1, s + 1)] for s in range(sectors)]
    for r in range(1, rings):
        for s in range(sectors):
            T += [[node(r, s), node(r + 1, s), node(r + 1, s + 1)], [node(r, s), node(r + 1, s + 1), node(r, s + 1)]]
    bc = np.arange(1 + (rings - 1) * sectors, 1 + rings * sectors)
    return mg.Mesh(mg.TRI3_POISSON, np.array(X), np.array(T)), bc


@pytest.mark.parametrize("name", ["fan", "square", "cube", "cube 16"])
def test_iterations_match_numpy(ctx, name):
    if name == "fan":
        mesh, bc = fan(40, 25)
    else:
        mesh = mg.unit_square_tri(37) if name == "square" else mg.unit_cube_hex(11 if name == "cube" else 16)
        bc = mg.dirichlet_dofs(mesh, "all")
    size = 3 if name == "cube" else 8
    coeff = np.exp(0.5 * np.random.default_rng(1).standard_normal(mesh.num_elems))
    gm = api.Mesh(ctx, mesh.kind, QPS[mesh.kind], mesh.coords, mesh.conn)
    gm.set_coefficients(coeff)
    s = api.SystemSolveCuda(ctx, mesh.num_dofs)
    s.set_options(method=api.SFC_SOLVER_PCG_FP64, tol=1e-10, precond=api.SFC_PRECOND_TWO_LEVEL, coarse_size=size)
    s.assemble(gm)
    s.assemble_load(gm, np.ones(1))
    s.applyConstraints((bc, np.zeros(len(bc))))
    s.solveSystem()
    st = s.last_stats()
    rp, col, val, F = O.fem(mesh, QPS[mesh.kind], np.ones(1), bc, coeff=coeff)
    mask = np.zeros(mesh.num_dofs, dtype=np.uint8)
    mask[bc] = 1
    S = sp.csr_matrix(R.symmetric_operator(rp, col, val, mask))
    b = np.where(mask, 0.0, F)
    agg = np.asarray(api.coarse_boxes(mesh.coords, mesh.conn, size)[0])
    P = sp.csr_matrix(((1 - mask).astype(float), (np.arange(len(b)), agg)))
    Ac = np.linalg.pinv((P.T @ S @ P).toarray(), rcond=1e-12, hermitian=True)
    d = S.diagonal()
    x, r = np.zeros_like(b), b.copy()
    z = r / d + P @ (Ac @ (P.T @ r))
    p, rz, n = z.copy(), r @ z, 0
    while np.linalg.norm(r) > 1e-10 * np.linalg.norm(b):
        q = S @ p
        al = rz / (p @ q)
        x += al * p
        r -= al * q
        z = r / d + P @ (Ac @ (P.T @ r))
        p, rz, n = z + (r @ z) / rz * p, r @ z, n + 1
    assert st["converged"] == 1 and abs(st["iterations"] - n) <= 1
    assert np.abs(s.giveSolution() - x).max() <= 1e-7 * np.abs(x).max()
