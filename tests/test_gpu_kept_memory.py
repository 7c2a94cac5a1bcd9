"""Device memory that calls keep: large arrays are given back, by calls that
fail too."""
import numpy as np
import pytest

from statfem_b200 import api
from statfem_b200 import meshgen as mg
from tests.problems import statfem_problem
from tests.test_gpu_statfem import HP, gpu_prior

pytestmark = pytest.mark.gpu


def free_bytes():
    import torch
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("call", ["solveSystemTranspose", "solveSystemMulti"])
def test_host_columns(ctx, call):
    """600 columns of 33,124 dofs, 159 MB an array; the second call is stopped
    by its cap."""
    mesh = mg.unit_square_tri(181)
    bc = mg.dirichlet_dofs(mesh, "all")
    gm = api.Mesh(ctx, mesh.kind, 3, mesh.coords, mesh.conn)
    gm.set_coefficients()
    s = api.SystemSolveCuda(ctx, mesh.num_dofs)
    s.assemble(gm)
    s.applyConstraints((bc, np.zeros(len(bc))))
    B = np.random.default_rng(0).standard_normal((600, mesh.num_dofs))
    s.set_options(method=api.SFC_SOLVER_PCG_MIXED, tol=1e-6, precond=api.SFC_PRECOND_TWO_LEVEL)
    getattr(s, call)(B[:128])  # the solver's workspaces
    ctx.synchronize()
    before = free_bytes()
    getattr(s, call)(B)
    # the lifted columns (solveSystemMulti) stay with the solver
    kept = 8 * B.size if call == "solveSystemMulti" else 0
    assert before - free_bytes() <= kept + (64 << 20)
    before = free_bytes()
    s.set_options(method=api.SFC_SOLVER_PCG_MIXED, tol=1e-6, max_iter=16)
    with pytest.raises(api.SfcError) as e:
        getattr(s, call)(B)
    assert e.value.code == api.SFC_ERR_NOT_CONVERGED
    assert before - free_bytes() <= 64 << 20
    s.close()
    gm.close()


def test_material_workspaces(ctx):
    """56 x 56 cells, chunks of 256 factor columns by 16 sensors: 106 MB an array, five of them."""
    prob = statfem_problem(mg.TRI3_POISSON, 56, 16, seed=2)
    g = gpu_prior(ctx, prob, HP, 1e-3, 1.0, api.SFC_SOLVER_PCG_MIXED, tol=1e-9)
    pt = api.ForwardPerturbation(g["fg"])
    hp = dict(HP, **{"material.sigma": 0.3, "material.length": 0.05})
    before = free_bytes()
    pt.updateSolution(hp, max_rank=300)
    first = pt.giveProjectedCovarU()
    assert before - free_bytes() <= 512 << 20  # what it keeps, and the solver's workspaces
    pt.updateSolution(hp, max_rank=300)
    assert np.abs(pt.giveProjectedCovarU() - first).max() <= 1e-10 * np.abs(first).max()
    pt.close()
    for k in ("fg", "cf", "s", "gm"):
        g[k].close()
