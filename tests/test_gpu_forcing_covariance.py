"""M C_f M^T on tensor grids against numpy at the edges of the kernels' tiles:
axes of 2 to 131 points (64-row tiles, 16-point steps, steps of 4), 1 to 257
projection rows (8, 64 and 128 columns), one to three axes and components."""
import numpy as np
import pytest

from oracle import oracle as O
from statfem_b200 import api
from statfem_b200 import meshgen as mg
from tests.problems import QPS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,cells,ns", [(mg.LINE2_POISSON, (1,), 1), (mg.LINE2_POISSON, (130,), 9),
                                           (mg.TRI3_POISSON, (63, 15), 64), (mg.TRI3_POISSON, (64, 16), 65),
                                           (mg.TRI3_POISSON, (2, 99), 129), (mg.HEX8_POISSON, (9,), 7),
                                           (mg.HEX8_ELASTIC, (4,), 128), (mg.HEX8_ELASTIC, (3,), 257)])
def test_projected_covariance(ctx, kind, cells, ns):
    mesh = (mg.bar(*cells) if kind == mg.LINE2_POISSON else mg.unit_square_tri(*cells) if kind == mg.TRI3_POISSON
            else mg.unit_cube_hex(cells[0], kind))
    gm = api.Mesh(ctx, kind, QPS[kind], mesh.coords, mesh.conn)
    cf = api.CovarianceForcing(ctx, gm)
    M = np.random.default_rng(ns).standard_normal((ns, mesh.num_dofs))
    hp = {"forcing.sigma": 0.7, "forcing.length": 0.3}
    got = cf.giveProjectedCovar(hp, M)
    phibar = cf.phibar()
    ref = M @ O.forcing_covariance_apply_grid(mesh, phibar, 0.7, 0.3, M.T.copy())
    # rounding of the sums over the axes and the dofs, relative to the sums of absolute values
    size = np.abs(M) @ O.forcing_covariance_apply_grid(mesh, np.abs(phibar), 0.7, 0.3, np.abs(M).T.copy())
    terms = mesh.num_dofs + sum(c + 1 for c in (cells * 3 if kind in (mg.HEX8_POISSON, mg.HEX8_ELASTIC) else cells)) + 16
    assert (np.abs(got - ref) <= 2 * terms * 1.2e-16 * size).all()
    np.testing.assert_array_equal(got, got.T)
    cf.close()
    gm.close()
