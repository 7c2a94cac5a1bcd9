"""Inference layers of the learned preconditioner at the sizes where the split
of the nodes over the CTAs changes (32 nodes a tile, a ragged last tile, more,
the MMA's 128 with several tiles per CTA): against the CPU oracle with the same
BF16 rounding points, within the bound the small meshes are held to (the slack
covers FP32 accumulation order and the BF16 roundings that it flips)."""
import numpy as np
import pytest

from oracle import mpnn_ref as R
from oracle import oracle as O
from statfem_b200 import api
from statfem_b200 import meshgen as mg
from tests.problems import QPS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,shape", [(mg.TRI3_POISSON, (2, 3)), (mg.TRI3_POISSON, (68, 69)), (mg.HEX8_POISSON, (28,)),
                                        (mg.HEX8_POISSON, (33,)), (mg.TRI3_POISSON, (286, 280))])
def test_apply_matches_oracle(ctx, kind, shape):
    rng = np.random.default_rng(sum(shape))
    mesh = mg.unit_square_tri(*shape) if kind == mg.TRI3_POISSON else mg.unit_cube_hex(*shape)
    coeff = np.exp(0.5 * rng.standard_normal(mesh.num_elems))
    gm = api.Mesh(ctx, kind, QPS[kind], mesh.coords, mesh.conn)
    gm.set_coefficients(coeff)
    s = api.SystemSolveCuda(ctx, mesh.num_dofs)
    s.assemble(gm)
    s.assemble_load(gm, np.ones(1))
    bc = mg.dirichlet_dofs(mesh, "all")
    s.applyConstraints((bc, np.zeros(len(bc))))
    rp, col, val, _ = O.fem(mesh, QPS[kind], np.ones(1), bc, coeff=coeff)
    mask = np.zeros(mesh.num_dofs, dtype=np.uint8)
    mask[bc] = 1
    Ahat, sdinv = R.scaled_operator(R.symmetric_operator(rp, col, val, mask))
    net = api.LearnedPreconditioner(ctx, seed=0)
    p = R.init_params(5, decoder_scale=0.3)
    net.set_params(p)
    r = rng.standard_normal(mesh.num_dofs) * 1e3
    z_ref = R.apply_inference(p, Ahat, sdinv, mask, r)
    assert np.linalg.norm(net.apply(s, r) - z_ref) <= 1e-3 * np.linalg.norm(z_ref)
