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
from tests.problems import QPS, small_mesh

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


# one CTA; several; a ragged last one; 54,872 nodes: more than one round of rows per CTA
@pytest.mark.parametrize("kind,n", [(mg.LINE2_POISSON, 3), (mg.TRI3_POISSON, 5), (mg.TRI3_POISSON, 97),
                                    (mg.HEX8_POISSON, 7), (mg.HEX8_POISSON, 16), (mg.HEX8_POISSON, 37),
                                    (mg.HEX8_ELASTIC, 4)])
def test_flexible_cg_forms_agree(ctx, kind, n):
    """The persistent solve over its operator forms: diagonals with the
    gather by windows (lattice numbering), rows or node blocks (nodes
    renumbered at random).  Both reach the residual asked for, within a few
    iterations of one another (they differ in rounding only)."""
    rng = np.random.default_rng(n)
    base = small_mesh(kind, n)
    perm = rng.permutation(base.num_nodes)
    inv = np.empty_like(perm)
    inv[perm] = np.arange(len(perm))
    coeff = np.exp(0.5 * rng.standard_normal(base.num_elems))
    f = np.array([1.0, -0.5, 0.25])[: base.dof]
    its = []
    for mesh in (base, mg.Mesh(kind, base.coords[perm], inv[base.conn.astype(np.int64)], grid=None)):
        bc = mg.dirichlet_dofs(mesh, "x" if kind == mg.LINE2_POISSON else "all")
        gm = api.Mesh(ctx, kind, QPS[kind], mesh.coords, mesh.conn)
        gm.set_coefficients(coeff)
        s = api.SystemSolveCuda(ctx, mesh.num_dofs)
        s.assemble(gm)
        s.assemble_load(gm, f)
        s.applyConstraints((bc, np.zeros(len(bc))))
        net = api.LearnedPreconditioner(ctx, seed=1)
        net.set_params(R.init_params(9, decoder_scale=0.01))
        net.attach(s)
        s.set_options(method=api.SFC_SOLVER_FCG_MPNN, tol=1e-10)
        s.solveSystem()
        st = s.last_stats()
        assert st["converged"] == 1 and st["fallback_columns"] == 0
        rp, col, val, F = O.fem(mesh, QPS[kind], f, bc, coeff=coeff)
        mask = np.zeros(mesh.num_dofs, dtype=np.uint8)
        mask[bc] = 1
        S = R.symmetric_operator(rp, col, val, mask)
        b = np.where(mask, 0.0, F)
        u = s.giveSolution()
        # 1e-10 and the rounding of a residual computed on another operator copy
        assert np.linalg.norm(b - S @ u) <= 1.01e-10 * np.linalg.norm(b)
        its.append(st["iterations"])
        net.close()
    assert abs(its[0] - its[1]) <= 2 + 0.05 * its[0]


# a tile of 32 nodes mostly empty; ragged last tiles; 18,944 nodes are one tile of 128 per SM: two rounds
@pytest.mark.parametrize("kind,shape", [(mg.TRI3_POISSON, (2, 3)), (mg.TRI3_POISSON, (68, 69)), (mg.HEX8_POISSON, (25,)),
                                        (mg.TRI3_POISSON, (150, 149))])
def test_gradient_matches_oracle(ctx, kind, shape):
    """The training kernels at the sizes where their split changes, to the
    bounds the small meshes are held to."""
    rng = np.random.default_rng(sum(shape))
    mesh = mg.unit_square_tri(*shape) if kind == mg.TRI3_POISSON else mg.unit_cube_hex(*shape)
    gm = api.Mesh(ctx, kind, QPS[kind], mesh.coords, mesh.conn)
    coeff = np.exp(0.5 * rng.standard_normal(mesh.num_elems))
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
    e = rng.standard_normal(mesh.num_dofs) * 1e-2
    loss, g = net.loss_grad(s, r, e)
    loss_ref, g_ref = R.loss_grad(p, Ahat, sdinv, mask, r, e, bf16_ops=True)
    assert abs(loss - loss_ref) <= 1e-4 * abs(loss_ref)
    cuts = [R.OFF_EW, R.OFF_EB] + [R.OFF_L + l * R.LSZ + o for l in range(R.LAYERS) for o in (0, R.H * 2 * R.H)]
    for a, b in zip(cuts, cuts[1:] + [R.OFF_DW]):
        assert np.linalg.norm(g[a:b] - g_ref[a:b]) <= 1e-2 * np.linalg.norm(g_ref[a:b]) + 1e-6 * np.linalg.norm(g_ref), (a, b)
    a, b = R.OFF_DW, R.NPARAM
    assert np.linalg.norm(g[a:b] - g_ref[a:b]) <= 1e-2 * np.linalg.norm(g_ref[a:b]) + 1e-6 * np.linalg.norm(g_ref)
    net.close()
