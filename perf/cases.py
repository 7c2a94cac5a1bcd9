"""Timed cases of the statFEM path, each a program's own calls of statfem_b200.api.

listed() names them; draw(rng) gives more of the same ranges; prepare(case,
seed) builds what the program holds before the call (mesh, system, sensors,
inputs made from the seed); run(state) is one pass; exact(case, seed) gives
the pass's results in 64-bit torch arithmetic without the library.

Kinds of case:
  field      statFEM on a bar or a small square with the full-field Woodbury
             posterior (mean and covariance of every dof)
  proposals  one step of many Metropolis chains: the log-likelihoods of a list
             of hyperparameter proposals
  posterior  one material proposal: assembly, forward solve, prior at the
             sensors, log-likelihood and posterior (square, cube, elastic cube)
  batch      many independent square instances of uneven size in one launch
  material   prior with first-order material uncertainty
  forward    assembly and forward solve of a heterogeneous Poisson cube
  learned    the same through flexible CG with the message-passing network
  gradient   loss and gradient of the network for one residual/error pair
  transpose  transposed solves of host right-hand sides on a distorted elastic mesh
  columns    many device-resident right-hand sides on an elastic cube
"""
import functools
import math

import numpy as np
import torch

from statfem_b200 import api
from statfem_b200 import meshgen as mg
from statfem_b200 import workloads

KINDS = {"bar": mg.LINE2_POISSON, "square": mg.TRI3_POISSON, "cube": mg.HEX8_POISSON, "elastic": mg.HEX8_ELASTIC}
QUAD = {"bar": 3, "square": 3, "cube": 8, "elastic": 8}
METHOD = {"fp64": api.SFC_SOLVER_PCG_FP64, "mixed": api.SFC_SOLVER_PCG_MIXED, "learned": api.SFC_SOLVER_FCG_MPNN}
PRECOND = {"jacobi": api.SFC_PRECOND_JACOBI, "block": api.SFC_PRECOND_BLOCK_JACOBI,
           "two-level": api.SFC_PRECOND_TWO_LEVEL}
REG = workloads.REG


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest program: the 32-element bar of the laplaceRHSinfer app, its full-field posterior
        dict(name="bar 32 field", kind="field", mesh="bar", n=32, sensors=11, readings=20, method="fp64", tol=1e-13),
        # one step of 64 chains over the mismatch hyperparameters, 32 sensors
        dict(name="proposals 64 x 32", kind="proposals", mesh="square", n=32, sensors=32, readings=4, proposals=64),
        # the plain 2-D problem: 64 x 64 cells, 16 sensors
        dict(name="square 64 posterior 16", kind="posterior", mesh="square", n=64, sensors=16, method="mixed",
             precond="two-level", tol=1e-11, eps=1e-3),
        # a larger square with a ragged number of sensors
        dict(name="square 181 posterior 75", kind="posterior", mesh="square", n=181, sensors=75, method="mixed",
             precond="two-level", tol=1e-11, eps=1e-3),
        # material proposals of uneven size in one launch
        dict(name="square batch 40", kind="batch", count=40, smin=32, smax=150, sensors=32, tol=1e-11),
        # first-order material uncertainty on a small square
        dict(name="square 20 material", kind="material", mesh="square", n=20, sensors=8, method="mixed", tol=1e-11),
        # heterogeneous conductivity on a cube, one right-hand side
        dict(name="cube 80 forward", kind="forward", mesh="cube", n=80, method="fp64", precond="two-level",
             tol=1e-11),
        # the same method with the learned preconditioner, odd size
        dict(name="cube 33 learned", kind="learned", mesh="cube", n=33, tol=1e-11),
        # one training pair of the network
        dict(name="cube 24 gradient", kind="gradient", mesh="cube", n=24),
        # a mesh that is no lattice, right-hand sides on the host
        dict(name="distorted elastic 25 transpose 40", kind="transpose", mesh="elastic", n=25, nrhs=40,
             method="mixed", precond="block", tol=1e-11),
        # covariance columns on the device, a ragged last block
        dict(name="elastic 31 columns 200", kind="columns", mesh="elastic", n=31, nrhs=200, method="mixed",
             precond="two-level", tol=1e-10),
        # the large problem: 48^3 elasticity with 256 sensors
        dict(name="elastic 48 posterior 256", kind="posterior", mesh="elastic", n=48, sensors=256, method="mixed",
             precond="two-level", tol=1e-11, eps=1e-3),
    ]


def draw(rng):
    def between(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["field", "proposals", "posterior", "posterior", "posterior", "batch", "material", "forward",
                       "learned", "gradient", "transpose", "columns"])
    if kind == "field":
        mesh = rng.choice(["bar", "square"])
        return dict(kind=kind, mesh=mesh, n=between(16, 150) if mesh == "bar" else between(6, 34),
                    sensors=between(4, 40), readings=rng.randint(1, 30),
                    **(dict(method="fp64", tol=1e-13) if mesh == "bar" else dict(method="mixed", tol=1e-11)))
    if kind == "proposals":
        return dict(kind=kind, mesh="square", n=between(12, 64), sensors=between(6, 64), readings=rng.randint(1, 8),
                    proposals=between(8, 600))
    if kind == "posterior":
        mesh = rng.choice(["square", "cube", "elastic"])
        n = {"square": between(24, 230), "cube": between(8, 40), "elastic": between(6, 36)}[mesh]
        precond = rng.choice(["jacobi", "two-level"]) if mesh == "square" else rng.choice(["block", "two-level"])
        return dict(kind=kind, mesh=mesh, n=n, sensors=between(5, 200), method="mixed", precond=precond, tol=1e-11,
                    eps=1e-3)
    if kind == "batch":
        smin = between(8, 40)
        return dict(kind=kind, count=between(6, 40), smin=smin, smax=between(smin, 150), sensors=rng.randint(4, 32),
                    tol=1e-11)
    if kind == "material":
        return dict(kind=kind, mesh="square", n=between(6, 20), sensors=rng.randint(3, 10), method="mixed", tol=1e-11)
    if kind == "forward":
        return dict(kind=kind, mesh="cube", n=between(10, 80), method="fp64",
                    precond=rng.choice(["jacobi", "two-level"]), tol=1e-11)
    if kind == "learned":
        return dict(kind=kind, mesh="cube", n=between(8, 33), tol=1e-11)
    if kind == "gradient":
        return dict(kind=kind, mesh="cube", n=between(6, 32))
    if kind == "transpose":
        return dict(kind=kind, mesh="elastic", n=between(5, 25), nrhs=between(1, 60), method="mixed", precond="block",
                    tol=1e-11)
    return dict(kind=kind, mesh="elastic", n=between(8, 31), nrhs=between(20, 300), method="mixed",
                precond=rng.choice(["block", "two-level"]), tol=1e-10)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _context():
    """One context per program, as the C ABI asks (one per host thread)."""
    return api.Context(0)


def _mesh(case, rng):
    n = case["n"]
    if case["mesh"] == "bar":
        return mg.bar(n)
    if case["mesh"] == "square":
        return mg.unit_square_tri(n)
    m = mg.unit_cube_hex(n, KINDS[case["mesh"]])
    if case["kind"] != "transpose":
        return m
    X = m.coords.copy()  # interior nodes moved: no tensor grid
    inner = np.all((X > 1e-9) & (X < 1 - 1e-9), axis=1)
    X[inner] += 0.3 / n * (rng.random((int(inner.sum()), 3)) - 0.5)
    return mg.Mesh(m.kind, X, m.conn, grid=m.grid)


def _coefficients(case, mesh, rng):
    """Lognormal fields: conductivity 0.5 (square, bar) or 1.0 (cube) with
    squared-exponential correlation, Young's modulus 0.3."""
    n = case["n"]
    ax = mg.cell_centre_axes(n)
    if case["mesh"] == "bar":
        return np.exp(mg.se_field_tensor(rng, [ax], 0.5, 0.3))
    if case["mesh"] == "square":
        return np.repeat(np.exp(mg.se_field_tensor(rng, [ax, ax], 0.5, rng.uniform(0.1, 0.5))), 2)
    sigma, length = (1.0, 0.1) if case["mesh"] == "cube" else (0.3, 0.25)
    return np.exp(mg.se_field_tensor(rng, [ax, ax, ax], sigma, length))


def _load(case):
    return np.array([0.0, 0.0, -1.0]) if case["mesh"] == "elastic" else np.array([1.0])


def _faces(case):
    return {"bar": "x", "elastic": "x0"}.get(case["mesh"], "all")


def _rough_solution(case, pts):
    """A closed-form guess of the solution at the sensors: what readings look
    like before the model is calibrated."""
    if case["mesh"] == "bar":
        return 0.5 * pts[:, 0] * (1 - pts[:, 0])
    if case["mesh"] == "square":
        return 0.0737 * np.prod(np.sin(np.pi * pts[:, :2]), axis=1)
    if case["mesh"] == "cube":
        return 0.0562 * np.prod(np.sin(np.pi * pts), axis=1)
    x, z = pts[:, 0], pts[:, 2]
    w = -(x * x * (6 - 4 * x + x * x) / 2 + 3.12 * (x - 0.5 * x * x))
    u = (z - 0.5) * (6 * x - 6 * x * x + 2 * x ** 3)
    return np.choose(np.arange(len(pts)) % 3, [u, np.zeros_like(u), w])


def _hparams(case):
    if case["mesh"] == "elastic":
        hp = dict(workloads.C2_HP)
    else:
        hp = dict(workloads.C1_HP, **{"mismatch.sigma": 0.01, "mismatch.length": 0.3})
    hp["mismatch.sensorEps"] = case.get("eps", 1e-3)
    return hp


def _problem(case, seed):
    """Host-side inputs of one problem, from the seed alone."""
    rng = np.random.default_rng([seed, 20])
    mesh = _mesh(case, rng)
    pr = dict(mesh=mesh, bc=mg.dirichlet_dofs(mesh, _faces(case)), load=_load(case),
              coeff=_coefficients(case, mesh, rng), hp=_hparams(case))
    if "sensors" in case:
        ns = case["sensors"]
        pts = mg.interior_points(rng, ns, mesh.dim, margin=0.02)
        comps = np.arange(ns) % 3 if mesh.dof == 3 else None
        pr["pts"], pr["P"] = pts, mg.projection_matrix(mesh, pts, comps)
        u = _rough_solution(case, pts)
        scale = 0.03 * np.abs(u).max()
        pr["Y"] = u[:, None] * (1 + 0.05 * rng.standard_normal()) + scale * rng.standard_normal(
            (ns, case.get("readings", 1)))
    if case["kind"] == "proposals":
        pr["proposals"] = [dict(pr["hp"], **{"rho": rng.uniform(0.7, 1.4), "mismatch.sigma": rng.uniform(0.002, 0.05),
                                             "mismatch.length": rng.uniform(0.1, 0.5)})
                           for _ in range(case["proposals"])]
    if case["kind"] == "transpose":
        pr["rhs"] = rng.standard_normal((case["nrhs"], mesh.num_dofs)) / case["n"]
    if case["kind"] == "gradient":
        # a residual and its error are smooth fields on the mesh; boundary values are zero
        x = mesh.coords
        k = rng.integers(1, 6, (6, 3))
        a = rng.standard_normal(6)
        e = sum(a[i] * np.prod(np.sin(np.pi * k[i] * x), axis=1) for i in range(6))
        pr["err"] = 0.05 * e
        pr["res"] = (0.5 * e + 0.2 * rng.standard_normal(len(e))) / case["n"] ** 3
        for v in (pr["err"], pr["res"]):
            v[pr["bc"]] = 0.0
    if case["kind"] in ("gradient", "learned"):
        pr["params"] = _network(rng, 0.3 if case["kind"] == "gradient" else 0.01)
    return pr


def _network(rng, decoder):
    """Network parameters with the trainer's initial distribution and a
    decoder of the given scale (E, e, three layers W, b, decoder w, c)."""
    p = [0.7 * rng.standard_normal(128), np.full(64, 0.05)]
    for _ in range(3):
        p += [rng.standard_normal(64 * 128) * math.sqrt(2.0 / 128), 0.01 * rng.standard_normal(64)]
    p += [decoder * rng.standard_normal(64), np.array([0.01 * decoder])]
    return np.concatenate(p).astype(np.float32)


def _batch_problem(case, seed):
    sides = np.linspace(case["smin"], case["smax"], case["count"]).round().astype(np.int64)
    wl = workloads.make_batch_workload(seed, n_inst=case["count"], ns=case["sensors"], sides=sides)
    rng = np.random.default_rng([seed, 21])
    wl["hps"] = [dict(workloads.C3_HP, **{"forcing.length": rng.uniform(0.15, 0.3), "rho": rng.uniform(0.8, 1.2),
                                          "mismatch.sigma": 0.005}) for _ in sides]
    wl["Y"] = [(0.0737 * np.prod(np.sin(np.pi * p), axis=1) * (1 + 0.1 * rng.standard_normal())
                + 0.002 * rng.standard_normal(len(p)))[:, None] for _, p in wl["sensors"]]
    return wl


# ---------------------------------------------------------------------------
# a program's state and its pass
# ---------------------------------------------------------------------------
class State:
    """The handles a program keeps; closed in reverse order of creation."""

    def __init__(self, case):
        self.case = case
        self.handles = []

    def keep(self, h):
        self.handles.append(h)
        return h

    def __del__(self):
        try:
            while self.handles:
                self.handles.pop().close()
        except Exception:
            pass


def prepare(case, seed):
    ctx = _context()
    st = State(case)
    kind = case["kind"]
    if kind == "batch":
        wl = _batch_problem(case, seed)
        gm = st.keep(api.Mesh(ctx, mg.TRI3_POISSON, 3, wl["union"].coords, wl["union"].conn))
        st.b = st.keep(api.BatchStatFEM(ctx, gm, wl["off"], wl["sides"], wl["bc"], wl["sensors"], 1.0))
        st.b.set_solver(tol=case["tol"])
        st.b.set_hparams(wl["hps"], REG)
        st.coeff, st.Y = wl["coeff"], wl["Y"]
        return st
    pr = st.pr = _problem(case, seed)
    mesh = pr["mesh"]
    st.gm = st.keep(api.Mesh(ctx, mesh.kind, QUAD[case["mesh"]], mesh.coords, mesh.conn))
    s = st.s = st.keep(api.SystemSolveCuda(ctx, mesh.num_dofs))
    st.bc_values = np.zeros(len(pr["bc"]))
    s.set_options(method=METHOD[case.get("method", "learned" if kind == "learned" else "fp64")],
                  precond=PRECOND[case.get("precond", "jacobi")], tol=case.get("tol", 1e-13), max_iter=30000)
    if "sensors" in case:
        cf = st.keep(api.CovarianceForcing(ctx, st.gm))
        cf.applyConstraints(pr["bc"])
        st.fg = st.keep(api.ForwardGaussRHS(s, cf, REG))
        st.fg.setProjectionMatrix(pr["P"])
    if kind in ("field", "proposals", "posterior"):
        st.koh = st.keep(api.LikelihoodKOH(st.fg, pr["pts"]))
        st.koh.setSensorValues(pr["Y"])
    if kind in ("learned", "gradient"):
        st.net = api.LearnedPreconditioner(ctx, seed=0)
        st.handles.insert(0, st.net)  # the system is closed before its network
        st.net.set_params(pr["params"])
        if kind == "learned":
            st.net.attach(s)
    if kind == "material":
        st.pt = st.keep(api.ForwardPerturbation(st.fg, reg=1e-4))
        st.hp = dict(pr["hp"], **{"material.sigma": 0.4, "material.length": 0.3})
    if kind in ("proposals", "gradient", "transpose", "columns"):
        _assemble(st)  # the material of these passes is fixed
    if kind == "proposals":
        st.fg.updateSolution(pr["hp"])
    if kind == "columns":
        B = np.ascontiguousarray(_columns(case, pr).T)  # interleaved [N][nrhs]
        st.B = torch.from_numpy(B).cuda()
        st.U = torch.empty_like(st.B)
    return st


def _columns(case, pr):
    """Leading columns of the body-force covariance's factor on the mesh."""
    mesh = pr["mesh"]
    phibar = _unit_load(mesh, pr["bc"]).cpu().numpy()
    return workloads.multi_rhs_columns(dict(mesh=mesh, phibar=phibar), case["nrhs"], 0.05, 0.3)


def _assemble(st):
    pr = st.pr
    st.gm.set_coefficients(pr["coeff"])
    st.s.assemble(st.gm)
    st.s.clearRhs()
    st.s.assemble_load(st.gm, pr["load"])
    st.s.applyConstraints((pr["bc"], st.bc_values))


def run(st):
    kind = st.case["kind"]
    if kind == "batch":
        st.b.set_coefficients(st.coeff)
        st.b.set_readings(st.Y)
        st.b.run()
        r = st.b.results()
        return {k: r[k] for k in ("loglik", "mean_s", "cov_s", "post_mean", "post_cov", "status")}
    pr = st.pr
    if kind == "proposals":
        return st.koh.giveLogLikelihoodBatch(pr["proposals"])
    if kind == "gradient":
        loss, g = st.net.loss_grad(st.s, pr["res"], pr["err"])
        return {"loss": loss, "grad": g}
    if kind == "transpose":
        return st.s.solveSystemTranspose(pr["rhs"])
    if kind == "columns":
        st.s.solve_multi_device(st.B.data_ptr(), st.U.data_ptr(), st.case["nrhs"])
        return st.U
    _assemble(st)
    if kind in ("forward", "learned"):
        st.s.solveSystem()
        return st.s.giveSolution()
    if kind == "material":
        st.pt.updateSolution(st.hp)
        return {"mean": st.pt.giveProjectedMeanU(), "cov": st.pt.giveProjectedCovarU()}
    if kind == "posterior":
        st.s.solveSystem()
    st.fg.updateSolution(pr["hp"])
    if kind == "field":
        mean, cov = st.koh.giveFEconditionedDataWoodbury(pr["hp"])
        return {"mean": mean, "cov": cov}
    ll = st.koh.giveLogLikelihood(pr["hp"])
    pm, pc = st.koh.giveProjFEconditionedData(pr["hp"])
    return {"u": st.s.giveSolution(), "prior_mean": st.fg.giveProjectedMeanU(),
            "prior_cov": st.fg.giveProjectedCovarU(), "loglik": ll, "mean": pm, "cov": pc}


# ---------------------------------------------------------------------------
# least work of a pass: inputs once, outputs once, one product with the
# operator per right-hand side and the dense sensor-space algebra
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "batch":
        sides = np.linspace(case["smin"], case["smax"], case["count"]).round()
        N, ns = float(((sides + 1) ** 2).sum()), case["sensors"]
        return dict(bytes=8.0 * (2 * (sides ** 2).sum() + 2 * case["count"] * (ns * ns + 2 * ns)),
                    flops=14.0 * N * ns + 4.0 * case["count"] * ns ** 3 + 2.0 * N * ns * ns)
    n, dim = case["n"], {"bar": 1, "square": 2}.get(case["mesh"], 3)
    dof = 3 if case["mesh"] == "elastic" else 1
    N = dof * (n + 1) ** dim
    elems = n ** dim * (2 if dim == 2 else 1)
    nnz = N * dof * {1: 3, 2: 7, 3: 27}[dim]
    ns = case.get("sensors", 0)
    if kind == "proposals":
        m = case["proposals"]
        return dict(bytes=8.0 * (7 * m + ns * ns + ns * (case["readings"] + 4)),
                    flops=float(m) * (ns ** 3 / 3.0 + 2 * ns * ns * case["readings"] + 10 * ns * ns))
    if kind == "gradient":
        return dict(bytes=12.0 * nnz + 16.0 * N, flops=3.0 * 3 * (2.0 * 64 * 128 * N + 128.0 * nnz))
    if kind == "transpose":
        return dict(bytes=12.0 * nnz + 16.0 * N * case["nrhs"], flops=2.0 * nnz * case["nrhs"])
    if kind == "columns":
        return dict(bytes=12.0 * nnz + 16.0 * N * case["nrhs"], flops=2.0 * nnz * case["nrhs"])
    if kind in ("forward", "learned"):
        return dict(bytes=8.0 * (elems + N) + 12.0 * nnz, flops=2.0 * nnz)
    nrhs = ns + 1
    out = ns * ns + 2 * ns
    if kind == "field":
        out = N * N + N
    return dict(bytes=8.0 * (elems + out) + 12.0 * nnz + 8.0 * N * nrhs,
                flops=2.0 * nnz * nrhs + 2.0 * N * ns * ns + 4.0 * ns ** 3 + (2.0 * N * N * ns if kind == "field" else 0))


# ---------------------------------------------------------------------------
# the same results in 64-bit torch arithmetic
# ---------------------------------------------------------------------------
_DEV = "cuda" if torch.cuda.is_available() else "cpu"
_G = 0.5 * (1 - 1 / math.sqrt(3.0))
_CORNER = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.asarray(a), dtype=dtype, device=_DEV)


def _quadrature(kind):
    """(weights, shape values [q][nn], reference gradients [q][dim][nn])"""
    if kind == mg.LINE2_POISSON:
        pts = [0.5]  # the gradients are constant and the load integrand linear
        return [1.0], [[1 - x, x] for x in pts], [[[-1.0, 1.0]] for _ in pts]
    if kind == mg.TRI3_POISSON:
        return [0.5], [[1 / 3.0] * 3], [[[-1.0, 1.0, 0.0], [-1.0, 0.0, 1.0]]]
    w, phi, dphi = [], [], []
    for z in (_G, 1 - _G):
        for y in (_G, 1 - _G):
            for x in (_G, 1 - _G):
                p = (x, y, z)
                f = [[p[a] if c[a] else 1 - p[a] for a in range(3)] for c in _CORNER]
                s = [[1.0 if c[a] else -1.0 for a in range(3)] for c in _CORNER]
                w.append(0.125)
                phi.append([v[0] * v[1] * v[2] for v in f])
                dphi.append([[s[k][a] * f[k][(a + 1) % 3] * f[k][(a + 2) % 3] for k in range(8)] for a in range(3)])
    return w, phi, dphi


def _geometry(mesh):
    """Per quadrature point: w detJ [E], shape values [nn], d phi_k / d x_i [E][dim][nn]."""
    X = _t(mesh.coords)[_t(mesh.conn.astype(np.int64), torch.int64)][:, :, :mesh.dim]
    for w, phi, dphi in zip(*_quadrature(mesh.kind)):
        J = torch.einsum("ak,ekj->eaj", _t(dphi), X)  # d x_j / d xi_a
        yield w * torch.linalg.det(J), _t(phi), torch.linalg.solve(J, _t(dphi).expand(X.shape[0], -1, -1))


def _element_matrices(mesh, coeff, nu=0.3):
    c, ke = _t(coeff), 0.0
    for wdet, _, g in _geometry(mesh):
        if mesh.dof == 1:
            k = torch.einsum("eim,ein->emn", g, g)
        else:
            lam, mu = nu / (1 + nu) / (1 - 2 * nu), 0.5 / (1 + nu)
            k = lam * torch.einsum("eim,ekn->emink", g, g) + mu * torch.einsum("ekm,ein->emink", g, g)
            k += mu * torch.einsum("eam,ean,ik->emink", g, g, torch.eye(3, dtype=torch.float64, device=_DEV))
            k = k.reshape(len(c), 3 * g.shape[2], -1)
        ke = ke + (wdet * c)[:, None, None] * k
    return ke


def _element_dofs(mesh):
    conn = _t(mesh.conn.astype(np.int64), torch.int64)
    d = mesh.dof
    return (conn[:, :, None] * d + torch.arange(d, device=_DEV)).reshape(conn.shape[0], -1)


def _unit_load(mesh, bc):
    """phibar: the unit load per dof, zero on constrained dofs."""
    fe = sum(wdet[:, None] * phi for wdet, phi, _ in _geometry(mesh))
    node = torch.zeros(mesh.num_nodes, dtype=torch.float64, device=_DEV)
    node.index_add_(0, _t(mesh.conn.astype(np.int64), torch.int64).reshape(-1), fe.reshape(-1))
    out = node.repeat_interleave(mesh.dof)
    out[_t(bc.astype(np.int64), torch.int64)] = 0.0
    return out


class _Exact:
    """The assembled problem: K (sparse), free dofs, load, and a solver."""

    def __init__(self, case, pr):
        mesh = self.mesh = pr["mesh"]
        N = self.N = mesh.num_dofs
        ke = _element_matrices(mesh, pr["coeff"])
        dofs = _element_dofs(mesh)
        L = dofs.shape[1]
        idx = torch.stack([dofs[:, :, None].expand(-1, -1, L).reshape(-1), dofs[:, None, :].expand(-1, L, -1).reshape(-1)])
        K = torch.sparse_coo_tensor(idx, ke.reshape(-1), (N, N)).coalesce()
        del ke, idx
        self.free = torch.ones(N, dtype=torch.bool, device=_DEV)
        self.free[_t(pr["bc"].astype(np.int64), torch.int64)] = False
        i, v = K.indices(), K.values()
        both = self.free[i[0]] & self.free[i[1]]
        self.fc = (i[0][self.free[i[0]] & ~self.free[i[1]]], i[1][self.free[i[0]] & ~self.free[i[1]]],
                   v[self.free[i[0]] & ~self.free[i[1]]])  # free row, constrained column
        num = torch.cumsum(self.free, 0) - 1
        nf = self.nf = int(self.free.sum())
        self.S = torch.sparse_coo_tensor(torch.stack([num[i[0][both]], num[i[1][both]]]), v[both], (nf, nf)).coalesce()
        self.phibar = _unit_load(mesh, pr["bc"])
        f = _t(pr["load"])
        self.F = self.phibar * f.repeat(mesh.num_nodes) if mesh.dof == 3 else self.phibar * f
        self.chol = None

    def solve(self, B):
        """S X = B on the free dofs (B: nf x m)."""
        if self.nf <= 20000:
            if self.chol is None:
                self.dense = self.S.to_dense()
                self.chol = torch.linalg.cholesky(self.dense)
            X = torch.cholesky_solve(B, self.chol)
            return X + torch.cholesky_solve(B - self.dense @ X, self.chol)
        S = self.S.to_sparse_csr()
        diag = torch.zeros(self.nf, dtype=torch.float64, device=_DEV)
        i = self.S.indices()
        diag[i[0][i[0] == i[1]]] = self.S.values()[i[0] == i[1]]
        X, R = torch.zeros_like(B), B.clone()
        for _ in range(2):  # to 1e-14 of the right-hand side, the residual recomputed once
            Z = R / diag[:, None]
            P = Z.clone()
            rz = (R * Z).sum(0)
            stop = 1e-14 * B.norm(dim=0)
            for it in range(20000):
                Q = S @ P
                a = rz / (P * Q).sum(0).clamp_min(1e-300)
                X += a * P
                R -= a * Q
                if it % 25 == 0 and bool((R.norm(dim=0) <= stop).all()):
                    break
                Z = R / diag[:, None]
                new = (R * Z).sum(0)
                P = Z + (new / rz.clamp_min(1e-300)) * P
                rz = new
            R = B - S @ X
        return X

    def solve_all(self, B):
        """A X = B and A^T X = B share S on the free dofs; constrained rows of
        A are identity rows, so X there is B (A) or B - K_fc^T X_f (A^T)."""
        X = B.clone()
        X[self.free] = self.solve(B[self.free])
        return X

    def forcing(self, W, sigma, length):
        """C_f W: squared-exponential over node coordinates, diag(phibar) on both sides."""
        d, out = self.mesh.dof, torch.zeros_like(W)
        T = self.phibar[:, None] * W
        shape = [g + 1 for g in self.mesh.grid][::-1]
        axes = [torch.arange(g + 1, dtype=torch.float64, device=_DEV) / g for g in self.mesh.grid]
        for c in range(d):
            t = T[c::d].reshape(shape + [W.shape[1]])
            for a, x in enumerate(axes):
                Kx = torch.exp(-(x[:, None] - x[None, :]) ** 2 / (2 * length * length))
                t = torch.movedim(torch.tensordot(Kx, t, dims=([1], [len(axes) - 1 - a])), 0, len(axes) - 1 - a)
            out[c::d] = t.reshape(-1, W.shape[1])
        return sigma * sigma * self.phibar[:, None] * out

    def prior(self, pr):
        ns = len(pr["P"][0]) - 1
        P = _dense_projection(pr["P"], self.N)
        R = torch.zeros(self.N, ns, dtype=torch.float64, device=_DEV)
        R[self.free] = self.solve(P.T[self.free].contiguous())
        hp = pr["hp"]
        C = R.T @ self.forcing(R, hp["forcing.sigma"], hp["forcing.length"])
        return P, R, R.T @ self.F, 0.5 * (C + C.T)


def _dense_projection(P, N):
    ip, ix, dv = (_t(P[0], torch.int64), _t(P[1], torch.int64), _t(P[2]))
    row = torch.repeat_interleave(torch.arange(len(ip) - 1, device=_DEV), ip[1:] - ip[:-1])
    out = torch.zeros(len(ip) - 1, N, dtype=torch.float64, device=_DEV)
    return out.index_put_((row, ix), dv, accumulate=True)


def _mismatch(pts, hp):
    X = _t(pts)
    D2 = ((X[:, None, :] - X[None, :, :]) ** 2).sum(2)
    K = hp["mismatch.sigma"] ** 2 * torch.exp(-D2 / (2 * hp["mismatch.length"] ** 2))
    return K + hp["mismatch.sensorEps"] ** 2 * torch.eye(len(X), dtype=torch.float64, device=_DEV)


def _loglik(mean, C, pts, Y, hp):
    L = torch.linalg.cholesky(_mismatch(pts, hp) + hp["rho"] ** 2 * C)
    Z = torch.linalg.solve_triangular(L, Y - hp["rho"] * mean[:, None], upper=False)
    ns, n_o = Y.shape
    return float(n_o * (-0.5 * ns * math.log(2 * math.pi) - L.diagonal().log().sum()) - 0.5 * (Z * Z).sum())


def _condition(mean, C, pts, Y, hp, cross=None, prior=None):
    """(posterior mean, covariance): of the sensors, or of the field whose
    covariance with them is `cross`, with `prior` = (its mean, its covariance)."""
    cross, (m0, C0) = (C, (mean, C)) if cross is None else (cross, prior)
    n_o, rho = Y.shape[1], hp["rho"]
    L = torch.linalg.cholesky(C + _mismatch(pts, hp) / (rho * rho * n_o))
    X = torch.linalg.solve_triangular(L, cross.T, upper=False)
    z = torch.linalg.solve_triangular(L, (Y.mean(1) / rho - mean)[:, None], upper=False)
    return m0 + (X.T @ z)[:, 0], C0 - X.T @ X


def _np(x):
    return x.cpu().numpy() if isinstance(x, torch.Tensor) else x


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _exact_batch(case, seed)
    if case["mesh"] == "elastic" and kind == "posterior" and (case["n"] + 1) ** 3 * case["sensors"] > 4e6:
        return None  # minutes
    pr = _problem(case, seed)
    ex = _Exact(case, pr)
    if kind in ("forward", "learned"):
        return _np(ex.solve_all(ex.F[:, None])[:, 0])
    if kind == "columns":
        return ex.solve_all(_t(_columns(case, pr)).T.contiguous())
    if kind == "transpose":
        B = _t(pr["rhs"]).T.contiguous()
        X = ex.solve_all(B)
        f, c, v = ex.fc
        X.index_add_(0, c, -v[:, None] * X[f])
        return _np(X.T.contiguous())
    if kind == "gradient":
        return _exact_gradient(pr, ex)
    P, R, mean, C = ex.prior(pr)
    Y, hp, pts = _t(pr["Y"]) if "Y" in pr else None, pr["hp"], pr["pts"]
    if kind == "material":
        return _exact_material(pr, ex, P, R, C)
    C = C + (hp["forcing.sigma"] * REG) ** 2 * (P @ P.T)
    if kind == "proposals":
        return np.array([_loglik(mean, C, pts, Y, h) for h in pr["proposals"]])
    if kind == "field":
        eye = torch.eye(ex.N, dtype=torch.float64, device=_DEV)
        A = torch.zeros_like(eye)
        A[ex.free] = ex.solve(eye[ex.free])  # rows of S^-1 on the free dofs
        Cu = A @ ex.forcing(A.T.contiguous(), hp["forcing.sigma"], hp["forcing.length"])
        Cu = 0.5 * (Cu + Cu.T) + (hp["forcing.sigma"] * REG) ** 2 * eye
        m, S = _condition(mean, C, pts, Y, hp, Cu @ P.T, (ex.solve_all(ex.F[:, None])[:, 0], Cu))
        return {"mean": _np(m), "cov": _np(S)}
    m, S = _condition(mean, C, pts, Y, hp)
    return {"u": _np(ex.solve_all(ex.F[:, None])[:, 0]), "prior_mean": _np(mean), "prior_cov": _np(C),
            "loglik": _loglik(mean, C, pts, Y, hp), "mean": _np(m), "cov": _np(S)}


def _exact_batch(case, seed):
    wl = _batch_problem(case, seed)
    n, K = case["count"], api.BatchStatFEM.MAX_SENSORS
    out = dict(loglik=np.zeros(n), mean_s=np.zeros((n, K)), cov_s=np.zeros((n, K, K)), post_mean=np.zeros((n, K)),
               post_cov=np.zeros((n, K, K)))
    for k in range(n):
        P, pts = wl["sensors"][k]
        pr = dict(mesh=wl["meshes"][k], bc=wl["bcs"][k], coeff=wl["coeffs"][k], load=np.array([1.0]), P=P, pts=pts,
                  hp=wl["hps"][k])
        P, _, mean, C = _Exact(case, pr).prior(pr)
        C = C + (pr["hp"]["forcing.sigma"] * REG) ** 2 * (P @ P.T)
        Y, m = _t(wl["Y"][k]), case["sensors"]
        pm, pc = _condition(mean, C, pts, Y, pr["hp"])
        out["loglik"][k] = _loglik(mean, C, pts, Y, pr["hp"])
        out["mean_s"][k, :m], out["cov_s"][k, :m, :m] = _np(mean), _np(C)
        out["post_mean"][k, :m], out["post_cov"][k, :m, :m] = _np(pm), _np(pc)
    return dict(out, status=None)


def _exact_material(pr, ex, P, R, C):
    """First-order material covariance: sum over element pairs of
    C_m[e,d] (R dA_e) M (R dA_d)^T with M the second moment of the solution."""
    mesh, hp = pr["mesh"], pr["hp"]
    ke = _element_matrices(mesh, np.ones(mesh.num_elems))
    dofs = _element_dofs(mesh)
    ns, N, E = R.shape[1], ex.N, mesh.num_elems
    Rf = torch.where(ex.free[:, None], R, torch.zeros_like(R))
    q = torch.einsum("eia,eij->eaj", Rf[dofs], ke)  # R dA_e on the element's dofs
    Q = torch.zeros(E, ns, N, dtype=torch.float64, device=_DEV)
    Q.scatter_add_(2, dofs[:, None, :].expand(-1, ns, -1), q)
    eye = torch.eye(N, dtype=torch.float64, device=_DEV)
    A = torch.zeros_like(eye)
    A[ex.free] = ex.solve(eye[ex.free])
    u = ex.solve_all(ex.F[:, None])
    M = A @ ex.forcing(A.T.contiguous(), hp["forcing.sigma"], hp["forcing.length"]) + u @ u.T
    cent = _t(mesh.centroids()[:, :mesh.dim])
    Cm = 0.4 ** 2 * torch.exp(-((cent[:, None, :] - cent[None, :, :]) ** 2).sum(2) / (2 * 0.3 ** 2))
    QS = (Cm @ Q.reshape(E, -1)).reshape(E, ns, N)
    Cmat = torch.einsum("eaj,ebj->ab", Q @ M, QS)
    return {"mean": _np((P @ u)[:, 0]), "cov": _np(C + Cmat + (1e-4 * 0.4) ** 2 * (P @ P.T))}


def _exact_gradient(pr, ex):
    """The network's loss and gradient by automatic differentiation, unrounded."""
    N, p = ex.N, _t(pr["params"]).requires_grad_(True)
    i, v = ex.S.indices(), ex.S.values()
    num = torch.nonzero(ex.free)[:, 0]
    diag = torch.zeros(N, dtype=torch.float64, device=_DEV)
    diag[num[i[0][i[0] == i[1]]]] = v[i[0] == i[1]]
    diag[~ex.free] = 1.0  # identity rows
    si = 1 / diag.sqrt()
    rows, cols = torch.cat([num[i[0]], torch.nonzero(~ex.free)[:, 0]]), torch.cat([num[i[1]], torch.nonzero(~ex.free)[:, 0]])
    vals = torch.cat([v * si[num[i[0]]] * si[num[i[1]]], torch.ones(int((~ex.free).sum()), dtype=torch.float64, device=_DEV)])

    def ahat(x):
        return torch.zeros_like(x).index_add(0, rows, vals[:, None] * x[cols])

    t = _t(pr["res"]) * si
    s = t.norm() / math.sqrt(N)
    x0 = (t / s)[:, None]
    E, e = p[:128].reshape(64, 2), p[128:192]
    h = torch.relu(torch.cat([x0, ahat(x0)], 1) @ E.T + e)
    for layer in range(3):
        o = 192 + layer * (64 * 128 + 64)
        W, b = p[o:o + 64 * 128].reshape(64, 128), p[o + 64 * 128:o + 64 * 128 + 64]
        h = torch.relu(torch.cat([h, ahat(h)], 1) @ W.T + b)
    y = x0[:, 0] + torch.where(ex.free, h @ p[-65:-1] + p[-1], torch.zeros_like(t))
    d = (y - _t(pr["err"]) / si / s)[:, None]
    loss = (d * ahat(d)).sum() / N
    loss.backward()
    return {"loss": float(loss.detach()), "grad": _np(p.grad)}
