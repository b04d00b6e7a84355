"""What the framework is timed on: its implicit steps, and the calls those steps are made of.

Every case is work that a program has the framework do through ``opendeformer_gb300.api``:

* ``newmark`` / ``be``: a scene advanced by whole time steps from a state the program holds (a rollout: the state goes
  in, the steps run, the new state comes out), FP64 or mixed precision, alone or as a batch of uneven scenes;
* ``evaluate``: the material seam (tangent matrix and internal forces of a deformed mesh), as a host program that keeps
  its own solver calls it;
* ``pcg`` / ``spmdv``: the solver and matrix-product seams, on a matrix the program hands over.

Meshes are the jittered tetrahedral grids of ``meshgen`` at the sizes of the tests, the benchmark and its tiers: from
96 to about 1.3 million tetrahedra.  ``exact`` restates every path in plain torch (64 bits, matrix-free products per
element, no code of the framework but the mesh generator that makes the inputs).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from opendeformer_gb300 import api, meshgen

# Neo-Hookean mu 3.4e4, lambda 3.1e5 as Young's modulus and Poisson ratio (the benchmark's beam and block)
SOFT_E, SOFT_NU = 98640.0, 0.4506
DENSITY, THRESHOLD = 1000.0, 0.1
YIELD, CREEP, MAX_PLASTIC = 1e-3, 0.5, 0.05      # corotational plastic material of the tests
ALPHA_M, BETA_K = 0.01, 0.001                    # Rayleigh damping of every workload here
GRAVITY, TRACTION = -9800.0, 500.0               # N/m^3 along z; Pa along -y on the x = max face

_ctx = None


def _context():
    global _ctx
    if _ctx is None:
        _ctx = api.Context(0)
    return _ctx


def listed():
    return [
        # the smallest scene anyone steps (smoke tests, a prop in a game): launches and latency only
        dict(name="newmark_nh_96", path="newmark", nx=4, ny=2, nz=2, per_cube=6, material="neohookean", precond="block_jacobi",
             precision="fp64", tol=1e-8, newton=2, dt=1 / 120, steps=2),
        # the reference's own integrator and solver on its classic cantilever: one linearised solve a step, Jacobi
        dict(name="be_corotational_3000", path="be", nx=20, ny=5, nz=5, per_cube=6, material="corotational", precond="jacobi",
             precision="fp64", tol=1e-8, newton=1, dt=1 / 60, steps=2),
        # a mid-size plastic body on an odd grid; its plastic strain is part of the state
        dict(name="be_plastic_11k", path="be", nx=23, ny=9, nz=9, per_cube=6, material="corotational_plastic",
             precond="block_jacobi", precision="fp64", tol=1e-8, newton=1, dt=1 / 60, steps=1),
        # the benchmark's headline: the 98k-tet beam under traction, three Newton iterations a step
        dict(name="newmark_nh_beam98k", path="newmark", nx=64, ny=16, nz=16, per_cube=6, material="neohookean",
             precond="block_jacobi", precision="fp64", tol=1e-8, newton=3, dt=1 / 120, steps=1),
        # a quarter of the large compressed block, everything in FP64: matrices that leave the cache
        dict(name="newmark_nh_block655k", path="newmark", nx=128, ny=64, nz=16, per_cube=5, material="neohookean",
             precond="block_jacobi", precision="fp64", tol=1e-10, newton=1, dt=1 / 120, steps=1),
        # the mixed-precision solver on half of the large compressed block
        dict(name="newmark_nh_block1m3_mixed", path="newmark", nx=128, ny=64, nz=32, per_cube=5, material="neohookean",
             precond="block_jacobi", precision="mixed", tol=1e-10, newton=1, dt=1 / 120, steps=1),
        # many uneven scenes stepped together: corotational and Neo-Hookean, soft and stiff
        dict(name="batch_24_mixed", path="batch", scenes=24, precision="mixed", tol=1e-8, newton=1, dt=1 / 60, steps=1),
        # the incomplete Cholesky option: triangular sweeps on a beam of the benchmark's shape
        dict(name="newmark_nh_beam12k_ic0", path="newmark", nx=32, ny=8, nz=8, per_cube=6, material="neohookean",
             precond="ic0", precision="fp64", tol=1e-8, newton=2, dt=1 / 120, steps=1),
        # the material seam alone, invertible Neo-Hookean on the beam
        dict(name="evaluate_nh_98k", path="evaluate", nx=64, ny=16, nz=16, per_cube=6, material="neohookean"),
        # the material seam alone, corotational on an odd grid
        dict(name="evaluate_corotational_27k", path="evaluate", nx=37, ny=11, nz=11, per_cube=6, material="corotational"),
        # the solver seam: a matrix and a right-hand side from the host, a solution back
        dict(name="pcg_beam24k", path="pcg", nx=40, ny=10, nz=10, per_cube=6, material="corotational", precond="block_jacobi",
             precision="fp64", tol=1e-10),
        # the matrix-product seam on the beam's matrix
        dict(name="spmdv_98k", path="spmdv", nx=64, ny=16, nz=16, per_cube=6, material="corotational"),
    ]


def _dims(rng, low, high, per_cube):
    """Cube counts of a box of about low..high tetrahedra (log-uniform), longer along x; odd ones among them."""
    tets = math.exp(rng.uniform(math.log(low), math.log(high)))
    ax, ay = rng.uniform(1.0, 5.0), rng.uniform(1.0, 1.6)
    s = (tets / per_cube / (ax * ay)) ** (1.0 / 3.0)
    return max(2, round(ax * s)), max(1, round(ay * s)), max(1, round(s))


def draw(rng):
    kind = rng.choice(["newmark", "newmark", "be", "block", "mixed", "batch", "ic0", "evaluate", "evaluate", "pcg", "spmdv"])
    soft = rng.choice(["neohookean", "stvk", "corotational"])
    pc = rng.choice(["jacobi", "block_jacobi", "block_jacobi"])
    if kind in ("newmark", "be", "evaluate", "pcg", "spmdv", "ic0"):
        nx, ny, nz = _dims(rng, 96, 24e3 if kind == "ic0" else 98e3, 6)
        case = dict(path=kind, nx=nx, ny=ny, nz=nz, per_cube=6, material=soft)
        if kind == "be":
            case.update(material=rng.choice(["corotational", "corotational_plastic", "neohookean"]), precond=pc, precision="fp64",
                        tol=1e-8, newton=1, dt=1 / rng.randint(50, 70), steps=rng.randint(1, 2))
        elif kind == "newmark":
            case.update(precond=pc, precision="fp64", tol=1e-8, newton=rng.randint(2, 3), dt=1 / rng.randint(100, 140), steps=1)
        elif kind == "ic0":
            case.update(path="newmark", precond="ic0", precision="fp64", tol=1e-8, newton=2, dt=1 / rng.randint(100, 140), steps=1)
        elif kind == "pcg":
            case.update(material="corotational", precond=rng.choice(["none", "jacobi", "block_jacobi"]), precision="fp64", tol=1e-10)
        elif kind == "spmdv":
            case.update(material="corotational")
        return case
    if kind == "batch":
        return dict(path="batch", scenes=rng.randint(3, 24), precision="mixed", tol=1e-8, newton=1, dt=1 / rng.randint(50, 70), steps=1)
    nx, ny, nz = _dims(rng, 60e3, 640e3 if kind == "block" else 1.2e6, 5)
    return dict(path="newmark", nx=nx, ny=ny, nz=nz, per_cube=5, material="neohookean", precond="block_jacobi",
                precision="fp64" if kind == "block" else "mixed", tol=1e-10, newton=1, dt=1 / rng.randint(100, 140), steps=1)


# ------------------------------------------------------------------ inputs
def _mesh(case, seed):
    """The grid, its constrained DOFs and the prescribed displacements: a 6-tets-per-cube body hangs on its x = 0 face;
    a 5-tets-per-cube block stands on its bottom with a fifth of its top nodes pressed down by 5% of its height."""
    five = case["per_cube"] == 5
    h = 1.0 / case["nx"] if five else 0.05
    g = meshgen.tet_grid(case["nx"], case["ny"], case["nz"], h=h, jitter=0.2 if five else 0.15, seed=seed, tets_per_cube=case["per_cube"])
    u0 = np.zeros((g.n_nodes, 3))
    if not five:
        return g, meshgen.constrained_dofs_for_nodes(g.face_nodes(0, 0)), u0
    top = g.face_nodes(2, 1)
    pressed = np.sort(np.random.default_rng(seed).choice(top, size=max(1, top.size // 5), replace=False))
    u0[pressed, 2] = -0.05 * g.dims[2] * g.h
    return g, meshgen.constrained_dofs_for_nodes(np.concatenate([g.face_nodes(2, 0), pressed])), u0


def _fields(g, seed):
    """A smooth displacement (a few percent of an edge between neighbours, growing from the fixed face) and a smooth
    velocity, both from the seed: the state a body in motion is in."""
    rng = np.random.default_rng([seed, 1])
    size = np.maximum(g.X.max(0), 1e-9)
    out = []
    for amplitude in (0.02, 0.2):
        f = np.zeros_like(g.X)
        for _ in range(3):
            k, ph, c = rng.integers(1, 3, 3), rng.uniform(0, 2 * np.pi, 3), rng.normal(size=3)
            f += np.sin(np.pi * g.X / size * k + ph).prod(1)[:, None] * c
        out.append(amplitude * size.min() * f * (g.X[:, :1] / size[0]))
    return out


def _instances(case, seed):
    """Uneven scenes as the benchmark's batch draws them, with the sizes of a batch and the materials of the seed."""
    sizes = meshgen.batch_instances(case["scenes"])
    return [dict(i, seed=1000 * seed + k) for k, i in enumerate(sizes)]


def _material(kind, youngs=SOFT_E, poisson=SOFT_NU):
    if kind == "corotational_plastic":
        return api.CorotationalPlasticMaterial(DENSITY, youngs, poisson, YIELD, CREEP, MAX_PLASTIC, THRESHOLD)
    return api.Material(kind, DENSITY, youngs, poisson, THRESHOLD)


def _integrator(case):
    solver = api.CGSolver(case["tol"], 20000, api.Preconditioner(case.get("precond", "block_jacobi")), precision=case["precision"])
    if case["path"] == "be":
        return api.NonlinearImplicitBackwardEuler(ALPHA_M, BETA_K, case["dt"], solver)
    return api.NewmarkIntegrator(0.25, 0.5, ALPHA_M, BETA_K, case["dt"], solver, case["newton"])


def _free(n_nodes, cdofs):
    return np.setdiff1d(np.arange(3 * n_nodes), cdofs)


def _loads(case, g):
    """Gravity on what backward Euler and the batch step, surface traction on the Newmark beams, none on the block."""
    if case["path"] in ("be", "batch"):
        return dict(body=(0.0, 0.0, GRAVITY))
    if case["per_cube"] == 6:
        return dict(tractions=[([0.0, -TRACTION, 0.0], g.face_facets(0, 1))])
    return {}


def _start(case, g, free, u0, seed):
    """(mesh displacement, displacement, velocity, acceleration) of the first step; the block starts at rest."""
    u, v = _fields(g, seed)
    if case["path"] != "batch" and case["per_cube"] == 5:
        u, v = 1e-3 * u, 1e-3 * v
    u0 = u0.copy()
    u0.reshape(-1)[free] = u.reshape(-1)[free]
    return u0, u0.reshape(-1)[free].copy(), v.reshape(-1)[free].copy(), np.zeros(free.size)


def _linear_system(case, seed):
    """A matrix in the framework's value layout (mass + h^2-weighted corotational tangent of a deformed body) and two
    vectors, in plain torch, so that it is an input like any other."""
    g, cd, _ = _mesh(case, seed)
    e = _Elements(g.X, g.tets, cd, case["material"], SOFT_E, SOFT_NU)
    u, _ = _fields(g, seed)
    u = torch.as_tensor(u, device=e.device)
    u.reshape(-1)[torch.as_tensor(cd.astype(np.int64), device=e.device)] = 0.0
    K, _f, _p = e.evaluate(u, None)
    A = (1.0 / 240) ** 2 * K + e.mass()
    rng = np.random.default_rng([seed, 2])
    x = rng.normal(size=e.free.numel())
    y = rng.normal(size=e.free.numel())
    return g, cd, e, A, x, y


def prepare(case, seed):
    ctx = _context()
    if case["path"] == "batch":
        scenes, starts = [], []
        for inst in _instances(case, seed):
            g = meshgen.instance_grid(inst)
            cd = meshgen.constrained_dofs_for_nodes(g.face_nodes(0, 0))
            s = api.Scene(ctx, g.X, g.tets, g.facets, cd, _material(inst["kind"], inst["E"], inst["nu"]))
            s.set_loads(**_loads(case, g))
            s.setup_integrator(_integrator(case))
            scenes.append(s)
            starts.append(_start(case, g, _free(g.n_nodes, cd), np.zeros((g.n_nodes, 3)), inst["seed"])[1:])
        return dict(case=case, batch=api.Batch(ctx, scenes), scenes=scenes, starts=starts)
    if case["path"] in ("pcg", "spmdv"):
        g, cd, e, A, x, y = _linear_system(case, seed)
        s = api.Scene(ctx, g.X, g.tets, g.facets, cd, _material(case["material"]))
        state = dict(case=case, scene=s, values=e.packed(A).cpu().numpy(), x=x, y=y)
        if case["path"] == "pcg":
            state["solver"] = api.CGSolver(case["tol"], 20000, api.Preconditioner(case["precond"]), precision=case["precision"])
        return state
    g, cd, u0 = _mesh(case, seed)
    s = api.Scene(ctx, g.X, g.tets, g.facets, cd, _material(case["material"]))
    u0, d, v, a = _start(case, g, _free(g.n_nodes, cd), u0, seed)
    state = dict(case=case, scene=s, u=u0, d=d, v=v, a=a)
    if case["path"] != "evaluate":
        s.set_loads(**_loads(case, g))
        s.set_displacements(u0)
        s.setup_integrator(_integrator(case))
        if case["material"] == "corotational_plastic":
            s.set_state(v=v)
            state["blob"] = s.save()
    return state


# --------------------------------------------------------------------- run
def run(state):
    case = state["case"]
    path = case["path"]
    if path == "batch":
        for s, (d, v, a) in zip(state["scenes"], state["starts"]):
            s.set_state(d, v, a)
        state["batch"].step(case["steps"])
        out = [s.state() for s in state["scenes"]]
        return {k: np.concatenate([o[i] for o in out]) for i, k in enumerate(("d", "v", "a"))}
    s = state["scene"]
    if path == "evaluate":
        s.set_displacements(state["u"])
        values, forces = s.evaluate()
        return dict(values=values, forces=forces)
    if path == "spmdv":
        return dict(y=s.spmdv(state["values"], state["x"], state["y"]))
    if path == "pcg":
        return dict(x=s.pcg(state["values"], state["x"], solver=state["solver"])[0])
    if path == "be":
        if "blob" in state:                      # the checkpoint holds the plastic strain too
            s.load(state["blob"])
            s.step(case["steps"])
            return dict(u=s.displacements(), v=s.state()[1], plastic=s.plastic_strain())
        s.set_displacements(state["u"])
        s.set_state(v=state["v"])
        s.step(case["steps"])
        return dict(u=s.displacements(), v=s.state()[1])
    s.set_state(state["d"], state["v"], state["a"])
    s.step(case["steps"])
    d, v, a = s.state()
    return dict(d=d, v=v, a=a)


# -------------------------------------------------------------------- work
def _counts(nx, ny, nz, per_cube):
    tets, nodes = per_cube * nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1)
    # stored 3x3 blocks of the full matrix: a block per node and two per edge (per cube 7 edges with the Kuhn split, 6
    # with the five-tet one)
    return tets, nodes, nodes + 2 * (7 if per_cube == 6 else 6) * nx * ny * nz


def _step_work(tets, nodes, blocks, case, solves, iterations):
    """Per solve: the elements (about 1,900 operations each; 12 floats of rest shape, 4 nodes), the system's lower
    triangle written once; per solver iteration the products of the full matrix and the vector updates, on operands
    that a chip can keep.  State and node positions in and out once."""
    low = (blocks + nodes) / 2
    half = 0.5 if case["precision"] == "mixed" else 1.0
    resident = 72 * low * half < 60e6            # the matrix fits the cache next to the vectors: read once a solve
    matrix = 72 * low * half * (1 if resident else iterations)
    return {"bytes": solves * (tets * (22 * 8 + 16) + 72 * low + matrix) + 2 * 9 * 8 * nodes,
            "flops": solves * (1900 * tets + iterations * (18 * blocks + 60 * nodes))}


def work(case):
    path = case["path"]
    if path == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for i in meshgen.batch_instances(case["scenes"]):
            w = _step_work(*_counts(*i["dims"], 6), case, case["steps"] * case["newton"], 200)
            total = {k: total[k] + w[k] for k in total}
        return total
    tets, nodes, blocks = _counts(case["nx"], case["ny"], case["nz"], case["per_cube"])
    low = (blocks + nodes) / 2
    if path == "evaluate":
        return {"bytes": tets * (22 * 8 + 16) + 24 * nodes * 3 + 72 * low, "flops": 1900 * tets}
    if path == "spmdv":
        return {"bytes": 72 * low + 4 * low + 3 * 24 * nodes, "flops": 18 * blocks}
    if path == "pcg":
        return {"bytes": 72 * low + 2 * 24 * nodes, "flops": 100 * (18 * blocks + 60 * nodes)}
    # solver iterations a solve, as these systems take them: they grow with the body's length in elements
    its = {"ic0": 20}.get(case["precond"], 50 if case["per_cube"] == 6 else 400)
    return _step_work(tets, nodes, blocks, case, case["steps"] * case["newton"], its)


# ------------------------------------------------------------------- exact
def _chunked(f, M):
    """A batched decomposition of many 3x3 matrices, some thousands at a time: the libraries' workspaces stay small."""
    parts = [f(M[i:i + 16384]) for i in range(0, M.shape[0], 16384)]
    return [torch.cat(p) for p in zip(*parts)]


class _Elements:
    """Linear tetrahedra in plain torch: element matrices, forces, consistent mass, and products element by element."""

    def __init__(self, X, tets, cdofs, material, youngs, poisson):
        self.device = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.kind = material
        self.X = torch.as_tensor(np.asarray(X), dtype=torch.float64, device=self.device)
        self.t = torch.as_tensor(np.asarray(tets).astype(np.int64), device=self.device)
        self.lam = poisson * youngs / ((1 + poisson) * (1 - 2 * poisson))
        self.mu = youngs / (2 * (1 + poisson))
        n3 = self.X.numel()
        fixed = torch.zeros(n3, dtype=torch.bool, device=self.device)
        fixed[torch.as_tensor(np.asarray(cdofs).astype(np.int64), device=self.device)] = True
        self.free = torch.nonzero(~fixed).reshape(-1)
        self.n3 = n3
        self.dof = (3 * self.t[:, :, None] + torch.arange(3, device=self.device)).reshape(-1, 12)
        x = self.X[self.t]
        D = (x[:, 1:] - x[:, :1]).transpose(1, 2)                      # columns x1 - x0, x2 - x0, x3 - x0
        self.Di = torch.linalg.inv(D)
        self.V = torch.linalg.det(D).abs() / 6
        self.G = torch.cat([-self.Di.sum(1, keepdim=True), self.Di], 1)   # shape gradients, (e, 4, 3)

    # vectors live on all DOFs, zero on the fixed ones
    def spread(self, f):
        out = torch.zeros(self.n3, dtype=torch.float64, device=self.device)
        out[self.free] = torch.as_tensor(f, dtype=torch.float64, device=self.device)
        return out

    def gather(self, fe):
        out = torch.zeros(self.n3, dtype=torch.float64, device=self.device)
        out.index_add_(0, self.dof.reshape(-1), fe.reshape(-1))
        keep = torch.zeros_like(out)
        keep[self.free] = out[self.free]
        return keep

    def product(self, A, x):
        return self.gather(torch.einsum("eij,ej->ei", A, x[self.dof]))

    def mass(self):
        m = (torch.ones(4, 4) + torch.eye(4)).to(self.X) / 20
        M = DENSITY * self.V[:, None, None] * m
        return torch.einsum("eab,ij->eaibj", M, torch.eye(3).to(self.X)).reshape(-1, 12, 12)

    def body(self, b):
        w = torch.zeros(self.X.shape[0], dtype=torch.float64, device=self.device)
        w.index_add_(0, self.t.reshape(-1), (self.V / 4).repeat_interleave(4))
        return (w[:, None] * torch.tensor(b, dtype=torch.float64, device=self.device)).reshape(-1)

    def traction(self, t, facets):
        f = torch.as_tensor(np.asarray(facets).astype(np.int64), device=self.device)
        p = self.X[f]
        area = torch.linalg.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]).norm(dim=1) / 2
        out = torch.zeros_like(self.X)
        out.index_add_(0, f.reshape(-1), (area / 3).repeat_interleave(3)[:, None] * torch.tensor(t, dtype=torch.float64, device=self.device))
        return out.reshape(-1)

    def evaluate(self, u, plastic):
        """(element matrices (e, 12, 12), internal forces on all DOFs, the plastic strain after the evaluation)."""
        c = (self.X + u.reshape(-1, 3))[self.t]
        Ds = (c[:, 1:] - c[:, :1]).transpose(1, 2)
        F = Ds @ self.Di
        if self.kind in ("neohookean", "stvk"):
            return self._hyperelastic(F) + (None,)
        R = self._rotation(F, torch.linalg.det(Ds).abs() / 6)
        g = self.G
        eye = torch.eye(3).to(self.X)
        K0 = self.V[:, None, None, None, None] * (
            self.lam * torch.einsum("eai,ebj->eabij", g, g) + self.mu * torch.einsum("eaj,ebi->eabij", g, g)
            + self.mu * torch.einsum("eab,ij->eabij", g @ g.transpose(1, 2), eye))
        K = torch.einsum("eik,eabkl,ejl->eaibj", R, K0, R).reshape(-1, 12, 12)
        if self.kind == "corotational":
            y = torch.einsum("eki,ebk->ebi", R, c) - self.X[self.t]      # R^T c - X
            f = torch.einsum("eik,eak->eai", R, torch.einsum("eabkl,ebl->eak", K0, y))
            return K, self.gather(f.reshape(-1, 12)), None
        S = R.transpose(1, 2) @ F
        strain = 0.5 * (S + S.transpose(1, 2)) - eye - plastic
        stress = 2 * self.mu * strain + self.lam * strain.diagonal(dim1=1, dim2=2).sum(1)[:, None, None] * eye
        f = self.V[:, None, None] * torch.einsum("eij,eaj->eai", R @ stress, g)
        # the material's norms take the first row's squares three times
        size = (3 * strain[:, 0].square().sum(1)).sqrt()
        grown = plastic + torch.where(size > YIELD, CREEP * (size - YIELD) / size.clamp_min(1e-300), torch.zeros_like(size))[:, None, None] * strain
        norm = (3 * grown[:, 0].square().sum(1)).sqrt()
        cut = torch.where((size > YIELD) & (norm > MAX_PLASTIC), MAX_PLASTIC / norm.clamp_min(1e-300), torch.ones_like(norm))
        return K, self.gather(f.reshape(-1, 12)), grown * cut[:, None, None]

    def _rotation(self, F, volume):
        U, s, Vh = _chunked(torch.linalg.svd, F)
        R = U @ Vh
        crushed = volume < THRESHOLD * self.V
        if bool(crushed.any()):                                       # Gram-Schmidt, a proper rotation
            Q, T = _chunked(torch.linalg.qr, F[crushed])
            Q = Q * torch.where(T.diagonal(dim1=1, dim2=2) < 0, -1.0, 1.0)[:, None, :]
            Q[:, :, 2] = torch.linalg.cross(Q[:, :, 0], Q[:, :, 1])
            R[crushed] = Q
        return R

    def _hyperelastic(self, F):
        U, s, Vh = _chunked(torch.linalg.svd, F)
        for M in (U, Vh):                                             # proper rotations; a reflection goes to the last value
            flip = torch.linalg.det(M) < 0
            s[flip, 2] = -s[flip, 2]
            if M is U:
                M[flip, :, 2] = -M[flip, :, 2]
            else:
                M[flip, 2] = -M[flip, 2]
        s = s.clamp_min(THRESHOLD)
        s2, I3 = s * s, (s * s).prod(1)
        zero = torch.zeros_like(I3)
        if self.kind == "neohookean":
            g0, g1, h0 = zero + 0.5 * self.mu, zero, zero
            g2 = (-0.5 * self.mu + 0.25 * self.lam * I3.log()) / I3
            h5 = (0.5 * self.mu + 0.25 * self.lam * (1 - I3.log())) / I3 ** 2
        else:
            g0 = 0.25 * self.lam * (s2.sum(1) - 3) - 0.5 * self.mu
            g1, g2, h0, h5 = zero + 0.25 * self.mu, zero, zero + 0.25 * self.lam, zero
        col = lambda q: q[:, None, None]                              # noqa: E731
        outer = s[:, :, None] * s[:, None, :]
        d = col(I3 * g2) / outer
        al = 2 * col(g0) + 4 * (s2[:, :, None] + s2[:, None, :]) * col(g1)
        be = 4 * outer * col(g1) - 2 * d
        w0, w2 = 2 * s, 2 * I3[:, None] / s
        T = 4 * d + col(h0) * w0[:, :, None] * w0[:, None, :] + col(h5) * w2[:, :, None] * w2[:, None, :]
        T = T + torch.diag_embed((al + be).diagonal(dim1=1, dim2=2))
        ev, Q = _chunked(torch.linalg.eigh, T)
        T = torch.where(col((ev < 0).any(1)), Q @ (ev.clamp_min(0)[:, :, None] * Q.transpose(1, 2)), T)
        sym, anti = (al + be).clamp_min(0), (al - be).clamp_min(0)    # the 2x2 blocks' eigenvalues
        al, be = 0.5 * (sym + anti), 0.5 * (sym - anti)
        off = (1 - torch.eye(3)).to(self.X)
        P = U @ ((2 * g0[:, None] * s + 4 * g1[:, None] * s ** 3 + w2 * g2[:, None])[:, :, None] * Vh)
        f = self.V[:, None, None] * torch.einsum("eij,eaj->eai", P, self.G)
        a = torch.einsum("eij,eaj->eai", Vh, self.G)                  # gradients in the singular frame
        n = torch.einsum("eij,eai,ebj->eabij", T, a, a) + torch.einsum("eij,eaj,ebi->eabij", be * off, a, a)
        n = n + torch.diag_embed(torch.einsum("eik,eak,ebk->eabi", al * off, a, a))
        K = torch.einsum("eik,eabkl,ejl->eaibj", U, n, U) * self.V[:, None, None, None, None]
        return K.reshape(-1, 12, 12), self.gather(f.reshape(-1, 12))

    def packed(self, A):
        """Element matrices summed in the framework's value layout: block columns of the free nodes, per column its
        diagonal block's six lower values by columns, then the blocks below it, nine values each by columns.  On the
        host, where the order of the additions is always the same."""
        A, t, free = A.cpu(), self.t.cpu(), self.free.cpu()
        node = torch.full((self.X.shape[0],), -1, dtype=torch.int64)
        ids = free[::3] // 3
        node[ids] = torch.arange(ids.numel())
        p = node[t]
        a, b = torch.triu_indices(4, 4)
        pa, pb = p[:, a], p[:, b]
        blocks = A.reshape(-1, 4, 3, 4, 3)[:, a, :, b, :].transpose(0, 1)       # (e, 10, 3, 3), rows of node a
        swap = pa < pb
        blocks = torch.where(swap[:, :, None, None], blocks.transpose(2, 3), blocks)
        use = (pa >= 0) & (pb >= 0)
        key = torch.minimum(pa, pb) * ids.numel() + torch.maximum(pa, pb)
        keys, inverse = torch.unique(key[use], return_inverse=True)              # by column, then by row
        total = torch.zeros((keys.numel(), 9), dtype=torch.float64)
        total.index_add_(0, inverse, blocks[use].transpose(1, 2).reshape(-1, 9))
        lower = torch.tensor([True, True, True, False, True, True, False, False, True])
        diagonal = (keys // ids.numel()) == (keys % ids.numel())
        return total[torch.where(diagonal[:, None], lower, torch.ones_like(lower))]

    def solve(self, A, b, tol=1e-14, most=20000):
        """Conjugate gradients on element products, 3x3 diagonal blocks inverted, to the rounding of 64 bits."""
        blk = torch.zeros((self.n3 // 3, 3, 3), dtype=torch.float64, device=self.device)
        d = A.reshape(-1, 4, 3, 4, 3).diagonal(dim1=1, dim2=3).permute(0, 3, 1, 2)
        blk.index_add_(0, self.t.reshape(-1), d.reshape(-1, 3, 3))
        inv = torch.linalg.inv(blk)

        def pre(r):
            z = (inv @ r.reshape(-1, 3, 1)).reshape(-1)
            keep = torch.zeros_like(z)
            keep[self.free] = z[self.free]
            return keep

        x = torch.zeros_like(b)
        for _ in range(2):                                            # once more from the true residual
            r = b - self.product(A, x)
            z = pre(r)
            p, rz, stop = z.clone(), torch.dot(r, z), (tol * b.norm()) ** 2
            for k in range(most):
                q = self.product(A, p)
                alpha = rz / torch.dot(p, q)
                x = x + alpha * p
                r = r - alpha * q
                if k % 16 == 15 and float(torch.dot(r, r)) <= float(stop):
                    break
                z = pre(r)
                new = torch.dot(r, z)
                p = z + (new / rz) * p
                rz = new
        return x


def _external(case, g, e):
    loads = _loads(case, g)
    f = torch.zeros(e.n3, dtype=torch.float64, device=e.device)
    if "body" in loads:
        f = f + e.body(loads["body"])
    for t, ids in loads.get("tractions", ()):
        f = f + e.traction(t, g.facets[ids])
    return e.spread(f[e.free])


def _newmark(case, g, e, u0, start):
    h, gamma, beta = case["dt"], 0.5, 0.25
    fixed = torch.as_tensor(u0, device=e.device).reshape(-1).clone()
    fixed[e.free] = 0.0
    d, v, a = (e.spread(q) for q in start)
    fext, M = _external(case, g, e), e.mass()
    for _ in range(case["steps"]):
        dp, vp = d + h * v + (0.5 - beta) * h * h * a, v + (1 - gamma) * h * a
        for _ in range(case["newton"]):
            K, fint, _p = e.evaluate(fixed + dp + beta * h * h * a, None)
            vk = vp + gamma * h * a
            r = fext - fint - e.product(M, ALPHA_M * vk + a) - BETA_K * e.product(K, vk)
            a = a + e.solve((1 + gamma * h * ALPHA_M) * M + (gamma * h * BETA_K + beta * h * h) * K, r)
        d, v = dp + beta * h * h * a, vp + gamma * h * a
    return {k: q[e.free].cpu() for k, q in (("d", d), ("v", v), ("a", a))}


def _backward_euler(case, g, e, u0, v):
    h = case["dt"]
    u, v = torch.as_tensor(u0, device=e.device).reshape(-1).clone(), e.spread(v)
    fext, M = _external(case, g, e), e.mass()
    plastic = torch.zeros((e.t.shape[0], 3, 3), dtype=torch.float64, device=e.device)
    for _ in range(case["steps"]):
        K, fint, plastic = e.evaluate(u, plastic)
        A0 = (h + BETA_K) * K + ALPHA_M * M
        v = v + e.solve(h * A0 + M, h * (fext - fint - e.product(A0, v)))
        u = u + h * v
    out = dict(u=u.reshape(-1, 3).cpu(), v=v[e.free].cpu())
    if case["material"] == "corotational_plastic":
        out["plastic"] = plastic.reshape(-1, 9).cpu()
    return out


def exact(case, seed):
    path = case["path"]
    if path == "batch":
        parts = []
        for inst in _instances(case, seed):
            g = meshgen.instance_grid(inst)
            cd = meshgen.constrained_dofs_for_nodes(g.face_nodes(0, 0))
            e = _Elements(g.X, g.tets, cd, inst["kind"], inst["E"], inst["nu"])
            u0, *start = _start(case, g, _free(g.n_nodes, cd), np.zeros((g.n_nodes, 3)), inst["seed"])
            parts.append(_newmark(case, g, e, np.zeros_like(u0), start))
        return {k: torch.cat([p[k] for p in parts]) for k in ("d", "v", "a")}
    if path in ("pcg", "spmdv"):
        _g, _cd, e, A, x, y = _linear_system(case, seed)
        if path == "pcg":
            return dict(x=e.solve(A, e.spread(x))[e.free].cpu())
        return dict(y=(e.product(A, e.spread(x)) + e.spread(y))[e.free].cpu())
    g, cd, u0 = _mesh(case, seed)
    e = _Elements(g.X, g.tets, cd, case["material"], SOFT_E, SOFT_NU)
    u0, d, v, a = _start(case, g, _free(g.n_nodes, cd), u0, seed)
    if path == "evaluate":
        K, f, _p = e.evaluate(torch.as_tensor(u0, device=e.device).reshape(-1), None)
        return dict(values=e.packed(K).cpu(), forces=f[e.free].cpu())
    if path == "be":
        return _backward_euler(case, g, e, u0, v)
    return _newmark(case, g, e, u0, (d, v, a))
