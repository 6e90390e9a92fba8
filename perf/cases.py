"""The work a user of topomax_gb300 has it do, as measurable cases.

Kinds of case (each through the package's public classes):

* ``elastic`` -- one design evaluation: ``ElasticityProblem.calculate_objective`` (Helmholtz
  filter, P2 state solve, compliance) and ``calculate_objective_gradient`` (sensitivity and its
  filter), from a design the problem has not seen (no warm start), the step every design loop,
  parameter sweep and gradient check repeats;
* ``loop`` -- ``FEMSolver.solve``: the whole mirror-descent loop with its warm starts,
  projections and stopping rules, a few iterations from a given design (plain FP64);
* ``filter`` -- ``HelmholtzFilter.apply`` by itself;
* ``dem`` -- the deep-energy-method's training evaluation: the masked strain energy with its
  gradients with respect to the displacement and the density, and the objective with its
  per-cell gradient;
* ``dem_filter`` -- the deep-energy-method's density filter, W rho and W^T g;
* ``fluid`` -- one design evaluation of the Stokes-Brinkman problem: state, objective, gradient.

Designs come from smooth random fields pushed through the logistic function to a given volume,
as the mirror-descent iterates are: ``contrast`` 0 is the uniform start, larger values stand for
later, nearly 0/1 designs.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import topomax_gb300 as tg
from topomax_gb300 import dem as tgdem
from topomax_gb300.designs import parse_design_dict

F64 = torch.float64
PMIN = 1e-6


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _elastic(nx, ny, design, contrast, precision="mixed"):
    # tolerances tight enough for a gradient check: the outputs are then the equations' solution
    rtol = 1e-10 if precision == "fp64" else 1e-12 if ny < 200 else 1e-11
    return {"kind": "elastic", "nx": nx, "ny": ny, "design": design, "contrast": contrast,
            "precision": precision, "rtol": rtol}


def listed():
    return [
        # the reference's own N = 40 cantilever: launch-bound, the size of a quick study
        dict(_elastic(80, 40, "cantilever", 2.0), name="elastic_80x40"),
        # an odd-sized 3 x 1 cantilever under a body force (N = 101), every level padded
        dict(_elastic(303, 101, "long_cantilever", 2.0), name="elastic_303x101"),
        # the 4M-dof headline grid
        dict(_elastic(1000, 500, "cantilever", 2.0), name="elastic_1000x500"),
        # the 16M-dof throughput grid
        dict(_elastic(2000, 1000, "cantilever", 1.5), name="elastic_2000x1000"),
        # the reference's N = 160 cantilever
        dict(_elastic(320, 160, "cantilever", 2.0), name="elastic_320x160"),
        # the whole design loop at the reference's N = 80, in plain FP64 (how the mixed path is checked)
        {"kind": "loop", "N": 80, "iterations": 6, "contrast": 0.5, "rtol": 1e-11, "name": "loop_fp64_160x80"},
        # the density filter of the headline grid by itself
        {"kind": "filter", "nx": 1000, "ny": 500, "radius": 0.05, "contrast": 2.0, "rtol": 1e-10,
         "name": "filter_1000x500"},
        # one training evaluation of the reference's short cantilever (N = 45): microseconds, launch-bound
        {"kind": "dem", "nx": 90, "ny": 45, "name": "dem_90x45"},
        # the 600 x 300 deep-energy workload
        {"kind": "dem", "nx": 600, "ny": 300, "name": "dem_600x300"},
        # its density filter (radius 2 sqrt 3 times the Helmholtz radius)
        {"kind": "dem_filter", "nx": 600, "ny": 300, "radius": 0.05 * 2 * math.sqrt(3), "name": "dem_filter_600x300"},
        # the reference's fluid diffuser at N = 40 and a finer one
        {"kind": "fluid", "n": 40, "contrast": 1.0, "rtol": 1e-12, "name": "fluid_40"},
        {"kind": "fluid", "n": 128, "contrast": 2.0, "rtol": 1e-12, "name": "fluid_128"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["elastic", "elastic", "elastic", "loop", "filter", "dem", "dem", "dem_filter", "fluid", "fluid"])
    if kind == "elastic":
        design = rng.choice(["cantilever", "cantilever", "long_cantilever"])
        precision = rng.choice(["mixed", "mixed", "mixed", "fp64"])
        ny = _log_int(rng, 20, 800 if precision == "mixed" else 200)
        width = 2 if design == "cantilever" else 3
        nx = min(width * ny + rng.randrange(-7, 8), 1600)
        while nx * (width / nx) != width:  # a traction acts where a mesh coordinate equals the width exactly
            nx -= 1
        return _elastic(nx, ny, design, round(rng.uniform(0.0, 3.0), 2), precision)
    if kind == "loop":
        return {"kind": "loop", "N": _log_int(rng, 20, 160), "iterations": rng.randrange(3, 9),
                "contrast": round(rng.uniform(0.0, 1.0), 2), "rtol": 1e-11}
    if kind == "filter":
        ny = _log_int(rng, 30, 1000)
        return {"kind": "filter", "nx": 2 * ny + rng.randrange(-7, 8), "ny": ny, "radius": rng.choice([0.02, 0.05]),
                "contrast": round(rng.uniform(0.0, 3.0), 2), "rtol": 1e-10}
    if kind == "dem":
        ny = _log_int(rng, 20, 400)
        return {"kind": "dem", "nx": 2 * ny + rng.randrange(-7, 8), "ny": ny}
    if kind == "dem_filter":
        ny = _log_int(rng, 20, 250)
        return {"kind": "dem_filter", "nx": 2 * ny + rng.randrange(-7, 8), "ny": ny,
                "radius": rng.choice([0.02, 0.05]) * 2 * math.sqrt(3)}
    return {"kind": "fluid", "n": _log_int(rng, 16, 110), "contrast": round(rng.uniform(0.0, 2.0), 2), "rtol": 1e-12}


# ---------------------------------------------------------------------------
# designs and inputs
# ---------------------------------------------------------------------------
def _elastic_dict(name):
    if name == "cantilever":  # the package's 2 x 1 cantilever
        dom = dict(width=2.0, height=1.0, fem_step_size=0.002, dem_step_size=0.002, penalties=[3.0],
                   volume_fraction=0.5)
        par = dict(fixed_sides=["Left"], body_force=None,
                   tractions=[dict(side="Right", center=0.5, length=0.5, value=[0.0, -1.0])],
                   filter_radius=0.05, young_modulus=1.0, poisson_ratio=0.3)
    else:  # the reference's 3 x 1 cantilever
        dom = dict(width=3.0, height=1.0, fem_step_size=25.0, dem_step_size=37500.0, penalties=[3.0],
                   volume_fraction=0.5)
        par = dict(fixed_sides=["Left"], body_force=dict(region=dict(center=[2.9, 0.5], radius=0.05), value=[0.0, -1.0]),
                   tractions=None, filter_radius=0.02, young_modulus=2.5, poisson_ratio=0.25)
    return {"Elasticity": {"domain_parameters": dom, "problem_parameters": par}}


def _fluid_dict():  # the reference's diffuser
    return {"Fluid": {
        "domain_parameters": dict(width=1.0, height=1.0, fem_step_size=0.0011, dem_step_size=0.0002, penalties=[0.1],
                                  volume_fraction=0.5),
        "problem_parameters": dict(flows=[dict(side="Left", center=0.5, length=1.0, rate=1.0),
                                          dict(side="Right", center=0.5, length=1.0 / 3.0, rate=-3.0)],
                                   viscosity=1.0)}}


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _grid_xy(width, height, nx, ny):
    x = torch.arange(nx + 1, device="cuda", dtype=F64) * (width / nx)
    y = torch.arange(ny + 1, device="cuda", dtype=F64) * (height / ny)
    return x[None, :], y[:, None]


def _waves(g, x, y, count=10):
    c = torch.rand((count, 4), generator=g, device="cuda", dtype=F64)
    f = 0
    for k in range(count):
        f = f + c[k, 0] * torch.sin(2 * math.pi * (4 * c[k, 1] * x + 4 * c[k, 2] * y + c[k, 3]))
    return f


def _to_volume(psi, volume_fraction):
    """logistic(psi + c) with the given mean (bisection on the device, no host reads)."""
    lo = torch.full((), -80.0, device="cuda", dtype=F64)
    hi = torch.full((), 80.0, device="cuda", dtype=F64)
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        above = torch.sigmoid(psi + mid).mean() > volume_fraction
        lo, hi = torch.where(above, lo, mid), torch.where(above, mid, hi)
    return torch.sigmoid(psi + lo).reshape(-1).contiguous()


def _design_field(seed, width, height, nx, ny, contrast, volume_fraction):
    """A random smooth design with material kept where the load acts, on the right at mid-height,
    as any iterate of the loop has it."""
    x, y = _grid_xy(width, height, nx, ny)
    load = 3.0 * torch.exp(-((x - width + 0.1) ** 2 + (y - 0.5 * height) ** 2) / 0.06)
    # a little noise also at contrast 0: the start is uniform up to small changes
    return _to_volume((contrast + 1e-3) * (_waves(_generator(seed), x, y) + load), volume_fraction)


def _mesh(case):
    width = 3.0 if case.get("design") == "long_cantilever" else 2.0
    return tg.RectangleMesh(width, 1.0, case["nx"], case["ny"])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "elastic":
        dom, par = parse_design_dict(_elastic_dict(case["design"]))
        mesh = _mesh(case)
        problem = tg.ElasticityProblem(mesh, tg.FunctionSpace(mesh, "CG", 1), dom, par, precision=case["precision"],
                                       rtol=case["rtol"], warm_start=False)
        problem.set_penalization(3.0)
        rho = _design_field(seed, mesh.width, mesh.height, mesh.nx, mesh.ny, case["contrast"], dom.volume_fraction)
        return {"kind": kind, "problem": problem, "rho": rho}
    if kind == "loop":
        solver = tg.FEMSolver(case["N"], dict(_elastic_dict("cantilever"), name="cantilever"),
                              precision="fp64", rtol=case["rtol"], verbose=False, save=False,
                              max_iterations=case["iterations"])
        m = solver.mesh
        rho = _design_field(seed, m.width, m.height, m.nx, m.ny, case["contrast"], solver.parameters.volume_fraction)
        return {"kind": kind, "solver": solver, "rho": rho}
    if kind == "filter":
        mesh = _mesh(case)
        filt = tg.HelmholtzFilter(case["radius"], tg.FunctionSpace(mesh, "CG", 1), rtol=case["rtol"])
        return {"kind": kind, "filter": filt,
                "rho": _design_field(seed, 2.0, 1.0, mesh.nx, mesh.ny, case["contrast"], 0.5)}
    if kind == "dem":
        nx, ny = case["nx"], case["ny"]
        mesh = tgdem.Mesh(nx, ny, 2.0, 1.0)
        _, par = parse_design_dict(_dem_dict())
        enforcer = tgdem.ElasticityEnforcer(par, mesh)
        energy = tgdem.StrainEnergy(mesh, None, par.young_modulus, par.poisson_ratio,
                                    [tgdem.TractionPoints(mesh, t) for t in par.tractions])
        energy.set_penalization(3.0)
        u, rho = _dem_inputs(seed, nx, ny)
        return {"kind": kind, "mesh": mesh, "enforcer": enforcer, "energy": energy,
                "u": u.requires_grad_(True), "rho": rho.requires_grad_(True)}
    if kind == "dem_filter":
        mesh = tgdem.Mesh(case["nx"], case["ny"], 2.0, 1.0)
        rho, g = _dem_filter_inputs(seed, case["nx"], case["ny"])
        return {"kind": kind, "filter": tgdem.create_density_filter(case["radius"], mesh), "rho": rho, "g": g}
    dom, par = parse_design_dict(_fluid_dict())
    mesh = tg.RectangleMesh(1.0, 1.0, case["n"], case["n"])
    problem = tg.FluidProblem(mesh, par, dom, rtol=case["rtol"])
    problem.set_penalization(0.1)
    return {"kind": kind, "problem": problem, "rho": _fluid_design(seed, case["n"], case["contrast"])}


def run(state):
    kind = state["kind"]
    if kind == "elastic":
        p = state["problem"]
        objective = p.calculate_objective(state["rho"])
        gradient = p.calculate_objective_gradient()
        return {"objective": objective, "u": p.u.tensor, "filtered": p.filtered_rho.tensor,
                "gradient": gradient.tensor}
    if kind == "loop":
        s = state["solver"]
        s.rho.tensor.copy_(state["rho"])
        history = s.solve()
        return {"objectives": history[3.0]["objectives"], "rho": s.rho.tensor}
    if kind == "filter":
        return state["filter"].apply(state["rho"]).tensor
    if kind == "dem":
        energy, u, rho = state["energy"], state["u"], state["rho"]
        psi = energy.calculate_energy_enforced(u, state["enforcer"], rho)
        du, drho = torch.autograd.grad(psi, (u, rho))
        objective, gradient = energy.calculate_objective_and_gradient(u, state["mesh"].shape, rho)
        return {"psi": psi, "du": du, "drho": drho, "objective": objective, "gradient": gradient}
    if kind == "dem_filter":
        f = state["filter"]
        return {"filtered": f @ state["rho"], "back": f.T @ state["g"]}
    p = state["problem"]
    objective = p.calculate_objective(state["rho"])
    gradient = p.calculate_objective_gradient()
    return {"objective": objective, "u": p.u.tensor, "p": p.p.tensor, "gradient": gradient.tensor}


def work(case):
    """Inputs read once and outputs written once; floating operations of one application of each
    operator on the path (an iterative solve cannot do with less)."""
    kind = case["kind"]
    if kind in ("elastic", "loop"):
        nx, ny = (case["nx"], case["ny"]) if kind == "elastic" else (2 * case["N"], case["N"])
        n = 1 if kind == "elastic" else case["iterations"] + 1
        nv, n2 = (nx + 1) * (ny + 1), (2 * nx + 1) * (2 * ny + 1)
        return {"bytes": 8.0 * n * (3 * nv + 2 * n2), "flops": 400.0 * n * nx * ny}
    if kind == "filter":
        nv = (case["nx"] + 1) * (case["ny"] + 1)
        return {"bytes": 16.0 * nv, "flops": 28.0 * nv}
    if kind == "dem":
        nc, nn = case["nx"] * case["ny"], (case["nx"] + 1) * (case["ny"] + 1)
        return {"bytes": 4.0 * (4 * nn + 3 * nc), "flops": 500.0 * nc}
    if kind == "dem_filter":
        nc = case["nx"] * case["ny"]
        return {"bytes": 32.0 * nc, "flops": 4.0 * nc * math.pi * case["radius"] ** 2 * nc / 2.0}
    n = case["n"]
    nv, n2 = (n + 1) ** 2, (2 * n + 1) ** 2
    return {"bytes": 8.0 * (3 * nv + 2 * n2), "flops": 600.0 * n * n}


# ---------------------------------------------------------------------------
# inputs of the deep-energy and fluid cases
# ---------------------------------------------------------------------------
def _dem_dict():
    d = _elastic_dict("cantilever")
    d["Elasticity"]["problem_parameters"]["tractions"][0]["length"] = 1.0  # the whole right side
    return d


def _dem_inputs(seed, nx, ny):
    """A network's output (smooth, O(1)) on the nodes in x-major order, and a cell density."""
    g = _generator(seed)
    x, y = _grid_xy(2.0, 1.0, nx, ny)
    u = torch.stack([(0.1 * _waves(g, x, y, 6)).expand(ny + 1, nx + 1).T.reshape(-1) for _ in range(2)], dim=1)
    xc = (torch.arange(nx, device="cuda", dtype=F64) + 0.5) * (2.0 / nx)
    yc = (torch.arange(ny, device="cuda", dtype=F64) + 0.5) * (1.0 / ny)
    rho = _to_volume(2.0 * _waves(g, xc[None, :], yc[:, None]), 0.5).reshape(ny, nx)
    return u.float().contiguous(), rho.float().contiguous()


def _dem_filter_inputs(seed, nx, ny):
    g = _generator(seed)
    xc = torch.linspace(0.0, 2.0, nx, device="cuda", dtype=F64)
    yc = torch.linspace(0.0, 1.0, ny, device="cuda", dtype=F64)
    rho = _to_volume(2.0 * _waves(g, xc[None, :], yc[:, None]), 0.5)
    return rho, -_waves(g, xc[None, :], yc[:, None]).square().reshape(-1).contiguous()


def _fluid_design(seed, n, contrast):
    """High density in the tapering channel between inflow and outflow, random detail on top."""
    x, y = _grid_xy(1.0, 1.0, n, n)
    channel = 4.0 * ((0.5 - x / 3.0) - (y - 0.5).abs())
    return _to_volume(contrast * channel + (0.3 * contrast + 1e-3) * _waves(_generator(seed), x, y), 0.5)


# ---------------------------------------------------------------------------
# the same results from plain torch and numpy in 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind == "elastic":
        if case["ny"] * case["ny"] * case["ny"] * case["nx"] > 1.3e9:  # minutes of block eliminations
            return None
        ref = _Elastic(case["design"], case["nx"], case["ny"])
        rho = _design_field(seed, ref.W, ref.H, ref.nx, ref.ny, case["contrast"], 0.5)
        objective, u, xi = ref.state(rho)
        return {"objective": objective, "u": u, "filtered": xi, "gradient": ref.gradient(u, xi)}
    if kind == "loop":
        if case["N"] > 100:
            return None
        ref = _Elastic("cantilever", 2 * case["N"], case["N"])
        rho = _design_field(seed, ref.W, ref.H, ref.nx, ref.ny, case["contrast"], 0.5)
        return _loop_exact(ref, rho, case["iterations"])
    if kind == "filter":
        if case["nx"] * case["ny"] ** 3 > 4e12:
            return None
        nx, ny = case["nx"], case["ny"]
        rho = _design_field(seed, 2.0, 1.0, nx, ny, case["contrast"], 0.5)
        return _Cg1(2.0, 1.0, nx, ny, case["radius"]).filter(rho)
    if kind == "dem":
        return _dem_exact(case, seed)
    if kind == "dem_filter":
        return _dem_filter_exact(case, seed)
    return _fluid_exact(case, seed) if case["n"] <= 44 else None


class _BlockTridiagonal:
    """Factors and solves a block-tridiagonal system given by its blocks (nb, m, m), one step
    of iterative refinement per solve."""

    def __init__(self, lower, diag, upper):
        self.lower, self.diag, self.upper = lower, diag, upper
        self.lu = []
        nb = diag.shape[0]
        d = diag[0]
        for i in range(nb):
            self.lu.append(torch.linalg.lu_factor(d))
            if i + 1 < nb:
                d = diag[i + 1] - lower[i] @ torch.linalg.lu_solve(*self.lu[i], upper[i])

    def _solve(self, b):
        nb = b.shape[0]
        y = [b[0]]
        for i in range(1, nb):
            y.append(b[i] - self.lower[i - 1] @ torch.linalg.lu_solve(*self.lu[i - 1], y[i - 1][:, None])[:, 0])
        x = [None] * nb
        for i in reversed(range(nb)):
            r = y[i] if i + 1 == nb else y[i] - self.upper[i] @ x[i + 1]
            x[i] = torch.linalg.lu_solve(*self.lu[i], r[:, None])[:, 0]
        return torch.stack(x)

    def _times(self, x):
        y = torch.einsum("nij,nj->ni", self.diag, x)
        y[:-1] += torch.einsum("nij,nj->ni", self.upper, x[1:])
        y[1:] += torch.einsum("nij,nj->ni", self.lower, x[:-1])
        return y

    def solve(self, b):
        x = self._solve(b)
        return x + self._solve(b - self._times(x))


def _triangle_rule(n):
    """Collapsed Gauss-Legendre rule with n x n points (exact to degree 2n - 2): barycentric
    points, weights summing to 1."""
    t, w = np.polynomial.legendre.leggauss(n)
    t, w = 0.5 * (t + 1), 0.5 * w
    pts, wts = [], []
    for a, wa in zip(t, w):
        for b, wb in zip(t, w):
            pts.append((1 - a, a * (1 - b), a * b))
            wts.append(2 * wa * wb * a)
    return np.array(pts), np.array(wts)


# vertices of the two triangles of a cell (half-cell offsets), then their P2 nodes
# [A, B, C, mid BC, mid AC, mid AB]
_TRI = (((0, 0), (2, 0), (2, 2), (2, 1), (1, 1), (1, 0)), ((0, 0), (0, 2), (2, 2), (1, 2), (1, 1), (0, 1)))


def _p2_basis(lam, G):
    l0, l1, l2 = lam.T
    N = np.stack([l0 * (2 * l0 - 1), l1 * (2 * l1 - 1), l2 * (2 * l2 - 1), 4 * l1 * l2, 4 * l0 * l2, 4 * l0 * l1], 1)
    dl = lambda a, b: 4 * (lam[:, a, None] * G[b] + lam[:, b, None] * G[a])  # noqa: E731
    dN = np.stack([(4 * l0 - 1)[:, None] * G[0], (4 * l1 - 1)[:, None] * G[1], (4 * l2 - 1)[:, None] * G[2],
                   dl(1, 2), dl(0, 2), dl(0, 1)], 1)
    return N, dN


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda")


class _Lattice:
    """Index arrays and triangle geometry of the structured mesh (right diagonals)."""

    def __init__(self, W, H, nx, ny):
        self.W, self.H, self.nx, self.ny = W, H, nx, ny
        self.hx, self.hy = W / nx, H / ny
        self.area = 0.5 * self.hx * self.hy
        self.nv, self.n2 = (nx + 1) * (ny + 1), (2 * nx + 1) * (2 * ny + 1)
        j, i = torch.meshgrid(torch.arange(ny, device="cuda"), torch.arange(nx, device="cuda"), indexing="ij")
        i, j = i.reshape(-1), j.reshape(-1)
        self.vert, self.node, self.G = [], [], []
        for o in (0, 1):
            self.vert.append(torch.stack([(j + b // 2) * (nx + 1) + i + a // 2 for a, b in _TRI[o][:3]], 1))
            self.node.append(torch.stack([(2 * j + b) * (2 * nx + 1) + 2 * i + a for a, b in _TRI[o]], 1))
            P = np.array([(a * self.hx / 2, b * self.hy / 2) for a, b in _TRI[o][:3]])
            E = np.stack([P[1] - P[0], P[2] - P[0]])
            g = np.linalg.inv(E)  # columns: gradients of the barycentric coordinates 1 and 2
            self.G.append(np.stack([-(g[:, 0] + g[:, 1]), g[:, 0], g[:, 1]]))


class _Cg1(_Lattice):
    """CG1 mass matrix and the Helmholtz filter (eps^2 K + M)."""

    def __init__(self, W, H, nx, ny, eps):
        super().__init__(W, H, nx, ny)
        Me = self.area / 12.0 * (np.ones((3, 3)) + np.eye(3))
        self.Me = _dev(Me)
        m = ny + 1
        D = torch.zeros((nx + 1, m, m), device="cuda", dtype=F64)
        U = torch.zeros((nx, m, m), device="cuda", dtype=F64)
        L = torch.zeros((nx, m, m), device="cuda", dtype=F64)
        for o in (0, 1):
            Ke = eps ** 2 * self.area * self.G[o] @ self.G[o].T + Me
            col, row = self.vert[o] % (nx + 1), self.vert[o] // (nx + 1)
            for k in range(3):
                for l in range(3):
                    c, d = col[:, k], col[:, l]
                    r, s = row[:, k], row[:, l]
                    v = torch.full((r.numel(),), Ke[k, l], device="cuda", dtype=F64)
                    which = int(_TRI[o][l][0] // 2 - _TRI[o][k][0] // 2)
                    target = (D, U, L)[which]
                    base = c if which >= 0 else d
                    target.view(-1).index_add_(0, (base * m + r) * m + s, v)
        self.A = _BlockTridiagonal(L, D, U)

    def mass(self, f):
        b = torch.zeros(self.nv, device="cuda", dtype=F64)
        for o in (0, 1):
            b.index_add_(0, self.vert[o].reshape(-1), (f[self.vert[o]] @ self.Me).reshape(-1))
        return b

    def solve(self, b):
        x = self.A.solve(b.reshape(self.ny + 1, self.nx + 1).T.contiguous())
        return x.T.reshape(-1).contiguous()

    def filter(self, f):
        return self.solve(self.mass(f))

    def weights(self):
        w = torch.zeros(self.nv, device="cuda", dtype=F64)
        for o in (0, 1):
            w.index_add_(0, self.vert[o].reshape(-1), torch.full((self.vert[o].numel(),), self.area / 3.0,
                                                                 device="cuda", dtype=F64))
        return w


class _Elastic(_Lattice):
    """The elasticity problem at penalisation 3: every integrand is a polynomial, so any exact
    rule gives the same operators."""

    def __init__(self, design, nx, ny):
        d = _elastic_dict(design)["Elasticity"]
        dom, self.par = d["domain_parameters"], d["problem_parameters"]
        super().__init__(dom["width"], dom["height"], nx, ny)
        self.volume = dom["volume_fraction"] * self.W * self.H
        self.step = dom["fem_step_size"]
        E, nu = self.par["young_modulus"], self.par["poisson_ratio"]
        self.mu = E / (2 * (1 + nu))
        self.lam = self.mu * nu / (0.5 - nu)
        self.cg1 = _Cg1(self.W, self.H, nx, ny, self.par["filter_radius"])
        pts, self.wq = _triangle_rule(4)
        self.lamq = pts
        self.tab = []
        for o in (0, 1):
            N, dN = _p2_basis(pts, self.G[o])
            K = np.zeros((len(pts), 12, 12))
            for c in range(2):
                for e in range(2):
                    k = self.lam * np.einsum("qm,qn->qmn", dN[:, :, c], dN[:, :, e])
                    k += self.mu * np.einsum("qn,qm->qmn", dN[:, :, c], dN[:, :, e])
                    if c == e:
                        k += self.mu * np.einsum("qmk,qnk->qmn", dN, dN)
                    K[:, c::2, e::2] = k
            self.tab.append((N, dN, _dev(K * (self.wq * self.area)[:, None, None])))
        self.load = self._load()

    def _coordinates(self):
        def line(L, n):
            v = np.array([k * (L / n) for k in range(n + 1)])
            out = np.empty(2 * n + 1)
            out[0::2], out[1::2] = v, 0.5 * v[:-1] + 0.5 * v[1:]
            return out
        return line(self.W, self.nx), line(self.H, self.ny)

    def _load(self):
        x, y = self._coordinates()
        b = np.zeros((2 * self.ny + 1, 2 * self.nx + 1, 2))
        for t in self.par["tractions"] or []:  # on the right side: the indicator's P2 interpolant
            on = (y >= t["center"] - t["length"] / 2 - 3e-16) & (y <= t["center"] + t["length"] / 2 + 3e-16)
            M = self.hy / 30.0 * np.array([[4.0, 2.0, -1.0], [2.0, 16.0, 2.0], [-1.0, 2.0, 4.0]])
            for j in range(self.ny):
                b[2 * j:2 * j + 3, -1] += np.outer(M @ on[2 * j:2 * j + 3], t["value"])
        b = b.reshape(-1, 2)
        if self.par["body_force"]:
            r = self.par["body_force"]["region"]
            inside = np.sqrt((x[None, :] - r["center"][0]) ** 2 + (y[:, None] - r["center"][1]) ** 2) < r["radius"]
            f = _dev(inside.reshape(-1).astype(float))
            acc = torch.zeros(self.n2, device="cuda", dtype=F64)
            for o in (0, 1):
                N = self.tab[o][0]
                M = _dev(self.area * np.einsum("q,qm,qn->mn", self.wq, N, N))
                acc.index_add_(0, self.node[o].reshape(-1), (f[self.node[o]] @ M).reshape(-1))
            b = b + np.outer(acc.cpu().numpy(), self.par["body_force"]["value"])
        return _dev(b.reshape(-1))

    def _blocks(self, xi):
        """Block-tridiagonal state matrix: block i holds the lattice columns 2i and 2i + 1."""
        nx, m = self.nx, 4 * (2 * self.ny + 1)
        D = torch.zeros((nx + 1, m, m), device="cuda", dtype=F64)
        U = torch.zeros((nx, m, m), device="cuda", dtype=F64)
        for o in (0, 1):
            xq = xi[self.vert[o]] @ _dev(self.lamq.T)
            r = PMIN + xq ** 3 * (1 - PMIN)
            Ke = torch.einsum("tq,qij->tij", r, self.tab[o][2])
            a, b = self.node[o] % (2 * nx + 1), self.node[o] // (2 * nx + 1)
            blk = a // 2
            pos = ((a % 2) * (2 * self.ny + 1) + b) * 2
            clamped = a == 0  # the left side
            for k in range(6):
                for l in range(6):
                    dk = _TRI[o][k][0] // 2, _TRI[o][l][0] // 2
                    if dk[0] > dk[1]:
                        continue  # the lower blocks are the transposed upper ones
                    free = (~(clamped[:, k] | clamped[:, l])).to(F64)
                    target = D if dk[0] == dk[1] else U
                    for c in range(2):
                        for e in range(2):
                            target.view(-1).index_add_(0, (blk[:, k] * m + pos[:, k] + c) * m + pos[:, l] + e,
                                                       Ke[:, 2 * k + c, 2 * l + e] * free)
        unit = torch.arange(2 * (2 * self.ny + 1), device="cuda")
        D[0, unit, unit] = 1.0  # clamped column
        D[nx, unit + unit.numel(), unit + unit.numel()] = 1.0  # the column past the right side
        return _BlockTridiagonal(U.transpose(1, 2), D, U)

    def state(self, rho):
        xi = self.cg1.filter(rho)
        nx, rows = self.nx, 2 * self.ny + 1
        b = self.load.reshape(rows, 2 * nx + 1, 2).clone()
        b[:, 0] = 0.0
        padded = torch.zeros((rows, 2 * nx + 2, 2), device="cuda", dtype=F64)
        padded[:, :-1] = b
        x = self._blocks(xi).solve(padded.permute(1, 0, 2).reshape(nx + 1, -1).contiguous())
        u = x.reshape(2 * nx + 2, rows, 2)[:-1].permute(1, 0, 2).reshape(-1).contiguous()
        return float(self.load @ u), u, xi

    def gradient(self, u, xi):
        b = torch.zeros(self.nv, device="cuda", dtype=F64)
        un = u.reshape(-1, 2)
        for o in (0, 1):
            g = torch.einsum("qkd,tkc->tqcd", _dev(self.tab[o][1]), un[self.node[o]])
            div = g[..., 0, 0] + g[..., 1, 1]
            e = 0.5 * (g + g.transpose(-1, -2))
            xq = xi[self.vert[o]] @ _dev(self.lamq.T)
            f = -3.0 * xq ** 2 * (1 - PMIN) * (self.lam * div ** 2 + 2 * self.mu * (e * e).sum((-1, -2)))
            b.index_add_(0, self.vert[o].reshape(-1), ((f * _dev(self.wq * self.area)) @ _dev(self.lamq)).reshape(-1))
        return self.cg1.solve(b)


def _loop_exact(ref, rho, iterations):
    """The mirror-descent loop (step size k + 1 times the base, Newton volume projection)."""
    w = ref.cg1.weights()
    psi = torch.log(rho / (1 - rho))
    objective, u, xi = ref.state(rho)
    objectives = [objective]
    for k in range(iterations):
        half = psi - ref.step * (k + 1) * ref.gradient(u, xi)
        c = 0.0
        for _ in range(50):
            e = torch.sigmoid(half + c)
            new = c - float(w @ e - ref.volume) / float(w @ (e * (1 - e)))
            done, c = abs(new - c) < 1e-12, new
            if done:
                break
        previous, psi = rho, half + c
        rho = torch.sigmoid(psi)
        objective, u, xi = ref.state(rho)
        objectives.append(objective)
        delta = float((w @ (rho - previous) ** 2).sqrt())
        best = int(np.argmin(objectives))
        if objectives[-1] > 2 * objectives[best] or delta < min(25 * (k + 1) * 1e-5, 1e-2):
            break
    return {"objectives": objectives, "rho": rho}


def _dem_exact(case, seed):
    nx, ny = case["nx"], case["ny"]
    u, rho = _dem_inputs(seed, nx, ny)
    u, rho = u.double().requires_grad_(True), rho.double().requires_grad_(True)
    hx, hy = 2.0 / nx, 1.0 / ny
    par = _dem_dict()["Elasticity"]["problem_parameters"]
    mu = par["young_modulus"] / (2 * (1 + par["poisson_ratio"]))
    lam = mu * par["poisson_ratio"] / (0.5 - par["poisson_ratio"])
    mask = (torch.arange(nx + 1, device="cuda", dtype=F64) / nx)[:, None, None]

    def strain_energy(v):  # integral of sigma : eps over each cell, (ny, nx)
        corner = {(a, b): v[a:nx + a, b:ny + b] for a in (0, 1) for b in (0, 1)}
        total = 0
        for s in (0.5 - 0.5 / math.sqrt(3), 0.5 + 0.5 / math.sqrt(3)):
            for t in (0.5 - 0.5 / math.sqrt(3), 0.5 + 0.5 / math.sqrt(3)):
                gx = sum((1 if a else -1) * (t if b else 1 - t) * c for (a, b), c in corner.items()) / hx
                gy = sum((s if a else 1 - s) * (1 if b else -1) * c for (a, b), c in corner.items()) / hy
                div = gx[..., 0] + gy[..., 1]
                shear = 0.5 * (gx[..., 1] + gy[..., 0])
                total = total + lam * div ** 2 + 2 * mu * (gx[..., 0] ** 2 + gy[..., 1] ** 2 + 2 * shear ** 2)
        return (total * (0.25 * hx * hy)).T

    v = u.reshape(nx + 1, ny + 1, 2)
    side = torch.full((ny + 1,), hy, device="cuda", dtype=F64)
    side[0] = side[-1] = hy / 2
    t = par["tractions"][0]["value"]
    r = PMIN + rho ** 3 * (1 - PMIN)
    vm = v * mask
    external = (side[:, None] * vm[-1] * torch.tensor(t, device="cuda", dtype=F64)).sum()
    psi = 0.5 * (r * strain_energy(vm)).sum() - external
    du, drho = torch.autograd.grad(psi, (u, rho))
    se = strain_energy(v)
    objective = (r * se).sum()
    gradient = -3.0 * rho ** 2 * (1 - PMIN) * se
    return {"psi": psi.detach(), "du": du, "drho": drho, "objective": objective.detach(),
            "gradient": gradient.detach()}


def _dem_filter_exact(case, seed):
    nx, ny, radius = case["nx"], case["ny"], case["radius"]
    rho, g = _dem_filter_inputs(seed, nx, ny)
    sx, sy = 2.0 / (nx - 1), 1.0 / (ny - 1)
    rx, ry = min(nx - 1, int(radius / sx) + 1), min(ny - 1, int(radius / sy) + 1)

    def convolve(f):
        """sum over the offsets within the radius of (radius - distance) f(shifted)."""
        f = f.reshape(ny, nx)
        dx = torch.arange(-rx, rx + 1, device="cuda", dtype=F64) * sx
        dy = torch.arange(-ry, ry + 1, device="cuda", dtype=F64) * sy
        k = (radius - torch.sqrt(dx[None, :] ** 2 + dy[:, None] ** 2)).clamp(min=0.0)
        n0, n1 = ny + 2 * ry, nx + 2 * rx
        full = torch.fft.irfft2(torch.fft.rfft2(f, s=(n0, n1)) * torch.fft.rfft2(k, s=(n0, n1)), s=(n0, n1))
        return full[ry:ry + ny, rx:rx + nx].reshape(-1)

    total = convolve(torch.ones_like(rho))
    return {"filtered": convolve(rho) / total, "back": convolve(g / total)}


def _fluid_exact(case, seed):
    """Dense solve of the reduced Taylor-Hood system (boundary velocities eliminated, the
    continuity right-hand side projected to zero sum, zero-sum pressure)."""
    n = case["n"]
    M = _Cg1(1.0, 1.0, n, n, 0.0)
    rho = _fluid_design(seed, n, case["contrast"])
    q, lo, hi = 0.1, 2.5 / 100 ** 2, 2.5 / 0.01 ** 2
    alpha = lambda r: hi + (lo - hi) * r * (1 + q) / (r + q)  # noqa: E731
    # degree-6 rule of Strang and Fix (12 points): the quadrature of the state and objective
    o3 = lambda a: [(1 - 2 * a, a, a), (a, 1 - 2 * a, a), (a, a, 1 - 2 * a)]  # noqa: E731
    a, b = 0.053145049844816, 0.310352451033785
    c = 1 - a - b
    p6 = np.array(o3(0.063089014491502) + o3(0.249286745170910)
                  + [(a, b, c), (a, c, b), (b, a, c), (b, c, a), (c, a, b), (c, b, a)])
    w6 = np.array([0.050844906370207] * 3 + [0.116786275726379] * 3 + [0.082851075618374] * 6)
    # degree-7 collapsed Gauss-Jacobi rule (4 x 4 points): the quadrature of the gradient
    tx, wx = np.polynomial.legendre.leggauss(4)
    k = np.arange(4)
    jd = -1.0 / ((2 * k + 1) * (2 * k + 3))
    k = np.arange(1, 4)
    jo = np.sqrt(k * (k + 1.0)) / (2 * k + 1)
    ty, vec = np.linalg.eigh(np.diag(jd) + np.diag(jo, 1) + np.diag(jo, -1))
    wy = 2 * vec[0] ** 2
    p7 = np.array([(1 - 0.25 * (1 + x) * (1 - e) - 0.5 * (1 + e), 0.25 * (1 + x) * (1 - e), 0.5 * (1 + e))
                   for x in tx for e in ty])
    w7 = np.array([0.25 * u * v for u in wx for v in wy])
    nx2, n2, nv, area = 2 * n + 1, M.n2, M.nv, M.area
    S = torch.zeros((2 * n2 + nv + 1, 2 * n2 + nv + 1), device="cuda", dtype=F64)
    flat, width = S.view(-1), 2 * n2 + nv + 1
    for o in (0, 1):
        N, dN = _p2_basis(p6, M.G[o])
        lap = _dev(area * np.einsum("q,qik,qjk->ij", w6, dN, dN))
        nn = _dev(area * np.einsum("q,qi,qj->qij", w6, N, N))
        grad = area * np.einsum("q,qi,kc->ick", w6, N, M.G[o])
        div = area * np.einsum("q,qk,qjc->kjc", w6, p6, dN)
        A = torch.einsum("tq,qij->tij", alpha(rho[M.vert[o]] @ _dev(p6.T)), nn) + lap
        nd, vt = M.node[o], M.vert[o]
        ones = torch.ones(nd.shape[0], device="cuda", dtype=F64)
        for i in range(6):
            for e in range(2):
                for j in range(6):
                    flat.index_add_(0, (2 * nd[:, i] + e) * width + 2 * nd[:, j] + e, A[:, i, j])
                for v in range(3):
                    flat.index_add_(0, (2 * nd[:, i] + e) * width + 2 * n2 + vt[:, v], float(grad[i, e, v]) * ones)
                    flat.index_add_(0, (2 * n2 + vt[:, v]) * width + 2 * nd[:, i] + e, float(div[v, i, e]) * ones)
    idx = np.arange(n2)
    xi, yi = idx % nx2, idx // nx2
    y = yi / (2.0 * n)
    ub = np.zeros((n2, 2))
    for f in _fluid_dict()["Fluid"]["problem_parameters"]["flows"]:
        s = 2 * (y - f["center"]) / f["length"]
        on = (xi == (0 if f["side"] == "Left" else nx2 - 1)) & (np.abs(s) < 1)
        ub[on, 0] += (1 if f["side"] == "Left" else -1) * f["rate"] * (1 - s[on] ** 2)
    ub[(yi == 0) | (yi == nx2 - 1)] = 0.0
    boundary = (xi == 0) | (xi == nx2 - 1) | (yi == 0) | (yi == nx2 - 1)
    ub = _dev(ub.reshape(-1))
    r = -(S[:-1, :2 * n2] @ ub)
    r[2 * n2:] -= r[2 * n2:].mean()
    S[-1, 2 * n2:-1] = S[2 * n2:-1, -1] = 1.0
    free = torch.cat([torch.nonzero(_dev(np.repeat(~boundary, 2))).reshape(-1),
                      torch.arange(2 * n2, width, device="cuda")])
    K = S[free][:, free]
    del S, flat
    f = torch.cat([r, torch.zeros(1, device="cuda", dtype=F64)])[free]
    lu = torch.linalg.lu_factor(K)
    x = torch.linalg.lu_solve(*lu, f[:, None])[:, 0]
    x = x + torch.linalg.lu_solve(*lu, (f - K @ x)[:, None])[:, 0]
    nf = free.numel() - nv - 1
    u = ub.clone()
    u[free[:nf]] = x[:nf]
    un = u.reshape(-1, 2)
    objective, rhs = 0.0, torch.zeros(nv, device="cuda", dtype=F64)
    for o in (0, 1):
        N, dN = _p2_basis(p6, M.G[o])
        ue, rv = un[M.node[o]], rho[M.vert[o]]
        uq = torch.einsum("qk,tkc->tqc", _dev(N), ue)
        gq = torch.einsum("qkd,tkc->tqcd", _dev(dN), ue)
        e = alpha(rv @ _dev(p6.T)) * (uq ** 2).sum(-1) + (gq ** 2).sum((-1, -2))
        objective += float((e @ _dev(w6 * area)).sum())
        N7, _ = _p2_basis(p7, M.G[o])
        uq = torch.einsum("qk,tkc->tqc", _dev(N7), ue)
        da = (lo - hi) * q * (1 + q) / (rv @ _dev(p7.T) + q) ** 2
        rhs.index_add_(0, M.vert[o].reshape(-1), ((0.5 * da * (uq ** 2).sum(-1) * _dev(w7 * area)) @ _dev(p7)).reshape(-1))
    return {"objective": 0.5 * objective, "u": u, "p": x[nf:nf + nv], "gradient": M.solve(rhs)}
