"""The fluid operator by output node (csrc/topo_fluid.cuh) against the oracle's assembled matrix,
and the device-driven solve on sizes around its kernels' block and restart edges."""
import ctypes

import numpy as np
import pytest


def _oracle(nx, ny, q=0.1):
    import json
    import os
    from oracle.fem import Lattice
    from oracle.fluid import FluidDesign, FluidOracle
    path = os.path.join(os.path.dirname(__file__), "golden", "designs", "diffuser.json")
    d = FluidDesign.from_dict(json.load(open(path)))
    o = FluidOracle(Lattice(d.width, d.height, nx, ny), d, pressure="mean")
    o.set_penalization(q)
    return o


@pytest.mark.parametrize("nx,ny", [(1, 1), (1, 4), (5, 1), (7, 6)])
def test_node_rows_match_oracle(nx, ny):
    """Every row, with a constant taken off the pressure; sums of some 40 products: 1e-13."""
    from tests import emu
    o = _oracle(nx, ny)
    rng = np.random.default_rng(nx + 10 * ny)
    rho, x = rng.uniform(0.0, 1.0, o.nv), rng.standard_normal(o.n)
    y, pm, D = np.full(o.n, np.nan), 0.7, ctypes.c_double
    E = emu.lib()
    E.emu_fluid_apply_nodes.argtypes = [ctypes.c_int, ctypes.c_int, D, D, D, D] + [emu.P_D] * 3
    E.emu_fluid_apply_nodes(nx, ny, 1.0, 1.0, 0.1, pm, emu.dp(rho), emu.dp(x), emu.dp(y))
    s = np.ones(o.n)
    s[o.nuv:] = -1.0
    xs = x.copy()
    xs[o.nuv:] -= pm
    ref = s * (o.assemble(rho) @ xs)
    assert np.max(np.abs(y - ref)) <= 1e-13 * np.max(np.abs(ref))


@pytest.mark.gpu
@pytest.mark.parametrize("graphs", ["1", "0"])
@pytest.mark.parametrize("n,kind", [(2, "uniform"), (9, "sharp"), (24, "sharp"), (33, "random")])
def test_solve_matches_oracle(n, kind, graphs, monkeypatch):
    """Velocity and pressure at a residual of 1e-12 against the oracle's sparse LU: the state
    amplifies it by some 1e3 on these meshes.  The 0/1 design takes several restart cycles."""
    import os
    import torch
    import topomax_gb300 as tg
    monkeypatch.setenv("TOPO_GRAPHS", graphs)
    o = _oracle(n, n)
    rng = np.random.default_rng(n)
    L = o.L
    X, Y = L.vertex_coords()
    rho = {"uniform": np.full(o.nv, 0.5), "random": rng.uniform(0.0, 1.0, o.nv),
           "sharp": (np.abs(Y - 0.5) < 0.5 - X / 3.0 + 1e-9).astype(float)}[kind]
    path = os.path.join(os.path.dirname(__file__), "golden", "designs", "diffuser.json")
    domain, params = tg.parse_design(path)
    prob = tg.FluidProblem(tg.RectangleMesh(1.0, 1.0, n, n), params, domain, rtol=1e-12)
    prob.set_penalization(0.1)
    ur, pr = o.state_solve(rho)
    for _ in range(2):  # the second solve replays the recorded cycle
        u, p = prob.forward(torch.as_tensor(rho).cuda())
        u, p = u.tensor.cpu().numpy(), p.tensor.cpu().numpy()
        assert np.linalg.norm(u - ur) <= 1e-9 * np.linalg.norm(ur)
        assert np.linalg.norm(p - (pr - pr.mean())) <= 1e-8 * np.linalg.norm(pr - pr.mean())
        assert abs(p.sum()) <= 1e-9 * np.abs(p).sum()
