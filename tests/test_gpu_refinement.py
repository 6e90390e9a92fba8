"""The mixed-precision refinement as a device-driven cycle (graphs) and from the host."""
import numpy as np
import pytest

from oracle.fem import FEMOracle, Lattice
from test_gpu_parity import _design, _gpu_problem

pytestmark = pytest.mark.gpu

RTOL = 1e-8


@pytest.mark.parametrize("graphs", ["1", "0"])
@pytest.mark.parametrize("nx,ny", [(2, 1), (7, 5), (40, 20), (101, 33)])
def test_residuals_with_the_oracle_operators(nx, ny, graphs, monkeypatch):
    """Both solves stop at half of rtol.  The operators' roundings differ by some 4e-15 |K| |u|, and
    |K| |u| is below 4e5 |b| at these sizes and densities: less than a fifth of rtol."""
    monkeypatch.setenv("TOPO_GRAPHS", graphs)
    d = _design()
    prob, _ = _gpu_problem(d, nx, ny, rtol=RTOL)
    o = FEMOracle(Lattice(2.0, 1.0, nx, ny), d)
    rng = np.random.default_rng(nx)
    for p, warm in ((3.0, False), (3.0, True), (1.5, False)):  # recorded, replayed, another operator
        prob.warm_start = warm
        prob.set_penalization(p)
        o.set_penalization(p)
        rho = rng.uniform(0.2, 1.0, o.L.n_vertices)
        prob.calculate_objective(rho)
        b = o.M1 @ rho
        xi = prob.filtered_rho.vector()[:]
        assert np.linalg.norm(b - o.A_filter @ xi) <= RTOL * np.linalg.norm(b)
        u = prob.u.vector()[:]
        r = (o.load - o.stiffness(xi) @ u)[o.free]
        assert np.linalg.norm(r) <= RTOL * np.linalg.norm(o.load[o.free])
        assert np.all(np.delete(u, o.free) == 0.0)


def test_large_vectors_match_the_host_driven_solve(monkeypatch):
    """More than eight entries per thread of a full grid (2.6 M unknowns).  A residual r moves the
    compliance b.u by u.r: relative to it at most rtol |u| |b| / (u.b), about
    rtol sqrt(nodes / loaded nodes) = 60 rtol for a load where u is largest."""
    got = []
    for graphs in ("1", "0"):
        monkeypatch.setenv("TOPO_GRAPHS", graphs)
        prob, V = _gpu_problem(_design(), 800, 400, rtol=RTOL)
        prob.set_penalization(3.0)
        got.append(prob.calculate_objective(np.random.default_rng(0).uniform(0.2, 1.0, V.dim())))
    assert abs(got[0] - got[1]) <= 2 * 60 * RTOL * abs(got[1])


def test_zero_load_gives_a_zero_state():
    """A right-hand side of zero leaves no residual to reduce: the cycle does not run."""
    import torch
    import topomax_gb300 as tg
    V = tg.FunctionSpace(tg.RectangleMesh(2.0, 1.0, 20, 10), "CG", 1)
    F = tg.HelmholtzFilter(0.05, V)
    assert torch.count_nonzero(F.apply(np.zeros(V.dim())).tensor) == 0
