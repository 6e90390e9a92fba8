"""The V-cycle's fused level sweeps (csrc/topo_p1level.cuh).

On the CPU the phases run over all blocks with NaN-filled shared memory and are compared with
the same steps composed from plain operator applies and the transfers; on the GPU a V-cycle
with the one-block tail is compared with one launch per level.  FP64 steps chain up to
five applications of a 7-point operator of O(1) values: 1e-12; FP32 likewise at 2^-24: 1e-5.
"""
import ctypes

import numpy as np
import pytest

from oracle.fem import lame
from tests import emu

# level sizes in cells: smaller than a block, its multiples and one past, odd (a padded coarse level), flat
SIZES = [(8, 4), (20, 8), (21, 9), (40, 16), (39, 17), (64, 1), (1, 32), (55, 23)]


def _level(NC, nx, ny, sides, rng):
    lam, mu = lame(1.0, 0.3)
    hx = hy = 0.05
    dirv = emu.no_dir(nx + 1, ny + 1)
    dirv[0], dirv[1] = "Left" in sides, "Bottom" in sides
    dirv[2] -= "Right" in sides
    dirv[3] -= "Top" in sides
    f, c = emu.build_levels(False, nx, ny, hx, hy, dirv, NC)[:2]
    kK = 10.0 ** rng.uniform(-3.0, 0.0, 2 * nx * ny)
    kM = 10.0 ** rng.uniform(-1.0, 1.0, 2 * nx * ny) if NC == 1 else None
    return lam, mu, hx, hy, dirv, f, c, kK, kM


def _free(dirv, NX, NY, NC):
    a, b = np.meshgrid(np.arange(NX), np.arange(NY))
    cl = ((dirv[0] != 0) & (a == 0)) | (a >= dirv[2]) | ((dirv[1] != 0) & (b == 0)) | (b >= dirv[3])
    return np.repeat(~cl.ravel(), NC)


@pytest.mark.parametrize("prec,tol", [(0, 1e-12), (1, 1e-5)])
@pytest.mark.parametrize("NC,sides", [(2, ["Left"]), (2, ["Left", "Right"]), (1, []),
                                      (1, ["Left", "Right", "Top", "Bottom"])])
@pytest.mark.parametrize("D", [2, 3, 4])
@pytest.mark.parametrize("nx,ny", SIZES)
def test_sweeps_match_composed_steps(nx, ny, D, NC, sides, prec, tol):
    rng = np.random.default_rng(100 * nx + ny)
    lam, mu, hx, hy, dirv, f, c, kK, kM = _level(NC, nx, ny, sides, rng)
    A = lambda u: emu.p1_apply(NC, nx, ny, hx, hy, lam, mu, dirv, kK, kM, u)  # noqa: E731
    n, nc = NC * f["NX"] * f["NY"], NC * c["NX"] * c["NY"]
    free, freec = _free(f["dir"], f["NX"], f["NY"], NC), _free(c["dir"], c["NX"], c["NY"], NC)
    b, x = rng.standard_normal(n) * free, rng.standard_normal(n) * free
    xc = rng.standard_normal(nc) * freec
    dinv = np.where(free, rng.uniform(0.5, 2.0, n), 1.0)
    cheb = np.array([0.7, 0.3, 0.9, 0.2, 0.6, 0.25, 0.5])[:2 * D - 1]
    xpre, bc, xpost = np.zeros(n), np.zeros(nc), np.zeros(n)
    P, I, F = emu.P_D, ctypes.c_int, ctypes.c_double
    E = emu.lib()
    E.emu_level_sweeps.argtypes = [I, I, I, I, I, F, F, F, F, emu.P_I, P, P, P, I, I, emu.P_I, I, I] + [P] * 7
    assert E.emu_level_sweeps(prec, NC, D, nx, ny, hx, hy, lam, mu, emu.ip(dirv), emu.dp(kK), emu.dp(kM), emu.dp(cheb),
                              c["NX"], c["NY"], emu.ip(c["dir"]), 10, 4, emu.dp(b), emu.dp(dinv), emu.dp(x),
                              emu.dp(xc), emu.dp(xpre), emu.dp(bc), emu.dp(xpost)) == 0

    def close(got, want):
        assert np.max(np.abs(got - want)) <= tol * max(np.max(np.abs(want)), 1e-30)

    def chebyshev(r, x):
        d = cheb[0] * dinv * r
        x = x + d
        for k in range(1, D):
            r = r - A(d)
            d = cheb[2 * k - 1] * d + cheb[2 * k] * dinv * r
            x = x + d
        return x

    ref = chebyshev(b, np.zeros(n))
    close(xpre, ref)
    close(bc, emu.restrict(NC, f["NX"], f["NY"], f["dir"], c["NX"], c["NY"], c["dir"], b - A(ref)))
    u = x + emu.prolong(NC, f["NX"], f["NY"], f["dir"], c["NX"], c["NY"], c["dir"], xc)
    close(xpost, chebyshev(b - A(u), u))


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,points", [(7, 3, False), (33, 31, False), (90, 2, False), (61, 45, True), (130, 17, False)])
def test_tail_matches_levels(nx, ny, points, monkeypatch):
    """Same steps in the same order and the same fused operations: equal bits."""
    import torch
    import topomax_gb300 as tg
    from topomax_gb300.designs import parse_design_dict
    out = []
    for tail in ("1", "0"):
        monkeypatch.setenv("TOPO_TAIL", tail)
        dom, par = parse_design_dict({"Elasticity": {
            "domain_parameters": dict(width=2.0, height=1.0, fem_step_size=1.0, dem_step_size=1.0, penalties=[3.0],
                                      volume_fraction=0.5),
            "problem_parameters": dict(fixed_sides=[] if points else ["Left"],
                                       fixed_points=[[0.0, 0.0], [2.0, 0.0]] if points else [],
                                       body_force=dict(region=dict(center=[1.0, 0.5], radius=0.3), value=[0.0, -1.0]),
                                       tractions=None, filter_radius=0.05, young_modulus=1.0, poisson_ratio=0.3)}})
        mesh = tg.RectangleMesh(2.0, 1.0, nx, ny)
        V = tg.FunctionSpace(mesh, "CG", 1)
        prob = tg.ElasticityProblem(mesh, V, dom, par, precision="mixed", rtol=1e-9)
        prob.set_penalization(3.0)
        rho = torch.rand(V.dim(), generator=torch.Generator().manual_seed(3), dtype=torch.float64) * 0.9 + 0.1
        prob.calculate_objective(rho)
        out.append((prob.stats["state_iterations"], prob.u.tensor.cpu().numpy()))
    assert out[0][0] == out[1][0] and np.array_equal(out[0][1], out[1][1])
