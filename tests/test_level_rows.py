"""Rows that a sweep builds from the triangles' coefficients (csrc/topo_p1level.cuh) against the
stored ones (csrc/topo_p1.cuh), and on the GPU a solve with every level's rows built against one
with all of them stored.

A row's values are sums of at most six products of numbers rounded once, and the row sum one of
six couplings: 40 roundings of the row's largest value bound the difference.
"""
import ctypes

import numpy as np
import pytest

from oracle.fem import lame
from tests import emu


def _dir(nx, ny, sides):
    d = emu.no_dir(nx + 1, ny + 1)
    d[0], d[1] = "Left" in sides, "Bottom" in sides
    d[2] -= "Right" in sides
    d[3] -= "Top" in sides
    return d


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("NC", [1, 2])
@pytest.mark.parametrize("sides", [[], ["Left"], ["Left", "Right", "Top", "Bottom"]])
@pytest.mark.parametrize("nx,ny", [(1, 1), (2, 3), (7, 1), (9, 6)])
def test_built_rows_match_the_stored_ones(nx, ny, sides, NC, prec):
    rng = np.random.default_rng(10 * nx + ny)
    lam, mu = lame(1.0, 0.3)
    SW = 28 if NC == 2 else 8
    kK, kM = 10.0 ** rng.uniform(-3.0, 0.0, 2 * nx * ny), 10.0 ** rng.uniform(-1.0, 1.0, 2 * nx * ny)
    stored, built = np.full(((nx + 1) * (ny + 1), SW), np.nan), np.full(((nx + 1) * (ny + 1), SW), np.nan)
    I, F, P = ctypes.c_int, ctypes.c_double, emu.P_D
    E = emu.lib()
    E.emu_level_rows.argtypes = [I, I, I, I, F, F, F, F, emu.P_I, P, P, P, P]
    assert E.emu_level_rows(prec, NC, nx, ny, 0.05, 0.04, lam, mu, emu.ip(_dir(nx, ny, sides)), emu.dp(kK),
                            emu.dp(kM), emu.dp(stored), emu.dp(built)) == SW
    eps = 2.0 ** -24 if prec else 2.0 ** -53
    assert np.all(np.abs(built - stored) <= 40 * eps * np.abs(stored).max(axis=1, keepdims=True))


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny", [(80, 40), (101, 33), (320, 90)])
def test_solve_with_built_rows(nx, ny, monkeypatch):
    """TOPO_STENCIL_NODES=600 leaves only the tail's levels their stored rows.  Both solves reach a
    relative residual of 1e-9 with an FP64 operator of condition below 1e7 per unit of the load's
    smooth part; the compliance, quadratic in the error, agrees to 1e-6."""
    from test_gpu_parity import _design, _gpu_problem
    got = []
    for nodes in (None, "600"):
        if nodes:
            monkeypatch.setenv("TOPO_STENCIL_NODES", nodes)
        prob, V = _gpu_problem(_design(), nx, ny, rtol=1e-9)
        prob.set_penalization(3.0)
        got.append((prob.calculate_objective(np.random.default_rng(nx).uniform(0.1, 1.0, V.dim())),
                    prob.stats["state_iterations"]))
    assert abs(got[0][0] - got[1][0]) <= 1e-6 * abs(got[0][0])
    assert abs(got[0][1] - got[1][1]) <= 3  # the same V-cycle up to rounding
