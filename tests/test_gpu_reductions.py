"""Grid reductions (csrc/topo_vec.cuh): one block, the edges of the four-values-a-thread rule, and
the largest grids, against numpy.  All terms are positive, so a sum in any tree order of depth
below 64 is within 64 eps = 1.5e-14 of the exact one; numpy's pairwise sum likewise."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(1, 1), (30, 32), (31, 31), (24, 40), (1023, 1), (63, 65), (700, 480), (1500, 1100)])
def test_integrate_is_the_weighted_sum(nx, ny):
    import torch
    import topomax_gb300 as tg
    from topomax_gb300.fem import _ptr, _stream
    from oracle.fem import Lattice
    V = tg.FunctionSpace(tg.RectangleMesh(2.0, 1.0, nx, ny), "CG", 1)
    F = tg.HelmholtzFilter(0.05, V)
    f = np.random.default_rng(nx + ny).uniform(0.5, 1.5, V.dim())
    L = Lattice(2.0, 1.0, nx, ny)
    w = np.zeros(V.dim())
    for o in (0, 1):
        np.add.at(w, L.triangle_vertices(o).ravel(), 0.5 * L.hx * L.hy / 3.0)
    t, out = torch.tensor(f, device="cuda"), torch.zeros(1, dtype=torch.float64, device="cuda")
    for _ in range(2):  # the counter is back at zero after a reduction
        F._ctx.check(F._ctx._lib.topo_integrate(F._ctx.ptr, _ptr(t), _ptr(out), _stream()))
        assert abs(float(out) - w @ f) <= 3e-14 * (w @ f)
