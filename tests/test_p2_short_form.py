"""The P2 kernel's short form, one cell row per warp (csrc/topo_p2.cuh, kRowsSegment), against the
march over segments on the CPU: the two differ in the order of a node row's sum of at most six
triangles, so by a few roundings: 1e-13 of the largest value in FP64, 2e-6 in FP32."""
import numpy as np
import pytest

from oracle.fem import lame
from tests import emu

# cells: within one warp and block, whole blocks, one row or column past them, interior (lean) warps
SIZES = [(1, 1), (3, 2), (30, 4), (31, 5), (32, 8), (34, 9), (70, 17), (65, 24)]


@pytest.fixture(autouse=True)
def _restore():
    yield
    emu.set_segment(0)


def _both(f):
    out = []
    for seg in (2, -1):
        emu.set_segment(seg)
        out.append(f())
    return out


@pytest.mark.parametrize("prec,tol", [(0, 1e-13), (1, 2e-6)])
@pytest.mark.parametrize("sides", [[], ["Left"], ["Bottom", "Right", "Top"]])
@pytest.mark.parametrize("nx,ny", SIZES)
def test_operator(nx, ny, sides, prec, tol):
    rng = np.random.default_rng(nx + 100 * ny)
    lam, mu = lame(1.0, 0.3)
    xi, u = rng.uniform(0.05, 1.0, (nx + 1) * (ny + 1)), rng.standard_normal(2 * (2 * nx + 1) * (2 * ny + 1))
    dirv = emu.make_dir(nx, ny, 0.05, 0.04, sides)
    march, short = _both(lambda: emu.p2_apply(nx, ny, 0.05, 0.04, lam, mu, 3.0, dirv, xi, u, prec=prec))
    assert np.max(np.abs(short - march)) <= tol * np.max(np.abs(march))


@pytest.mark.parametrize("mode,out", [("pre", ["x"]), ("res", ["r"]), ("first", ["d", "x2"]), ("post2", ["x"])])
@pytest.mark.parametrize("nx,ny", SIZES)
def test_smoothing(nx, ny, mode, out):
    rng = np.random.default_rng(nx + 100 * ny)
    lam, mu = lame(1.0, 0.3)
    xi = rng.uniform(0.05, 1.0, (nx + 1) * (ny + 1))
    dirv = emu.make_dir(nx, ny, 0.05, 0.04, ["Left"])
    n = 2 * (2 * nx + 1) * (2 * ny + 1)
    vec = {k: rng.standard_normal(n) for k in ("b", "dinv", "x", "x2", "r", "d")}
    xc = rng.standard_normal(2 * (nx + 1) * (ny + 1)) if mode == "first" else None

    def run():
        bufs = {k: v.copy() for k, v in vec.items()}
        emu.smooth(mode, True, 2, nx, ny, 0.05, 0.04, lam, mu, 3.0, dirv, xi, None, bufs, [0.7, 0.3, 0.9],
                   NXc=nx + 1, NYc=ny + 1, xc=xc)
        return bufs
    march, short = _both(run)
    for k in out:
        assert np.max(np.abs(short[k] - march[k])) <= 1e-13 * np.max(np.abs(march[k]))
