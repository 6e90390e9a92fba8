"""The density filter's weight table and integer quotient (csrc/topo_dens.cuh).

Every result is a correctly rounded FP64 operation in a fixed order, so all comparisons are
for equal bits: the quotient against the host's IEEE division, the filter against the oracle's
restatement of DEM_src/filter.py:8-31.
"""
import ctypes

import numpy as np
import pytest

from oracle import dem as O

# radius below a step (own element only), at exactly a step, past the whole mesh, single rows and
# columns, odd sizes, a warp's remainder
FORMS = [(5, 4, 1.0, 1.0, 0.05), (11, 3, 1.0, 1.0, 0.1), (7, 9, 1.3, 0.7, 5.0), (1, 13, 1.0, 2.0, 0.3),
         (17, 1, 2.0, 1.0, 0.2), (1, 1, 1.0, 1.0, 0.4), (33, 31, 2.0, 1.0, 0.1732), (64, 20, 10.0, 5.0, 0.83)]


def _quotient_inputs():
    rng = np.random.default_rng(5)
    n = 400_000
    s = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(-20, 20, n))
    w = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(-70, 10, n))
    # significands at the ends of their range, quotients near one, near powers of two and near
    # rounding boundaries (w = the rounded product of s and a 53-bit value, one unit either way)
    edge = np.array([1.0, np.nextafter(1.0, 2), np.nextafter(2.0, 0), 1.5])
    es, ew = [a.ravel() for a in np.meshgrid(edge, edge)]
    q = rng.uniform(1.0, 2.0, n) + 0.5 * np.spacing(1.0)
    near = s * q
    s = np.concatenate([s, es, s, s, s, s[:100]])
    w = np.concatenate([w, ew, near, np.nextafter(near, 0), np.nextafter(near, 1e300), np.zeros(100)])
    return np.ascontiguousarray(w), np.ascontiguousarray(s)


def test_integer_quotient_is_the_rounded_division():
    from tests.native.build_emulator import load
    E = load()
    w, s = _quotient_inputs()
    out = np.empty_like(w)
    P = ctypes.POINTER(ctypes.c_double)
    E.emu_dens_quotient(ctypes.c_long(w.size), w.ctypes.data_as(P), s.ctypes.data_as(P), out.ctypes.data_as(P))
    assert np.array_equal((w / s).view(np.int64), out.view(np.int64))


def _vector(Nx, Ny):
    v = np.random.default_rng(Nx * 100 + Ny).normal(size=Nx * Ny)
    return v


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("transpose", [False, True])
def test_table_matches_oracle_on_the_cpu(form, transpose):
    from tests.native.build_emulator import load
    E = load()
    Nx, Ny, W, H, r = form
    x = _vector(Nx, Ny)
    y = np.empty_like(x)
    P = ctypes.POINTER(ctypes.c_double)
    D = ctypes.c_double
    assert E.emu_dens_filter(Nx, Ny, D(W), D(H), D(r), int(transpose), x.ctypes.data_as(P), y.ctypes.data_as(P)) == 0
    assert np.array_equal(y, O.density_filter_apply(Nx, Ny, W, H, r, x, transpose))


@pytest.mark.gpu
@pytest.mark.parametrize("form", FORMS + [(6, 5, 1.0, 1.0, 0.0)])  # radius 0: the general kernels
@pytest.mark.parametrize("transpose", [False, True])
def test_filter_matches_oracle_on_the_gpu(form, transpose):
    from topomax_gb300 import dem
    Nx, Ny, W, H, r = form
    F = dem.create_density_filter(r, dem.Mesh(Nx, Ny, W, H))
    assert F.nnz == sum(len(nb) for nb, _, _ in O.density_filter_rows(Nx, Ny, W, H, r))
    x = _vector(Nx, Ny)
    y = (F.T if transpose else F) @ x
    assert np.array_equal(y, O.density_filter_apply(Nx, Ny, W, H, r, x, transpose))


@pytest.mark.gpu
def test_non_finite_values_stay_within_the_radius():
    from topomax_gb300 import dem
    Nx, Ny, W, H, r = 33, 31, 2.0, 1.0, 0.1732
    x = _vector(Nx, Ny)
    x[16 * Nx + 5], x[3 * Nx + 30] = np.inf, np.nan
    with np.errstate(invalid="ignore"):
        want = O.density_filter_apply(Nx, Ny, W, H, r, x)
    got = dem.create_density_filter(r, dem.Mesh(Nx, Ny, W, H)) @ x
    assert np.array_equal(got, want, equal_nan=True)
