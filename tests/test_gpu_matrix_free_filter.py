"""The Helmholtz filter with its finest level matrix-free (TOPO_STENCIL_NODES below that level's
node count, so that set-up times the column march on it) against the assembled default.  Both
solves stop at a relative residual of 1e-12; the filter matrix scaled by the lumped mass has
eigenvalues between 1/4 and 1 + 12 eps^2 max(1/hx, 1/hy)^2 < 40 here, so the solutions agree to
2e-12 * 160 < 1e-9."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(64, 32), (65, 33), (127, 40)])
def test_matrix_free_finest_level(nx, ny, monkeypatch):
    import topomax_gb300 as tg

    V = tg.FunctionSpace(tg.RectangleMesh(2.0, 1.0, nx, ny), "CG", 1)
    f = np.random.default_rng(nx).uniform(0.0, 1.0, V.dim())
    want = tg.HelmholtzFilter(0.02, V, rtol=1e-12).apply(f).tensor.cpu().numpy()
    monkeypatch.setenv("TOPO_STENCIL_NODES", str(V.dim() - 1))
    got = tg.HelmholtzFilter(0.02, V, rtol=1e-12).apply(f).tensor.cpu().numpy()
    assert np.linalg.norm(got - want) <= 1e-9 * np.linalg.norm(want)
