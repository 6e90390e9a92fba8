"""A DEM evaluation's Dirichlet mask and gradients: the mask stays on the device between
evaluations, and one launch gives both gradients.  Equal bits throughout."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _setup(nx, ny):
    import torch
    from topomax_gb300 import dem
    from topomax_gb300.designs import ElasticityParameters, Side
    mesh = dem.Mesh(nx, ny, 2.0, 1.0)

    def enforcer(side):
        return dem.ElasticityEnforcer(ElasticityParameters(
            fixed_sides=[side], body_force=None, tractions=None, filter_radius=0.05, young_modulus=1.0,
            poisson_ratio=0.3), mesh)
    energy = dem.StrainEnergy(mesh, None, 1.0, 0.3, None)
    energy.set_penalization(3.0)
    g = torch.Generator().manual_seed(nx)
    u = torch.randn(((nx + 1) * (ny + 1), 2), generator=g).cuda()
    rho = torch.rand((ny, nx), generator=g).cuda()
    return mesh, energy, enforcer(Side.LEFT), enforcer(Side.TOP), u, rho


def test_masks_alternate_and_follow_writes():
    import torch
    mesh, energy, left, top, u, rho = _setup(9, 6)

    def want(enf):
        return energy.calculate_energy(u * torch.from_numpy(enf._mask).cuda(), mesh.shape, rho)

    for enf in (left, top, left, left, top):
        assert torch.equal(energy.calculate_energy_enforced(u, enf, rho), want(enf))
    for k in (1, 2):  # a mask written to through its host array is used as written
        left.mask_host[k] = 0.25 * k
        assert torch.equal(energy.calculate_energy_enforced(u, left, rho), want(left))


@pytest.mark.parametrize("nx,ny", [(1, 1), (16, 15), (17, 16), (300, 260)])
def test_gradients_alone_and_together(nx, ny):
    import torch
    mesh, energy, left, _, u, rho = _setup(nx, ny)
    both = [t.clone().requires_grad_(True) for t in (u, rho)]
    du, dr = torch.autograd.grad(energy.calculate_energy_enforced(both[0], left, both[1]), both)
    a, b = u.clone().requires_grad_(True), rho.clone().requires_grad_(True)
    assert torch.equal(du, torch.autograd.grad(energy.calculate_energy_enforced(a, left, rho), a)[0])
    assert torch.equal(dr, torch.autograd.grad(energy.calculate_energy_enforced(u, left, b), b)[0])
    # other layouts and types of the same values
    c, d = u.double().requires_grad_(True), rho.reshape(-1).clone().requires_grad_(True)
    dc, dd = torch.autograd.grad(energy.calculate_energy_enforced(c, left, d), (c, d))
    assert torch.equal(dc.float(), du) and torch.equal(dd.reshape(ny, nx), dr) and dd.shape == d.shape
    s = u.t().contiguous().t()
    assert torch.equal(energy.calculate_energy_enforced(s, left, rho), energy.calculate_energy_enforced(u, left, rho))
    e = energy.calculate_energy_enforced(u, left, rho)
    assert e.dtype is torch.float32 and e.shape == () and np.isfinite(float(e))
