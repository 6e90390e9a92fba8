"""Evaluations that share a context each keep their own Dirichlet mask.  Equal bits throughout."""
import pytest

from test_gpu_dem_evaluation import _setup

pytestmark = pytest.mark.gpu


def _grads(energy, enf, u, rho):
    import torch
    a, b = u.clone().requires_grad_(True), rho.clone().requires_grad_(True)
    return torch.autograd.grad(energy.calculate_energy_enforced(a, enf, b), (a, b))


@pytest.mark.parametrize("nx,ny", [(1, 1), (9, 6), (40, 33)])
def test_backward_uses_the_mask_of_its_forward(nx, ny):
    import torch
    _, energy, left, top, u, rho = _setup(nx, ny)
    want = [_grads(energy, e, u, rho) for e in (left, top)]
    leaves = [(u.clone().requires_grad_(True), rho.clone().requires_grad_(True)) for _ in range(2)]
    psi = [energy.calculate_energy_enforced(a, e, b) for e, (a, b) in zip((left, top), leaves)]
    for k in (0, 1, 0):  # first, second, and the first again
        got = torch.autograd.grad(psi[k], leaves[k], retain_graph=True)
        assert torch.equal(got[0], want[k][0]) and torch.equal(got[1], want[k][1])


def test_an_enforcer_applies_its_own_mask():
    import torch
    _, energy, left, top, u, rho = _setup(9, 6)
    for enf in (left, top):  # both in the energy's context now, the second one's mask on the device
        energy.calculate_energy_enforced(u, enf, rho)
    for enf in (left, top, left):
        assert torch.equal(enf(u), u * torch.from_numpy(enf._mask).cuda())


def test_a_new_mask_waits_for_queued_evaluations():
    """On a stream that does not wait for the default stream's copies."""
    import torch
    _, energy, left, top, u, rho = _setup(40, 33)
    want = [energy.calculate_energy_enforced(u, e, rho).item() for e in (left, top)]
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        torch.cuda._sleep(20_000_000)  # some 10 ms
        got = [energy.calculate_energy_enforced(u, e, rho) for e in (left, top, left)]
    torch.cuda.synchronize()
    assert [g.item() for g in got] == [want[0], want[1], want[0]]
