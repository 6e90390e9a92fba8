"""topo_fluid_launch_count against the kernels that the profiler sees, per iteration."""
import pytest

pytestmark = pytest.mark.gpu


def _solve(n, rtol):
    """(iterations, counted launches, kernels seen) of one host-driven state solve."""
    import torch
    import topomax_gb300 as tg
    from topomax_gb300.designs import parse_design_dict
    dom, par = parse_design_dict({"Fluid": {
        "domain_parameters": dict(width=1.0, height=1.0, fem_step_size=0.001, dem_step_size=0.001, penalties=[0.1],
                                  volume_fraction=0.5),
        "problem_parameters": dict(flows=[dict(side="Left", center=0.5, length=1.0, rate=1.0),
                                          dict(side="Right", center=0.5, length=1.0, rate=-1.0)], viscosity=1.0)}})
    mesh = tg.RectangleMesh(1.0, 1.0, n, n)
    prob = tg.FluidProblem(mesh, par, dom, rtol=rtol)
    prob.set_penalization(0.1)
    rho = torch.full(((n + 1) ** 2,), 0.5, dtype=torch.float64, device="cuda")
    prob.forward(rho)
    i0, l0 = prob.stats["state_iterations"], prob.launch_count()
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        prob.forward(rho)
        torch.cuda.synchronize()
    seen = sum(e.count for e in prof.key_averages() if "topo::" in e.key or "k_fluid" in e.key or "k_krylov" in e.key)
    return prob.stats["state_iterations"] - i0, prob.launch_count() - l0, seen


def test_launches_per_iteration_are_the_kernels_that_run(monkeypatch):
    monkeypatch.setenv("TOPO_GRAPHS", "0")
    _solve(24, 1e-2)  # (a process's first profile can be empty)
    few, many = _solve(24, 1e-2), _solve(24, 1e-5)  # one restart cycle each
    if not (few[2] and many[2]):
        pytest.skip("no profiler")
    assert few[0] < many[0] < 60
    assert many[1] - few[1] == many[2] - few[2]
    assert (many[1] - few[1]) % (many[0] - few[0]) == 0
