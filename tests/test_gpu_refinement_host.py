"""The refinement launched from the host is the recorded one kernel by kernel: equal bits, with
graphs off (as after a recording that failed) and traced."""
import numpy as np
import pytest

from test_gpu_parity import _design, _gpu_problem

pytestmark = pytest.mark.gpu


def _run(nx, ny, monkeypatch, **env):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    prob, V = _gpu_problem(_design(), nx, ny, rtol=1e-11)
    rng = np.random.default_rng(nx)
    out = []
    for p, warm in ((3.0, False), (3.0, True), (1.5, False)):  # recorded, replayed, another operator
        prob.warm_start = warm
        prob.set_penalization(p)
        out.append(prob.calculate_objective(rng.uniform(0.2, 1.0, V.dim())))
        out += [prob.u.tensor.clone(), prob.filtered_rho.tensor.clone(), prob.calculate_objective_gradient().tensor.clone()]
    for k in env:
        monkeypatch.delenv(k)
    return out


# the short and the march form of the P2 kernels, the Krylov kernels' small and large form
@pytest.mark.parametrize("nx,ny", [(7, 5), (101, 33), (400, 200), (1000, 500)])
def test_host_driven_solves_give_the_same_bits(nx, ny, monkeypatch):
    import torch
    want = _run(nx, ny, monkeypatch)
    for env in ({"TOPO_GRAPHS": "0"}, {"TOPO_TRACE_SOLVES": "1"}):
        for a, b in zip(_run(nx, ny, monkeypatch, **env), want):
            assert torch.equal(torch.as_tensor(a), torch.as_tensor(b)), env


def test_an_unreached_iteration_limit_changes_no_bit():
    import torch
    got = []
    for limit in (0, 5000):
        prob, V = _gpu_problem(_design(), 101, 33, rtol=1e-11)
        prob.set_penalization(3.0)
        prob.set_iteration_limit(limit)
        prob.calculate_objective(np.random.default_rng(3).uniform(0.2, 1.0, V.dim()))
        got.append(prob.u.tensor.clone())
    assert torch.equal(*got)


def test_the_trace_names_every_step(monkeypatch, capfd):
    import re
    monkeypatch.setenv("TOPO_TRACE_SOLVES", "1")
    prob, V = _gpu_problem(_design(), 40, 20, rtol=1e-11)
    prob.set_penalization(3.0)
    prob.calculate_objective(np.random.default_rng(3).uniform(0.2, 1.0, V.dim()))
    err = capfd.readouterr().err
    inner = re.findall(r"inner (\d+): tol ([\d.e+-]+), (\d+) iterations, FP32 relres ([\d.e+-]+), rc (-?\d+)", err)
    assert len(inner) >= 4 and all(int(i[4]) == 0 and float(i[3]) <= 1.01 * float(i[1]) for i in inner)
    assert len(re.findall(r"fgmres cycle \d+: ", err)) >= 2 and len(re.findall(r"fgmres converged: ", err)) >= 2
