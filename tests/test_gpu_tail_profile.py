"""TOPO_PROFILE=1 reports the phases of the one-block tail; the traced kernel gives the same bits."""
import gc
import re

import numpy as np
import pytest

from test_gpu_parity import _design, _gpu_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", ["0", "1"])
def test_tail_phases_are_reported(graphs, monkeypatch, capfd):
    import torch
    got = []
    for profile in (False, True):
        monkeypatch.setenv("TOPO_GRAPHS", graphs)
        if profile:
            monkeypatch.setenv("TOPO_PROFILE", "1")
        prob, V = _gpu_problem(_design(), 80, 40, rtol=1e-8)
        prob.set_penalization(3.0)
        prob.calculate_objective(np.full(V.dim(), 0.5))
        got.append(prob.u.tensor.clone())
        capfd.readouterr()
        del prob
        gc.collect()
    assert torch.equal(*got)
    line = re.search(r"state32 tail: levels (\d+)\.\., (\d+) launches; k-cycles per phase: (.*)", capfd.readouterr().err)
    first, launches = int(line[1]), int(line[2])
    phases = re.findall(r"([a-z]+)(\d+)=([\d.]+)", line[3])
    assert launches > 0 and all(0.01 < float(c) < 100.0 for _, _, c in phases)
    order = [(p, int(l)) for p, l, _ in phases]
    n = (len(order) - 1) // 2
    assert order == [("down", first + k) for k in range(n)] + [("coarsest", first + n)] + \
        [("up", first + k) for k in reversed(range(n))]
