"""The march autotuner times only kernels that a solve launches."""
import ctypes

import numpy as np
import pytest

from test_gpu_parity import _design, _gpu_problem

pytestmark = pytest.mark.gpu


def _tiles():
    from topomax_gb300 import _capi
    lib = _capi.load_library()
    buf = ctypes.create_string_buffer(lib.topo_march_tiles_report(None, 0))
    lib.topo_march_tiles_report(buf, len(buf))
    return buf.value.decode()


def test_levels_that_the_sweeps_smooth_are_not_tuned():
    prob, V = _gpu_problem(_design(), 900, 450, rtol=1e-8)  # level 1 is too large for an assembled stencil
    prob.set_penalization(3.0)
    prob.calculate_objective(np.full(V.dim(), 0.5))
    lines = [t.split("\t") for t in _tiles().splitlines()]
    assert any("P2" in t[0] and t[1:3] == ["900", "450"] for t in lines)
    assert not any("P1" in t[0] and t[1:3] == ["900", "450"] for t in lines), lines
