"""A level's coefficients are made for as many Chebyshev steps as its sweeps take: a degree without
kernels counts as two (csrc/topo_p1level.cuh)."""
import pytest


@pytest.mark.parametrize("single", [0, 1])
@pytest.mark.parametrize("NC", [1, 2])
def test_only_degrees_with_kernels(single, NC):
    from tests.native.build_emulator import load
    have = {2, 4} if single and NC == 2 else {2}
    for wanted in range(1, 7):
        assert load().emu_sweep_degree(single, NC, wanted) == (wanted if wanted in have else 2)
