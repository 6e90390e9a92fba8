"""The fluid solve's restart length: the long basis only where it leaves room (csrc/topo_fluid_setup.h)."""
import ctypes

import pytest

GB = 1 << 30
VECTORS = 121  # of the long restart


@pytest.mark.parametrize("n,free,want", [
    (150_000, 250 * GB, 60),
    (16 * GB // (8 * VECTORS), 250 * GB, 60), (16 * GB // (8 * VECTORS) + 1, 250 * GB, 30),
    (10**6, 2 * 8 * VECTORS * 10**6, 60), (10**6, 2 * 8 * VECTORS * 10**6 - 1, 30),  # little memory free
    (10**6, 0, 30), (1 << 29, 280 * GB, 30),
])
def test_restart_length_follows_the_memory(n, free, want):
    from tests import emu
    f = emu.lib().emu_fluid_restart
    f.argtypes = [ctypes.c_longlong] * 2
    assert f(n, free) == want
