"""A density-filter row's sum and reciprocal are one aligned 16-byte load (csrc/topo_dens.cuh)."""


def test_rows_are_aligned_to_their_size():
    from tests.native.build_emulator import load
    assert load().emu_dens_row_alignment() == 16
