"""Rings of row tiles that several sets of warps take turns on (host logic, no GPU needed)."""

import pytest

from ternel_b200.dispatch import ring_layout

ROWS = (100, 5120, 9000, 17408, 20000, 34816, 50000, 100000, 151936, 262144)
COLUMNS = (*range(512, 5121, 512), 7680, 9728, 10240, 15360, 17408, 19456, 20480, 32768, 40960, 65536)


@pytest.mark.parametrize(("form", "batch"), (("stream_gemv", 1), ("stream_gemv", 2), ("slices", 3), ("slices", 9)))
def test_a_barrier_of_the_ring_belongs_to_one_set(form, batch):
    """A wait for a phase's parity returns at once while the phase before that is still open. So whoever waits for a tile has to have
    waited for the tile before it on the same barrier: tiles on one barrier are whole turns of the sets apart. And a stage is not
    filled again before its tile was read."""
    around = 0
    for columns in COLUMNS:
        for rows in ROWS:
            layout = ring_layout(form, batch, rows, columns) if rows * columns < 1.3e9 else None
            if layout is None:
                continue
            assert 1 <= layout.sets <= 20 and 1 <= layout.stages
            if layout.stages >= layout.tiles:
                continue
            around += 1
            assert layout.stages % layout.sets == 0, (rows, columns, layout)
            assert layout.stages > layout.sets, (rows, columns, layout)
    assert around > 40


@pytest.mark.parametrize(("batch", "rows", "columns"), (
    (1, 60000, 18944), (1, 9000, 25600), (1, 20000, 25600), (1, 34816, 32768), (1, 9000, 49152), (2, 9000, 25600), (2, 20000, 25600)))
def test_wide_matrices_that_the_chain_kernel_is_faster_for(batch, rows, columns):
    """By 6% and more in recorded times: clusters of four and eight CTAs leave SMs idle, and these have work for all of them."""
    assert not ring_layout("stream_gemv", batch, rows, columns).preferred


@pytest.mark.parametrize(("batch", "rows", "columns"), (
    (1, 1024, 5120), (1, 151936, 5120), (1, 34816, 17408), (1, 100000, 10240), (2, 17408, 5120), (2, 5120, 17408), (2, 20000, 10240),
    (1, 1000, 25600), (1, 9000, 20480), (1, 5000, 40960), (2, 5000, 20480), (2, 1000, 40960)))
def test_matrices_that_the_tile_kernel_is_faster_for(batch, rows, columns):
    assert ring_layout("stream_gemv", batch, rows, columns).preferred


def test_cluster_sizes_that_the_device_cannot_run_are_left_out():
    """The driver answers 0 of them; only a machine without a device has no answer (calls are planned for a B200 there)."""
    import ctypes
    from ternel_b200 import _native
    count = _native.lib().tq1_debug_cluster_count
    count.restype, count.argtypes = ctypes.c_int, [ctypes.c_int] * 4
    assert count(1, 33, 1, 4) == 33 and count(1, 0, 1, 16) == 0         # answered
    assert count(0, 0, 1, 16) == 0 and count(0, 0, 0, 16) == 8          # an error, with a device and without one
    none, pairs = {1: 148}, {1: 148, 2: 74}
    for form, batch in (("stream_gemv", 1), ("slices", 8)):
        assert ring_layout(form, batch, 1024, 2560, rooms=none).cluster == 1
        assert ring_layout(form, batch, 5120, 17408).cluster > 1
        assert ring_layout(form, batch, 5120, 17408, rooms=none) is None
        assert ring_layout(form, batch, 1024, 10240, rooms=pairs).cluster == 2
    assert ring_layout("tcgen05", 100, 130, 16384).cluster == 16
    assert ring_layout("tcgen05", 100, 130, 16384, rooms=none).cluster == 1
