"""Workspace sizes of the C ABI (host logic)."""

import ctypes

import pytest

from ternel_b200 import _native

SLOTS = 16 << 20


class Link(ctypes.Structure):
    _fields_ = [("blocks", ctypes.c_void_p), ("N", ctypes.c_int), ("K", ctypes.c_int), ("x", ctypes.c_void_p),
                ("source", ctypes.c_int), ("source_offset", ctypes.c_int), ("y", ctypes.c_void_p),
                ("y_is_f32", ctypes.c_int), ("swiglu", ctypes.c_int), ("out_scale", ctypes.c_float),
                ("layout", ctypes.c_int), ("partial", ctypes.c_int)]


@pytest.mark.parametrize("rows,columns", [(131072, 8192), (262144, 4096), (1 << 20, 1024)])
def test_the_slot_region_holds_two_to_the_21_slots(rows, columns):
    """A matrix whose row and K chunk pairs just fill the region is one launch, and so is half of it as a link of a chain."""
    lib = _native.lib()
    assert lib.tq1_linear_workspace_bytes(1, rows, columns) == 256 + SLOTS
    one, half = Link(N=1024, K=1024, blocks=16, x=16), Link(N=rows // 2, K=columns, blocks=16, x=16)
    lib.tq1_chain_table_bytes.restype = ctypes.c_size_t
    assert lib.tq1_chain_table_bytes(ctypes.byref(half), 1) == lib.tq1_chain_table_bytes(ctypes.byref(one), 1)


def test_one_workspace_serves_all_smaller_shapes():
    """Sized for the largest batch, rows and columns, as callers are told to: no smaller call asks for more."""
    import itertools
    bytes_for = _native.lib().tq1_linear_workspace_bytes
    batches = (1, 2, 3, 16, 17, 32, 33, 48, 64, 65, 96, 128, 129, 160, 200, 255, 256, 257, 300, 384, 512, 513, 777, 1100, 2048, 5000)
    rows = (1, 100, 1024, 4099, 5120, 17408, 104800, 104880, 151936, 209600, 250000)
    columns = (512, 1024, 2560, 5120, 17408)
    sizes = {s: bytes_for(*s) for s in itertools.product(batches, rows, columns)}
    for axis, values in enumerate((batches, rows, columns)):
        for shape, size in sizes.items():
            at = values.index(shape[axis])
            if at:
                smaller = shape[:axis] + (values[at - 1],) + shape[axis + 1:]
                assert sizes[smaller] <= size, (smaller, shape)
