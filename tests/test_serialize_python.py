"""VoxelGrid.serialize around the C entry point, which is replaced by a fake (no GPU)."""
import ctypes as C

import bonxai_gb300 as bx


class Fake:
    """A map that shrinks between the call for the size and the one for the bytes."""

    def __init__(self, sizes):
        self.sizes = sizes

    def bxg_grid_serialize(self, h, name, out, cap, n):
        size = self.sizes.pop(0)
        n._obj.value = size
        if out is not None:
            assert cap >= size
            C.memmove(out, b"0123456789"[:size], size)
        return 0


def grid(sizes):
    g = bx.VoxelGrid.__new__(bx.VoxelGrid)
    g.lib, g.h, g.dtype = Fake(sizes), None, None
    return g


def test_as_many_bytes_as_were_written():
    assert grid([10, 10]).serialize() == b"0123456789"
    assert grid([10, 4]).serialize() == b"0123"


def test_the_interpreters_function_is_left_alone():
    before = C.pythonapi.PyBytes_FromStringAndSize.restype
    grid([10, 10]).serialize()
    assert C.pythonapi.PyBytes_FromStringAndSize.restype is before is C.c_int
