"""Cells that a caller's own kernel turns off in the masks of bxg_grid_device_view: value()
does not find them and gives T{}, whatever the cell holds."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


class View(C.Structure):
    _fields_ = [("leaf_mask", C.c_void_p), ("leaf_data", C.c_void_p), ("leaf_key", C.c_void_p),
                ("n_leaves", C.c_uint32), ("inner_bits", C.c_int), ("leaf_bits", C.c_int),
                ("value_bytes", C.c_int), ("resolution", C.c_double), ("stream", C.c_void_p)]


class Words:  # 64-bit words of device memory
    def __init__(self, p, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i8", "data": (p, False),
                                         "version": 3}


@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.float32, np.float64])
@pytest.mark.parametrize("ib,lb", [(2, 3), (3, 2)])
def test_values_of_masked_cells(gpu, dtype, ib, lb):
    rng = np.random.default_rng(ib)
    g = gpu.VoxelGrid(0.1, ib, lb, dtype=dtype)
    xyz = np.unique(rng.integers(-40, 40, (5000, 3)).astype(np.int32), axis=0)
    g.set_values(xyz, rng.integers(1, 100, len(xyz)).astype(dtype))
    view = View()
    assert gpu.load_library().bxg_grid_device_view(g.h, C.byref(view)) == 0
    words = view.n_leaves * max(8**lb // 64, 1)
    torch.as_tensor(Words(view.leaf_mask, words), device="cuda").zero_()
    torch.cuda.synchronize()
    values, found = g.get_values(xyz)
    assert not found.any() and not values.any()
