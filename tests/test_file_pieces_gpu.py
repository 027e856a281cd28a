"""Saving a map takes a bounded piece of device memory, whatever the size of its file."""
import struct

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIDE = 264  # 9^3 roots of 32 cells, the last ones a quarter full: 74 MB of values


def dense_file():
    """The file of a cube of SIDE cells a side that hold their index, and its cells."""
    at = np.arange(SIDE, dtype=np.int64)
    index = (at[:, None, None] * SIDE + at[:, None]) * SIDE + at  # [x, y, z]
    value = index.astype(np.float32)
    full = np.full(8, -1, np.int64).tobytes()
    out = [b"Bonxai::VoxelGrid<float,2,3>(%f)\n" % 0.5]
    keys = range(0, SIDE, 32)
    out.append(struct.pack("<I", len(keys) ** 3))
    for x in keys:
        for y in keys:
            for z in keys:
                n = [min(4, (SIDE - c) // 8) for c in (x, y, z)]
                leaves = [(i, j, k) for k in range(n[2]) for j in range(n[1]) for i in range(n[0])]
                mask = sum(1 << (i + 4 * j + 16 * k) for i, j, k in leaves)
                out.append(struct.pack("<iiiQ", x, y, z, mask))
                for i, j, k in leaves:
                    a, b, c = x + 8 * i, y + 8 * j, z + 8 * k
                    cells = value[a:a + 8, b:b + 8, c:c + 8].transpose(2, 1, 0)
                    out += [full, np.ascontiguousarray(cells).tobytes()]
    return b"".join(out)


def test_file_larger_than_a_piece(gpu):
    want = dense_file()
    leaves = (SIDE // 8) ** 3
    g = gpu.VoxelGrid(0.5, dtype=np.float32, config=gpu.Config(initial_leaves=2 * leaves))
    g.deserialize(want)
    assert g.active_cells_count() == SIDE ** 3
    small = gpu.VoxelGrid(0.5, dtype=np.float32)
    small.set_values(np.zeros((1, 3), np.int32), np.ones(1, np.float32))
    assert len(small.serialize()) < 4096  # its kernels are loaded
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    got = g.serialize()
    # a piece of 64 MB and the list of roots
    assert before - torch.cuda.mem_get_info()[0] <= 68 << 20
    assert len(got) == len(want) and got == want
