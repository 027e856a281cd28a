"""Saved files of every value size and node size, against a file written here from the
grid's dump, and loading of files that name a cell twice or whose bits go past a node."""
import struct

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAMES = {np.uint8: "unsigned char", np.int16: "short", np.float32: "float", np.float64: "double",
         None: "Bonxai::EmptyVoxel"}


def words(bits, n):
    return np.packbits(bits, bitorder="little").tobytes().ljust(8 * max(n // 64, 1), b"\0")


def write_file(name, ib, lb, res, xyz, vals):
    """The file of the cells, roots in ascending order."""
    out = [b"Bonxai::VoxelGrid<%s,%d,%d>(%f)\n" % (name.encode(), ib, lb, res)]
    key = xyz & ~((1 << (ib + lb)) - 1)
    roots = np.unique(key, axis=0)
    out.append(struct.pack("<I", len(roots)))
    im, lm = (1 << ib) - 1, (1 << lb) - 1
    inner = ((xyz >> lb) & im) @ np.array([1, 1 << ib, 1 << (2 * ib)])
    cell = (xyz & lm) @ np.array([1, 1 << lb, 1 << (2 * lb)])
    for r in roots:
        of = np.all(key == r, axis=1)
        has = np.zeros(1 << (3 * ib), np.uint8)
        has[inner[of]] = 1
        out += [r.astype("<i4").tobytes(), words(has, len(has))]
        for i in np.nonzero(has)[0]:
            at = np.nonzero(of & (inner == i))[0]
            at = at[np.argsort(cell[at])]
            on = np.zeros(1 << (3 * lb), np.uint8)
            on[cell[at]] = 1
            out.append(words(on, len(on)))
            if vals is not None:
                out.append(vals[at].tobytes())
    return b"".join(out)


@pytest.mark.parametrize("dtype", list(NAMES))
@pytest.mark.parametrize("ib,lb", [(1, 1), (2, 3), (3, 2), (4, 1), (1, 5)])
@pytest.mark.parametrize("n", [1, 700])
def test_files(gpu, dtype, ib, lb, n):
    rng = np.random.default_rng(ib * 10 + lb + n)
    reach = 3 * (1 << (ib + lb))
    xyz = np.unique(rng.integers(-reach, reach, (n, 3)).astype(np.int32), axis=0)
    vals = None
    if dtype is not None:
        vals = rng.integers(1, 120, len(xyz)).astype(dtype)
    want = write_file(NAMES[dtype], ib, lb, 0.25, xyz, vals)
    g = gpu.VoxelGrid(0.25, ib, lb, dtype=dtype)
    if dtype is None:
        g.set_cells_on(xyz)
    else:
        g.set_values(xyz, vals)
    assert g.serialize() == want
    small = gpu.Config(initial_leaves=1, initial_inners=1, hash_buckets=16)  # grows on the way
    h = gpu.VoxelGrid(0.25, ib, lb, dtype=dtype, config=small)
    h.deserialize(want)
    assert h.serialize() == want
    # loading sets values: cells that are there keep theirs unless the file has them
    more = np.array([[reach + 5, 2, 3], xyz[0]], np.int32)
    k = gpu.VoxelGrid(0.25, ib, lb, dtype=dtype)
    if dtype is None:
        k.set_cells_on(more)
    else:
        k.set_values(more, np.array([7, 99]).astype(dtype))
    k.deserialize(want)
    a, av = k.dump()
    assert len(a) == len(xyz) + 1
    if dtype is not None:
        assert dict(zip(map(tuple, a), av))[tuple(xyz[0])] == vals[0]


def test_files_that_name_cells_twice(gpu):
    xyz = np.array([[1, 2, 3], [9, 9, 9], [-5, 0, 40]], np.int32)
    a = write_file("float", 2, 3, 0.1, xyz, np.array([1, 2, 3], np.float32))
    b = write_file("float", 2, 3, 0.1, xyz[:2], np.array([10, 20], np.float32))
    head = a.index(b"\n") + 1
    both = a[:head] + struct.pack("<I", 3) + a[head + 4:] + b[head + 4:]  # a root comes again
    g = gpu.VoxelGrid(0.1)
    g.deserialize(both)
    x, v = g.dump()
    assert dict(zip(map(tuple, x.tolist()), v.tolist())) == \
        {(1, 2, 3): 10.0, (9, 9, 9): 20.0, (-5, 0, 40): 3.0}
    for cut in (head + 2, head + 10, len(a) - 1):
        h = gpu.VoxelGrid(0.1)
        with pytest.raises(gpu.BonxaiError):
            h.deserialize(a[:cut])
        assert h.active_cells_count() == 0
