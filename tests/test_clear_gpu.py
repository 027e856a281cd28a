"""clear() of grids of every value size and node size after different amounts of use: what
is written afterwards is all there is, as in a new grid."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [None, np.uint8, np.int16, np.float32, np.float64])
@pytest.mark.parametrize("ib,lb", [(1, 1), (2, 3), (3, 2), (1, 5)])
def test_nothing_survives_a_clear(gpu, dtype, ib, lb):
    rng = np.random.default_rng(ib * 7 + lb)
    g = gpu.VoxelGrid(0.1, ib, lb, dtype=dtype,
                      config=gpu.Config(initial_leaves=3, initial_inners=1, hash_buckets=16))
    for k, n in enumerate((1, 3000, 0, 40, 20000, 7)):
        xyz = np.unique(rng.integers(-60 - 40 * k, 70, (n, 3)).astype(np.int32), axis=0) \
            if n else np.zeros((0, 3), np.int32)
        if dtype is None:
            g.set_cells_on(xyz)
        else:
            vals = rng.integers(1, 100, len(xyz)).astype(dtype)
            g.set_values(xyz, vals)
        if k == 3:
            g.set_cells_off(xyz[::2])
            g.release_unused_memory()  # free slots, which a clear forgets
        else:
            a, av = g.dump()
            assert np.array_equal(a, xyz)
            if dtype is not None:
                assert np.array_equal(av, vals)
        # cells turned on without a value read as zero everywhere
        g.clear()
        assert g.active_cells_count() == 0 and g.node_counts() == (0, 0)
        ask = np.concatenate([xyz, xyz + 1])
        if len(ask):
            v, f = g.get_values(ask, create=True)
            assert f.all() and (dtype is None or not np.any(v))
            g.clear()


def test_map_clear_and_scan(gpu, port):
    rng = np.random.default_rng(1)
    m = gpu.ProbabilisticMap(0.1)
    for k in range(3):
        p = rng.uniform(-6 - k, 6, (4000, 3)).astype(np.float32)
        m.insert_point_cloud(p, np.zeros(3, np.float32), 5.0)
        m.clear()
        o = port.pmap(0.1)
        for _ in range(k + 1):  # the counter is kept by clear()
            o.update_free_cells(np.zeros(3))
        assert m.insert_point_cloud(p, np.zeros(3, np.float32), 5.0) == \
            o.insert(p, np.zeros(3, np.float32), 5.0)
        a, ac = m.dump()
        b, bc = o.dump()
        assert np.array_equal(a, b) and np.array_equal(ac >> 4, bc >> 4)
        m.clear()
