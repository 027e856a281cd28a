"""Batches of one cell, of few cells and around the sizes of the dedup table and of the blocks
of the grid kernels, last writer (setValue) and first caller (setCellOn/Off) checked
against calls one after the other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 33, 255, 256, 257, 4095, 4097])
@pytest.mark.parametrize("cells", [1, 5, 100000])
def test_batches_equal_single_calls(gpu, n, cells):
    rng = np.random.default_rng(n * 7 + cells)
    pool = rng.integers(-90, 90, (cells, 3)).astype(np.int32)
    state = {}

    def on(c):
        return c in state

    g = gpu.VoxelGrid(0.1, dtype=np.int32)
    for k in range(3):
        xyz = pool[rng.integers(0, cells, n)]
        keys = list(map(tuple, xyz.tolist()))
        vals = rng.integers(1, 1 << 30, n).astype(np.int32)
        want = []
        for c, v in zip(keys, vals):
            want.append(on(c))
            state[c] = int(v)
        got = g.set_values(xyz, vals, return_was_on=k != 1)
        if k != 1:
            assert np.array_equal(got, np.array(want, np.uint8))
        drop = pool[rng.integers(0, cells, max(1, n // 3))]
        want = []
        for c in map(tuple, drop.tolist()):
            want.append(on(c))
            state.pop(c, None)
        assert np.array_equal(g.set_cells_off(drop), np.array(want, np.uint8))
        turn = pool[rng.integers(0, cells, max(1, n // 2))]
        want = []
        for c in map(tuple, turn.tolist()):
            want.append(on(c))
            state.setdefault(c, 77)
        assert np.array_equal(g.set_cells_on(turn, 77), np.array(want, np.uint8))
        ask = np.concatenate([xyz, drop, rng.integers(-95, 95, (50, 3)).astype(np.int32)])
        v, f = g.get_values(ask)
        keys = list(map(tuple, ask.tolist()))
        assert np.array_equal(f, np.array([on(c) for c in keys], np.uint8))
        assert np.array_equal(v, np.array([state.get(c, 0) for c in keys], np.int32))
    a, av = g.dump()
    assert dict(zip(map(tuple, a.tolist()), av.tolist())) == state
