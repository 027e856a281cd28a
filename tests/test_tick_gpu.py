"""Batched ticks in the two-phase form: scans without points, of one point and of a few
around the 256 points of a chunk, without a range limit (rays past the cube), many scans,
and ticks of other sizes on the same batch, bit-exact with the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(rng, n, reach, origin):
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True) + 1e-9
    return (origin + d * reach * rng.uniform(0.02, 1.5, (n, 1))).astype(np.float32)


@pytest.mark.parametrize("n_maps,sizes,max_range", [
    (7, [0, 1, 255, 256, 257, 0, 3000], 6.0),
    (5, [700, 0, 40, 513, 1], float("inf")),
    (128, [1, 37, 0, 300], 4.0),
])
def test_tick_forms_vs_oracle(gpu, port, n_maps, sizes, max_range):
    rng = np.random.default_rng(n_maps)
    res = [0.05, 0.1, 0.2]
    batch = gpu.Batch()
    maps = [gpu.ProbabilisticMap(res[i % 3]) for i in range(n_maps)]
    want = [port.pmap(res[i % 3]) for i in range(n_maps)]
    for tick in range(3):
        use = list(range(n_maps))[: n_maps - tick]  # other tick sizes on the same batch
        scans = []
        for i in use:
            o = np.array([0.3 * tick, -0.1 * i, 1.0], np.float32)
            scans.append((_points(rng, sizes[(i + tick) % len(sizes)], 60.0 if np.isinf(max_range)
                                  and i % 2 else 5.0, o), o))
        off = np.concatenate([[0], np.cumsum([len(p) for p, _ in scans])])
        got = batch.insert([maps[i] for i in use], np.concatenate([p for p, _ in scans]), off,
                           np.stack([o for _, o in scans]), max_range)
        for k, i in enumerate(use):
            assert got[k] == want[i].insert(scans[k][0], scans[k][1], max_range), (tick, i)
    for i in range(n_maps):
        gx, gc = maps[i].dump()
        ox, oc = want[i].dump()
        assert np.array_equal(gx, ox) and np.array_equal(gc, oc), i
    # a map's own scans and its ticks share its bitmap
    p, o = _points(rng, 2000, 5.0, 0.0), np.zeros(3, np.float32)
    assert maps[0].insert_point_cloud(p, o, 5.0) == want[0].insert(p, o, 5.0)
    assert np.array_equal(maps[0].dump()[1], want[0].dump()[1])
