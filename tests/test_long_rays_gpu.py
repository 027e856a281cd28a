"""Rays that leave the cube of a scan without a range limit: few of them (walked in many
pieces each), some, and so many that a warp walks each whole."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

RES = 0.05


def rays(rng, n, lo, hi):
    """n points lo to hi cells away, in a cone around an axis (few leaves are crossed)."""
    d = np.concatenate([np.ones((n, 1)), rng.uniform(-0.15, 0.15, (n, 2))], 1)
    return (d * rng.uniform(lo, hi, (n, 1)) * RES).astype(np.float32)


@pytest.mark.parametrize("n,lo,hi", [(3, 500, 9000), (800, 510, 530), (800, 480, 3000),
                                     (5000, 300, 1200), (45000, 400, 650)])
@pytest.mark.parametrize("max_range", [np.inf, 900 * RES])
def test_long_rays_vs_oracle(gpu, port, n, lo, hi, max_range):
    rng = np.random.default_rng(n)
    m = gpu.ProbabilisticMap(RES, gpu.Config(initial_leaves=1 << 16))
    o = port.pmap(RES)
    for k in range(2):
        org = np.array([0.4 * k, -0.1, 0.2], np.float32)
        p = org + rays(rng, n, lo, hi)
        assert m.insert_point_cloud(p, org, max_range) == o.insert(p, org, max_range)
    assert all(np.array_equal(a, b) for a, b in zip(m.dump(), o.dump()))


def test_all_rays_long_no_slower_than_on_the_tree(gpu):
    rng = np.random.default_rng(1)
    scans = [torch.from_numpy(rays(rng, 100000, 780, 790)).cuda() for _ in range(4)]
    maps = [gpu.ProbabilisticMap(RES, gpu.Config(flags=f | gpu.FLAG_TIMING,
                                                  initial_leaves=1 << 17))
            for f in (0, gpu.FLAG_RAYS_SINGLE_PASS)]
    took = [[], []]
    for k in range(16):
        for m, t in zip(maps, took):
            m.insert_point_cloud(scans[k % 4], np.zeros(3, np.float32), np.inf)
            t.append(m.kernel_times()[3])
    # 0.85 of it for a LiDAR's 131 k rays of 800 cells; 2.9 with 32 pieces for each ray
    assert np.median(took[0][8:]) < 1.5 * np.median(took[1][8:])


@pytest.mark.parametrize("cells,n,on_tree", [(769, 60000, True), (1020, 2000, True),
                                             (1100, 2000, False)])
def test_ranges_above_the_cube(gpu, port, cells, n, on_tree):
    """Scans of a range just above the largest cube are walked on the tree: by one kernel after
    those of the endpoints and winners, not by three."""
    rng = np.random.default_rng(cells)
    m = gpu.ProbabilisticMap(RES, gpu.Config(initial_leaves=1 << 16))
    o = port.pmap(RES)
    for _ in range(2):
        p = rays(rng, n, 300, 1.5 * cells)
        before = m.last_stats()["launches"]
        assert m.insert_point_cloud(p, np.zeros(3, np.float32), cells * RES) == \
            o.insert(p, np.zeros(3, np.float32), cells * RES)
    assert m.last_stats()["launches"] - before == (3 if on_tree else 5)
    assert all(np.array_equal(a, b) for a, b in zip(m.dump(), o.dump()))
