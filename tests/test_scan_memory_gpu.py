"""Scratch memory that a scan can do without (the bitmap of a scan whose rays have no range
limit) is held within the map's budget; without it the scan gives the same map."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

MB = 1 << 20
INF = float("inf")


def clouds(seed, k, n=4000, far=30.0):
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(k):
        d = rng.normal(size=(n, 3))
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        out.append((d * rng.uniform(1, far, (n, 1))).astype(np.float32))
    return out


def free_bytes():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def same(gmap, omap):
    assert all(np.array_equal(a, b) for a, b in zip(gmap.dump(), omap.dump()))


# 14 k leaves at most, 30 MB: the bitmap of 147 MB fits behind the pools, or never, or only
# until the pools have grown
@pytest.mark.parametrize("budget,leaves", [(0, 16384), (100 * MB, 16384), (170 * MB, 0)])
def test_scans_without_a_range_limit(gpu, port, budget, leaves):
    scans = clouds(1, 6, 1000, 12.0)
    m = gpu.ProbabilisticMap(0.1, gpu.Config(pool_budget_bytes=budget, initial_leaves=leaves))
    o = port.pmap(0.1)
    for k, p in enumerate(scans):
        m.insert_point_cloud(p[:200], np.zeros(3, np.float32), 2.0)  # buffers of the staging
        o.insert(p[:200], np.zeros(3, np.float32), 2.0)
        before = free_bytes()
        assert m.insert_point_cloud(p, np.zeros(3, np.float32), INF) == \
            o.insert(p, np.zeros(3, np.float32), INF)
        if k == 0 and leaves:  # no pool grows: the bitmap, and some hundred bytes a point
            assert before - free_bytes() < (8 * MB if budget else 155 * MB)
        if budget:
            assert m.mem_usage() <= budget
    same(m, o)


def test_a_tick_without_a_range_limit(gpu, port):
    maps = [gpu.ProbabilisticMap(0.1, gpu.Config(pool_budget_bytes=b))
            for b in (0, 100 * MB, 0)]
    orc = [port.pmap(0.1) for _ in maps]
    b = gpu.Batch()
    for k in range(3):
        scans = clouds(10 + k, len(maps), 2000, 12.0)
        off = np.arange(len(maps) + 1) * 2000
        got = b.insert(maps, np.concatenate(scans), off, np.zeros((len(maps), 3)),
                       [INF, INF, 10.0])
        assert [int(v) for v in got] == [o.insert(p, np.zeros(3, np.float32), r)
                                         for o, p, r in zip(orc, scans, (INF, INF, 10.0))]
    for m, o in zip(maps, orc):
        same(m, o)


def test_a_server_without_a_range_limit(gpu, port):
    """The bitmaps of a server's maps are within its budget, behind the pools."""
    n, budget = 6, 400 * MB
    first = gpu.Server([0.2])  # loads the kernels
    first.wait_insert(first.insert(0, clouds(0, 1, 100)[0], np.zeros(3, np.float32), INF))
    first.close()
    before = free_bytes()
    s = gpu.Server([0.2] * n, gpu.ServerConfig(pool_budget_bytes=budget))
    orc = [port.pmap(0.2) for _ in range(n)]
    for k in range(4):
        scans = clouds(20 + k, n, 1000, 20.0)
        tickets = [s.insert(i, p, np.zeros(3, np.float32), INF) for i, p in enumerate(scans)]
        for t, p, o in zip(tickets, scans, orc):
            assert s.wait_insert(t)["ray_cells"] == o.insert(p, np.zeros(3, np.float32), INF)
    s.drain()
    # beside the budget: the lists and tables of ticks of 6,000 points
    assert before - free_bytes() < budget + 64 * MB
    for i, o in enumerate(orc):
        assert all(np.array_equal(a, b) for a, b in zip(s.map_dump(i), o.dump()))
    s.close()


@pytest.fixture
def alloc_limit(gpu):
    """Sets the largest request for device memory that does not fail."""
    lib = gpu.load_library()
    yield lib.bxg_debug_alloc_limit
    lib.bxg_debug_alloc_limit(2**64 - 1)


def sphere(rng, n, radius):
    """n points in all directions; far ones in a cone, which crosses few leaves."""
    d = rng.normal(size=(n, 3))
    if radius > 20:
        d = d * (0.0, 0.05, 0.05) + (1.0, 0.0, 0.0)
    return (d / np.linalg.norm(d, axis=1, keepdims=True) * radius).astype(np.float32)


# the first scans' buffers are made before the limit: then only the list of segments has to
# grow, or the bitmap (and what follows it), or the list of rays that leave the cube
@pytest.mark.parametrize("warm,max_range", [((10.0, 100), 10.0), ((3.0, 100), 10.0),
                                            ((INF, 100), INF)])
def test_a_scan_that_finds_no_memory_for_its_lists(gpu, port, alloc_limit, warm, max_range):
    rng = np.random.default_rng(7)
    n, zero = 60000, np.zeros(3, np.float32)
    m = gpu.ProbabilisticMap(0.1, gpu.Config(initial_leaves=1 << 17, initial_inners=1 << 13,
                                             hash_buckets=1 << 15))
    o = port.pmap(0.1)
    big = [sphere(rng, n, 9.0 if np.isfinite(max_range) else 60.0) for _ in range(3)]
    first = [(sphere(rng, n, 2.0), 2.5), (big[0][:warm[1]], warm[0])]
    for p, r in first:
        assert m.insert_point_cloud(p, zero, r) == o.insert(p, zero, r)
    p = sphere(rng, n, 2.0).astype(np.float64)  # the table of a scan without a bitmap
    m.add_hit_points(p)
    o.add_hit(p)
    assert m.update_free_cells(np.zeros(3)) == o.update_free_cells(np.zeros(3))
    assert alloc_limit(60000) == 0  # less than four bytes a point
    for p in big:
        assert m.insert_point_cloud(p, zero, max_range) == o.insert(p, zero, max_range)
    alloc_limit(2**64 - 1)
    for p in big:
        assert m.insert_point_cloud(p, zero, max_range) == o.insert(p, zero, max_range)
    same(m, o)


@pytest.mark.parametrize("max_range", [10.0, INF])
def test_a_tick_that_finds_no_memory_for_its_lists(gpu, port, alloc_limit, max_range):
    rng = np.random.default_rng(8)
    n, k, zero = 20000, 3, np.zeros((3, 3), np.float32)
    cfg = gpu.Config(initial_leaves=1 << 17, initial_inners=1 << 13, hash_buckets=1 << 15)
    maps = [gpu.ProbabilisticMap(0.1, cfg) for _ in range(k)]
    orc = [port.pmap(0.1) for _ in range(k)]
    b = gpu.Batch()

    def tick(scans, r):
        off = np.concatenate([[0], np.cumsum([len(p) for p in scans])])
        got = b.insert(maps, np.concatenate(scans), off, zero, r)
        assert [int(v) for v in got] == [w.insert(p, z, r) for w, p, z in zip(orc, scans, zero)]

    tick([sphere(rng, n, 2.0) for _ in maps], 2.5)
    tick([sphere(rng, 50, 9.0) for _ in maps], max_range)
    assert alloc_limit(60000) == 0
    for _ in range(2):
        tick([sphere(rng, n, 9.0 if np.isfinite(max_range) else 60.0) for _ in maps], max_range)
    alloc_limit(2**64 - 1)
    tick([sphere(rng, n, 9.0) for _ in maps], max_range)
    for m, o in zip(maps, orc):
        same(m, o)


def test_loading_over_the_same_leaves_needs_no_pool(gpu, alloc_limit):
    """A file whose leaves the grid has is loaded without memory for other ones."""
    rng = np.random.default_rng(9)
    leaf = np.stack(np.meshgrid(*[np.arange(8)] * 3, indexing="ij"), -1).reshape(-1, 3) * 8
    xyz = np.concatenate([leaf + rng.integers(0, 8, leaf.shape) for _ in range(3)])
    xyz = np.unique(xyz, axis=0).astype(np.int32)
    g = gpu.VoxelGrid(0.1, dtype=np.float32, config=gpu.Config(initial_leaves=700))
    g.set_values(xyz, rng.normal(size=len(xyz)).astype(np.float32))
    want, saved = g.dump(), g.serialize()
    g.set_values(xyz, np.zeros(len(xyz), np.float32))
    assert alloc_limit(1 << 20) == 0  # the pool of 700 leaves has more
    g.deserialize(saved)
    assert all(np.array_equal(a, b) for a, b in zip(g.dump(), want))
