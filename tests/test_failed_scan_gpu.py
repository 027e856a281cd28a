"""The rays of a scan that failed stay queued and are cast by the next updateFreeCells or scan,
from its origin: nothing that was made for the failed scan's origin may be used for them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RES = 0.1


def failed_scan(gpu, pts, max_range):
    """A map whose scan from (0, 0, 0) ran out of a wait on the origin's leaf."""
    m = gpu.ProbabilisticMap(RES)
    lib = gpu.load_library()
    held = np.zeros(3, np.int32)
    assert lib.bxg_debug_hold_leaf(lib.bxg_pmap_grid(m.h), held.ctypes.data) == 0
    with pytest.raises(gpu.BonxaiError) as ei:
        m.insert_point_cloud(pts, np.zeros(3, np.float32), max_range)
    assert ei.value.status == 4  # BXG_ERR_WAIT_TIMEOUT
    return m


def cells_of(pmap):
    xyz, c = pmap.dump()
    return {tuple(k): w for k, w in zip(xyz.tolist(), c.tolist())}


# from beyond the points (rays that are longer or shorter than the failed scan's), from beside
# them, and further away than the failed scan's range
@pytest.mark.parametrize("origin", [(14.0, 0.2, 0.1), (7.5, 6.0, 0.3), (40.0, 1.0, -2.0)])
@pytest.mark.parametrize("max_range", [12.0, np.inf])
@pytest.mark.parametrize("by_scan", [False, True])
def test_rays_of_a_failed_scan_from_another_origin(gpu, port, origin, max_range, by_scan):
    rng = np.random.default_rng(int(origin[0]))
    pts = rng.uniform((6, -2, -2), (9, 2, 2), (3000, 3)).astype(np.float32)
    m = failed_scan(gpu, pts, max_range)
    org = np.array(origin)
    expected = []
    for o in (np.zeros(3), org):  # the cells that each of the origins' rays visit
        om = port.pmap(RES)
        om.add_hit(pts.astype(np.float64))
        n = om.update_free_cells(o)
        expected.append(cells_of(om))
    if by_scan:
        assert m.insert_point_cloud(np.zeros((0, 3), np.float32), org.astype(np.float32),
                                    max_range) >= n
    else:
        assert m.update_free_cells(org) == n
    first, second = expected
    got = cells_of(m)
    assert all(got.get(k) == w for k, w in second.items())
    assert all(first.get(k, second.get(k)) == w for k, w in got.items())
    # no ray is queued any more
    assert m.update_free_cells(org) == 0
    m.grid().clear()
    m.synchronize()
