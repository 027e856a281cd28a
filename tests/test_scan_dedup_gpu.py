"""The endpoint dedup table of a scan: many points of few cells, endpoints at the faces of the
cube that a scan's cells lie in (packed entries), and scans of any range (unpacked), at the
sizes where the table's entries per point change. Hits and misses of one cell are mixed, so
that the lowest index decides the cell's value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 8192, 8193, 65537])
@pytest.mark.parametrize("res,max_range", [(0.5, 1.2), (0.1, 76.6), (0.1, float("inf"))])
def test_scans_vs_oracle(gpu, port, n, res, max_range):
    rng = np.random.default_rng(n + int(res * 10))
    m, o = gpu.ProbabilisticMap(res), port.pmap(res)
    reach = min(max_range, 76.6)
    for k in range(4):
        org = np.array([[0, 0, 0], [-7.77, 3.1, 0.2], [15.99, -16.01, 31.95], [0, 0, 0]][k], np.float32)
        d = rng.normal(size=(n, 3))
        axis = rng.integers(0, 4, n)  # along an axis: to the faces of the cube
        for a in range(3):
            d[axis == a] = 0
            d[axis == a, a] = rng.choice([-1.0, 1.0], (axis == a).sum())
        d = d[rng.integers(0, max(1, min(n, 200)), n)]  # few directions: shared cells
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        far = rng.choice([0.999, 1.0, 1.001, 2.0, 0.1], (n, 1))  # hits, misses, on the sphere
        pts = (org + reach * far * d).astype(np.float32)
        assert m.insert_point_cloud(pts, org, max_range) == o.insert(pts, org, max_range)
    gx, gc = m.dump()
    ox, oc = o.dump()
    assert np.array_equal(gx, ox) and np.array_equal(gc, oc)
