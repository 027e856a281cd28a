"""The occupied export at the edges of its rows and of its blocks of leaves: bands that cut
a leaf, few and many leaves, thresholds, against the map's own dump."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 7, 300, 20000])
def test_export_equals_the_dump(gpu, n):
    rng = np.random.default_rng(n)
    m = gpu.ProbabilisticMap(0.1)
    if n:
        pts = rng.uniform(-12, 12, (n, 3)).astype(np.float32)
        pts[:, 2] *= 0.2
        m.insert_point_cloud(pts, np.zeros(3, np.float32), 15.0)
    for thr in (0, -600000, 10 ** 7):
        o = m.options
        o[4] = thr
        m.options = o
        xyz, cells = m.dump()
        pos = xyz.astype(np.float64) * m.resolution
        for lo, hi in ((-np.inf, np.inf), (0.0, 0.05), (-0.45, 0.73), (0.2, 0.1)):
            keep = ((cells >> 4) > thr) & (pos[:, 2] >= lo) & (pos[:, 2] <= hi)
            want = pos[keep].astype(np.float32)
            want = want[np.lexsort((want[:, 2], want[:, 1], want[:, 0]))]
            got = m.export_occupied(lo, hi)
            assert np.array_equal(got, want), (thr, lo, hi)
