"""Maps that time their kernels: calls without some of the phases leave no error behind."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", ["empty scan", "update", "queued"])
def test_first_call_without_all_phases(gpu, port, first):
    m = gpu.ProbabilisticMap(0.1, gpu.Config(flags=gpu.FLAG_TIMING))
    o = port.pmap(0.1)
    zero, pts = np.zeros(3, np.float32), np.ones((5, 3), np.float32)
    for x in (m, o):
        if first == "empty scan":
            (x.insert_point_cloud if x is m else x.insert)(pts[:0], zero, 5.0)
        elif first == "update":
            x.update_free_cells(np.zeros(3))
        else:
            (x.add_hit_points if x is m else x.add_hit)(np.ones((2, 3)))
            x.update_free_cells(np.zeros(3))
    assert m.insert_point_cloud(pts, zero, 5.0) == o.insert(pts, zero, 5.0)
    assert all(np.array_equal(a, b) for a, b in zip(m.dump(), o.dump()))
    assert all(np.isfinite(t) and t >= 0 for t in m.kernel_times())
