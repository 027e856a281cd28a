"""An asynchronous scan captured into a graph by its caller: the kernels that follow one
another as programmatic dependents keep their order in the graph."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,max_range", [(300, 8.0), (20000, 8.0), (20000, float("inf"))])
def test_captured_scan_equals_a_call(gpu, n, max_range):
    import torch
    rng = np.random.default_rng(n)
    stream = torch.cuda.Stream()
    a = gpu.ProbabilisticMap(0.1, config=gpu.Config(stream=stream.cuda_stream))
    b = gpu.ProbabilisticMap(0.1)
    pts = [torch.tensor((rng.normal(size=(n, 3)) * 4).astype(np.float32), device="cuda")
           for _ in range(6)]
    org = [np.array([0.1 * k, 0, 0], np.float32) for k in range(6)]
    torch.cuda.synchronize()
    for k in range(5):  # the last one through the form that is captured
        if k < 4:
            a.insert_point_cloud(pts[k], org[k], max_range)
        else:
            a.insert_point_cloud_async(pts[k], org[k], max_range)
            a.synchronize()
        b.insert_point_cloud(pts[k], org[k], max_range)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        a.insert_point_cloud_async(pts[5], org[5], max_range)
    graph.replay()
    torch.cuda.synchronize()
    a.synchronize()
    b.insert_point_cloud(pts[5], org[5], max_range)
    (ax, ac), (bx, bc) = a.dump(), b.dump()
    assert np.array_equal(ax, bx) and np.array_equal(ac, bc)
