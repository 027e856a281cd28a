"""Scans of more than 2^24 rays: the list of segments against the walk on the tree."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [270])  # 19.7 M endpoint cells, each with a ray of its own
def test_rays_past_24_bits(gpu, side):
    res = 0.25
    at = (torch.arange(side, device="cuda", dtype=torch.float32) - side // 2 + 0.5) * res
    pts = torch.cartesian_prod(at, at, at).contiguous()
    origin = np.array([0.1, 0.1, 0.1], np.float32)
    files, stats = [], []
    for flags in (0, gpu.FLAG_RAYS_SINGLE_PASS):
        m = gpu.ProbabilisticMap(res, gpu.Config(flags=flags, initial_leaves=1 << 16))
        v = m.insert_point_cloud(pts, origin, 1000 * res / 2)
        s = m.last_stats()
        stats.append((v, s["cast_rays"], s["ray_cells_visited"], s["ray_cells_updated"]))
        files.append(m.grid().serialize())
        m.close()
    assert stats[0][1] > 1 << 24
    assert stats[0] == stats[1] and files[0] == files[1]
