"""Batch statistics are those of the last tick, whatever its form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_grid_of_the_last_tick(gpu):
    rng = np.random.default_rng(0)
    two_phase, single = (gpu.ProbabilisticMap(0.1, gpu.Config(flags=f))
                         for f in (0, gpu.FLAG_RAYS_SINGLE_PASS))
    b = gpu.Batch()

    def tick(m):
        b.insert([m], rng.uniform(-3, 3, (100, 3)).astype(np.float32), [0, 100], np.zeros((1, 3)),
                 5.0)
        return b.stats()["grid"]

    mark = tick(two_phase)
    persistent = tick(single)
    assert mark > 0 and persistent > 0 and mark != persistent
    assert tick(two_phase) == mark
    assert tick(single) == persistent
