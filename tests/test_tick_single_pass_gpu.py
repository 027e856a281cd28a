"""Batched ticks in the single-pass form, where the lanes of a warp may work for different
maps: every map's nodes come from its own pools, bit-exact with the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(rng, n, origin):
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return (origin + d * rng.uniform(0.5, 12.0, (n, 1))).astype(np.float32)


@pytest.mark.parametrize("rpw,unroll", [(1, 1), (2, 1), (4, 1), (4, 2)])
@pytest.mark.parametrize("flag", ["FLAG_RAYS_SINGLE_PASS", "FLAG_KEEP_NONFINITE"])
@pytest.mark.parametrize("leaves", [0, 65536])  # pools that run out in the tick, and not
def test_single_pass_ticks_vs_oracle(gpu, port, rpw, unroll, flag, leaves):
    rng = np.random.default_rng(rpw)
    # none of them a multiple of a warp: warps straddle two scans, or several
    sizes = [2000, 1, 33, 1501, 5, 7, 1999, 12]
    cfg = gpu.Config(flags=getattr(gpu, flag), initial_leaves=leaves)
    maps = [gpu.ProbabilisticMap(0.1, cfg) for _ in sizes]
    want = [port.pmap(0.1) for _ in sizes]
    batch = gpu.Batch(gpu.Config(rays_per_warp=rpw, ray_unroll=unroll))
    for tick in range(3):
        org = rng.uniform(-1, 1, (len(sizes), 3)).astype(np.float32)
        scans = [_points(rng, sizes[(i + tick) % len(sizes)], o) for i, o in enumerate(org)]
        off = np.concatenate([[0], np.cumsum([len(p) for p in scans])])
        got = batch.insert(maps, np.concatenate(scans), off, org, 10.0)
        assert [int(v) for v in got] == [w.insert(p, o, 10.0)
                                         for w, p, o in zip(want, scans, org)]
    for i, (m, w) in enumerate(zip(maps, want)):
        gx, gc = m.dump()
        ox, oc = w.dump()
        assert np.array_equal(gx, ox) and np.array_equal(gc, oc), i
