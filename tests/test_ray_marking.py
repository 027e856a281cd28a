"""The marking of ray cells (bonxai_gb300/csrc/bxg_mark.cuh): the closed form of a
cell as one float multiply-add, and scans whose rays end on either side of each limit
of the marking (the shared neighbourhood, a segment, the cube, long rays)."""
from __future__ import annotations

import numpy as np
import pytest

MAX_M, MAX_K = 2047, 801  # kFmaMaxRay; cells of a ray in the largest cube


def fma_steps(k, d, m):
    """floor(fma(k, fl(d/m), 1/2 + 1/(4m))) in float32: the products and sums here
    are exact in float64 (24 + 10 bits), so one rounding to float32 is the fma."""
    s = (d.astype(np.float32) / m.astype(np.float32)).astype(np.float64)
    off = (np.float32(0.5) + np.float32(0.25) / m.astype(np.float32)).astype(np.float64)
    return np.floor((k * s + off).astype(np.float32)).astype(np.int64)


def test_fma_gives_the_bresenham_cell():
    rng = np.random.default_rng(3)
    for m in list(range(1, 130)) + [255, 256, 257, 511, 769, 801, 1023, 1024, 1500, 2046, 2047]:
        d = np.arange(m + 1) if m < 130 else np.unique(
            np.concatenate([rng.integers(0, m + 1, 200), [0, 1, m // 2, m - 1, m]]))
        k = np.arange(min(m, MAX_K))
        kk, dd = (x.ravel() for x in np.meshgrid(k, d))
        mm = np.full(kk.shape, m)
        assert np.array_equal(fma_steps(kk, dd, mm), (2 * kk * dd + m) // (2 * m))
    # the values nearest to an integer: 2 k d + m = -1 mod 2 m
    m = rng.integers(1000, MAX_M + 1, 200_000)
    k = rng.integers(1, MAX_K, 200_000)
    d = np.minimum(m, np.rint((np.rint(k * rng.random(200_000)) + 0.5) * m / k - 0.5).astype(np.int64))
    d = np.maximum(d, 0)
    assert np.array_equal(fma_steps(k, d, m), (2 * k * d + m) // (2 * m))


def _cloud(rng, lengths, res, origin):
    d = rng.normal(size=(len(lengths), 3))
    d /= np.abs(d).max(1, keepdims=True)
    axis = rng.integers(0, 4, len(lengths))  # some rays along an axis or a diagonal
    for a in range(3):
        d[axis == a] = 0
        d[axis == a, a] = rng.choice([-1.0, 1.0], (axis == a).sum())
    d[axis == 3] = rng.choice([-1.0, 1.0], ((axis == 3).sum(), 3))
    keep = rng.random(len(lengths)) < 0.7
    d[keep] = rng.uniform(-1, 1, (keep.sum(), 3))
    d[keep, rng.integers(0, 3, keep.sum())] = 1.0
    return (origin + (np.asarray(lengths)[:, None] + 0.3) * d * res).astype(np.float32)


def test_signed_fma_gives_the_bresenham_cell():
    """floor(fma(k, fl(d fl(1/m)), 1/2 + sign(d)/(4m))), the form with the sign in it."""
    one, q, h = np.float32(1), np.float32(0.25), np.float64(0.5)
    for m in list(range(1, 100)) + [255, 256, 257, 511, 769, 801, 1023, 1024, 1500, 2046, 2047]:
        d = np.arange(-m, m + 1) if m < 100 else np.unique(np.concatenate(
            [np.random.default_rng(m).integers(-m, m + 1, 400), [-m, 1 - m, -1, 0, 1, m - 1, m]]))
        inv = one / np.float32(m)
        s = (d.astype(np.float32) * inv).astype(np.float64)
        off = (h + np.where(d < 0, -q, q).astype(np.float64) * np.float64(inv)).astype(np.float32)
        k = np.arange(min(m, MAX_K))[:, None]
        got = np.floor((k * s + off.astype(np.float64)).astype(np.float32)).astype(np.int64)
        assert np.array_equal(got, np.sign(d) * ((2 * k * np.abs(d) + m) // (2 * m)))


@pytest.mark.gpu
@pytest.mark.parametrize("res,max_range", [
    (0.1, 0.25),           # one root on each side of the origin's
    (0.1, 3.0), (0.1, 3.1),     # 32 and 33 cells: one and two roots
    (0.1, 76.6), (0.1, 76.8),   # the largest cube, and one cell more
    (0.05, 25.0),
    (0.25, float("inf")),
])
def test_rays_around_the_limits(gpu, port, res, max_range):
    rng = np.random.default_rng(int(res * 100) + 7)
    edges = [1, 2, 24, 25, 26, 31, 32, 33, 56, 57, 58, 88, 89, 90, 255, 256, 257, 511, 512, 513, 514,
             767, 768, 769, 770, 2046, 2047, 2048, 2049, 5000]
    lengths = np.array(edges * 6 + [32767, 32768, 40000] + list(np.exp(rng.uniform(0, 7.5, 1500))))
    m = gpu.ProbabilisticMap(res)
    o = port.pmap(res)
    for k in range(4):
        org = np.array([0.31 * k - 7.77, 13.3 + 0.5 * k, -0.05], np.float32)
        pts = _cloud(rng, lengths, res, org)
        assert m.insert_point_cloud(pts, org, max_range) == o.insert(pts, org, max_range)
        if k == 2:  # rays queued ahead of a scan are cast by it, from its origin
            far = _cloud(rng, lengths[::9], res, org).astype(np.float64)
            m.add_hit_points(far)
            o.add_hit(far)
            if np.isfinite(max_range):
                assert m.update_free_cells(org.astype(np.float64)) == \
                    o.update_free_cells(org.astype(np.float64))
    gx, gc = m.dump()
    ox, oc = o.dump()
    assert np.array_equal(gx, ox) and np.array_equal(gc, oc)
    # nothing is left behind: an empty neighbourhood of the last scan stays empty
    one = org + np.array([[0.3, 0.2, 0.1]], np.float32)
    assert m.insert_point_cloud(one, org, 1.0) == o.insert(one, org, 1.0)
    assert np.array_equal(m.dump()[1], o.dump()[1])
