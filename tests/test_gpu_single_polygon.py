"""lp_convex_hull and the single-polygon boxes at the edges of their dispatch: below and above the
filter's and the shared-memory sort's sizes, binary32 and genuine binary64 coordinates, clouds that keep
every point, ties, degenerate and far-off clouds. Index sequences and boxes equal the oracle's (the
boxes' FP64 expressions are the oracle's, so no tolerance)."""
import ctypes

import numpy as np
import pytest

import lidar_gb300 as lp
import lp_testlib as T

pytestmark = pytest.mark.gpu


def cloud(kind, n, rng):
    if kind == "footprint":  # two sides of a rectangle, centimetre noise, 20 m away
        t, far = rng.random(n), rng.random(n) < 0.6
        p = np.stack([np.where(far, 8 * t, 0), np.where(far, 0, 3 * t)], 1) + rng.normal(0, 0.02, (n, 2))
        c, s = np.cos(0.4), np.sin(0.4)
        return (p @ np.array([[c, s], [-s, c]]) + 20).astype(np.float32).astype(np.float64)
    if kind == "binary64":
        return rng.normal(size=(n, 2)) * [9.0, 0.3] + [1e4, -3e3]
    if kind == "circle":  # every point a vertex: nothing can be dropped
        a = rng.permutation(n) * (2 * np.pi / n)
        return np.stack([np.cos(a), np.sin(a)], 1) * 50.0
    if kind == "grid":  # ties and collinear runs
        return np.round(rng.normal(size=(n, 2)) * 3.0)
    if kind == "line":
        return np.stack([np.arange(n) * 0.25, np.arange(n) * 0.5], 1)[rng.permutation(n)]
    if kind == "tiny":  # float products would underflow: the filter steps aside
        return rng.normal(size=(n, 2)) * 1e-14
    raise ValueError(kind)


@pytest.mark.parametrize("kind", ["footprint", "binary64", "circle", "grid", "line", "tiny"])
@pytest.mark.parametrize("n", [3, 64, 65, 511, 513, 1023, 5000, 20011])
def test_hull_sizes(ctx, kind, n):
    pts = np.ascontiguousarray(cloud(kind, n, np.random.default_rng([n, len(kind)])))
    # the device orders by exact (x, y) where the reference takes x less than DBL_EPSILON apart as equal;
    # scaled by a power of two (exact) the tiny cloud has no such x and the oracle's order is the exact one
    want = T.o_hull(pts * 2.0**50 if kind == "tiny" else pts, T.TIES_LIBSTDCXX)
    assert np.array_equal(lp.Polygonizer(ctx).convexHull(pts), want)


@pytest.mark.parametrize("n", [3, 31, 33, 1024, 1025])
@pytest.mark.parametrize("single", [True, False])
def test_boxes_sizes(ctx, n, single):
    a = np.arange(n) * (2 * np.pi / n)
    hp = np.stack([30 + 12 * np.cos(a), 5 * np.sin(a) - 8], 1)
    hp = np.ascontiguousarray(hp.astype(np.float32).astype(np.float64) if single else hp)
    poly = lp.Polygonizer(ctx)
    assert np.array_equal(poly.findAntipodalPairsOfConvexHull(hp), T.o_antipodal(hp))
    assert T.boxes_identical(poly.boundingBoxRotatingCalipers(hp), T.o_calipers(hp))
    assert T.pca_boxes_equal(poly.boundingBoxPrincipalComponentAnalysis(hp), T.o_pca(hp)[0])


def parallel_sided(kind, rng):
    """Polygons whose opposite sides are parallel up to binary32 rounding: the pair walk's area comparisons are ties."""
    c, s = np.cos(a := rng.uniform(0, 2 * np.pi)), np.sin(a)
    if kind in ("rectangle", "parallelogram"):
        w, h, k = rng.uniform(0.2, 12), rng.uniform(0.2, 4), rng.uniform(-1, 1) if kind == "parallelogram" else 0.0
        p = np.array([[0, 0], [w, 0], [w + k, h], [k, h]])
    elif kind == "regular":
        n = 2 * rng.integers(2, 17)
        p = rng.uniform(0.1, 30) * np.stack([np.cos(t := np.arange(n) * (2 * np.pi / n)), np.sin(t)], 1)
    else:  # the hull of points along a rectangle's sides
        t, w, h = rng.random((200, 2)), rng.uniform(1, 6), rng.uniform(1, 3)
        side = rng.integers(0, 2, 200)
        p = np.stack([np.where(side == 0, t[:, 0] * w, (t[:, 1] < 0.5) * w), np.where(side == 1, t[:, 0] * h, (t[:, 1] < 0.5) * h)], 1)
    p = p @ np.array([[c, s], [-s, c]]) + rng.uniform(-1, 1, 2) * rng.choice([0.0, 1.0, 60.0])
    p = np.ascontiguousarray(p.astype(np.float32).astype(np.float64))
    return np.ascontiguousarray(p[T.o_hull(p)]) if kind == "footprint" else p


@pytest.mark.parametrize("kind", ["rectangle", "parallelogram", "regular", "footprint"])
def test_boxes_of_parallel_sides(ctx, kind):
    rng = np.random.default_rng(len(kind))
    poly = lp.Polygonizer(ctx)
    for k in range(1000):
        hp = parallel_sided(kind, rng)
        if len(hp) < 3:
            continue
        assert np.array_equal(poly.findAntipodalPairsOfConvexHull(hp), T.o_antipodal(hp)), (k, hp)
        assert T.boxes_identical(poly.boundingBoxRotatingCalipers(hp), T.o_calipers(hp)), (k, hp)


def test_box_of_a_turned_rectangle(ctx):
    hp = np.array([[3.01463151, -2.00201011], [3.29160833, -2.88407683], [11.3488865, -0.354019314], [11.071909, 0.528047264]],
                  np.float32).astype(np.float64)
    poly = lp.Polygonizer(ctx)
    assert np.array_equal(poly.findAntipodalPairsOfConvexHull(hp), T.o_antipodal(hp))
    assert T.boxes_identical(poly.boundingBoxRotatingCalipers(hp), T.o_calipers(hp))


def far_points(n, scale, rng):
    """Binary32 points on an integer grid scaled by a power of two: the products of their differences leave binary32."""
    if n == 3:
        return np.array([[0.0, 0.0], [1.0, 1.0], [2.0, 3.0]]) * scale
    return np.round(rng.normal(size=(n, 2)) * 12).clip(-30, 30) * scale


@pytest.mark.parametrize("log2", [59, 62, 65, 100, 122])
@pytest.mark.parametrize("n", [3, 40, 64, 700, 5000])
def test_hull_of_far_points(ctx, n, log2):
    pts = np.ascontiguousarray(far_points(n, 2.0**log2, np.random.default_rng([n, log2])))
    assert np.array_equal(pts, pts.astype(np.float32))
    assert np.array_equal(lp.Polygonizer(ctx).convexHull(pts), T.o_hull(pts, T.TIES_LIBSTDCXX))


@pytest.mark.parametrize("log2", [65, 100])
def test_noalloc_hull_of_far_points(ctx, log2):
    torch = pytest.importorskip("torch")
    fn = lp.library().lp_convex_hull_noalloc
    fn.restype, fn.argtypes = ctypes.c_int32, [ctypes.c_void_p, ctypes.c_uint32] + [ctypes.c_void_p] * 3
    for n in (3, 40, 700):
        pts = np.ascontiguousarray(far_points(n, 2.0**log2, np.random.default_rng([n, log2])))
        xy, idx, cnt = torch.from_numpy(pts).cuda(), torch.zeros(n, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
        assert fn(xy.data_ptr(), n, idx.data_ptr(), cnt.data_ptr(), None) == lp.LP_OK
        assert np.array_equal(idx.cpu().numpy()[:int(cnt.item())], T.o_hull(pts, T.TIES_LIBSTDCXX))


@pytest.mark.parametrize("n", [3, 64, 700])
@pytest.mark.parametrize("value", [np.nan, np.inf, 1e200])
def test_hull_without_orientations(ctx, n, value):
    """NaN, infinite and overflowing coordinates: no more indices than the output holds, each of a point."""
    pts = np.random.default_rng(n).normal(size=(n, 2)) * 5
    for share in (0.1, 1.0):
        bad = np.random.default_rng([n, 1]).random((n, 2)) < share
        hull = lp.Polygonizer(ctx).convexHull(np.where(bad, value * np.sign(pts), pts))
        assert len(hull) <= n + 1 and (hull >= 0).all() and (hull < n).all()
