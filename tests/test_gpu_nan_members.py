"""Obstacle points whose x or y is NaN (their height is not): they cluster together, in the voxel at the origin, but
take no place in a hull. Hulls of clusters with few, many and only such members on both hull paths (a warp or a
CTA per cluster); every other cluster keeps its hull and boxes."""
import numpy as np
import pytest

import lp_testlib as T

lp = T.lp
pytestmark = pytest.mark.gpu


def scene(finite, nan, seed):
    """A ray-cast scan with a thing straight below the sensor, `finite` points of it and `nan` with an unknown x or y, one
    to an image row; the rest of the scan keeps clear of the first columns."""
    rng = np.random.default_rng(seed)
    x, ring, cfg = T.synth_scan(1, 3)
    cfg.image_height, cfg.min_distance_m = 256, 0.0
    away = np.arctan2(x[:, 1], x[:, 0]) % (2 * np.pi) > 0.05
    d = np.sort(rng.uniform(0.0005, 0.0035, finite))
    below = np.zeros((finite + nan, 4))
    below[:finite, 0], below[:finite, 1], below[:finite, 2] = d, d * rng.uniform(0, 0.003, finite), -0.45
    kind = rng.integers(0, 3, nan)
    below[finite:, 0] = np.where(kind != 1, np.nan, 0.0)  # (any other known coordinate gives the point a column)
    below[finite:, 1] = np.where(kind != 0, np.nan, 0.0)
    below[finite:, 2] = -0.45
    below = below.astype(np.float32)[rng.permutation(finite + nan)]
    return x[away], ring[away], below, cfg


@pytest.mark.parametrize("cta_min", [64, 512])  # above: a CTA per cluster
@pytest.mark.parametrize("finite,nan", [(0, 40), (1, 39), (2, 30), (30, 1), (30, 25), (90, 30), (20, 200)])
def test_hulls_with_nan_members(ctx, finite, nan, cta_min):
    x, ring, below, cfg = scene(finite, nan, finite + nan)
    pipe = lp.PipelineConfig.default()
    pipe.cluster.min_cluster_size = 4
    rings = np.concatenate([ring, np.arange(len(below), dtype=np.uint16)])
    cloud = np.ascontiguousarray(np.concatenate([x, below]))
    tab = lp.Tuning.default(hull_cta_min=cta_min)
    res = []
    for xs, rs in ((x, ring), (cloud, rings)):
        b = lp.PreparedBatch(ctx, [np.ascontiguousarray(xs)], pipe, [cfg], [np.ascontiguousarray(rs)], tuning=tab)
        b.execute()
        res.append(b.download()[0])
        b.close()
    want, got = res
    n = len(x)
    assert np.array_equal(got.seg_labels[:n], want.seg_labels)
    assert np.array_equal(got.cluster_labels[:n], want.cluster_labels)
    K = want.n_clusters
    assert got.n_clusters == K + 1 and (got.cluster_labels[n:] == K).all()
    at = want.hull_offsets[K]
    assert np.array_equal(got.hull_offsets[:K + 1], want.hull_offsets[:K + 1])
    assert np.array_equal(got.hull_indices[:at], want.hull_indices[:at])
    for k in range(K):
        assert T.boxes_identical(got.obb_calipers[k], want.obb_calipers[k])
        assert T.pca_boxes_equal(got.obb_pca[k], want.obb_pca[k])
    place = np.flatnonzero(~np.isnan(below[:, :2]).any(1))
    xy = below[place, :2].astype(np.float64)
    hull = T.o_hull(xy) if len(place) > 2 else np.argsort(xy[:, 0])
    assert np.array_equal(got.hull_indices[at:got.hull_offsets[K + 1]], place[hull])
