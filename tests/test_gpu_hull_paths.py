"""Hulls and boxes of clusters about the sizes where their path changes (one warp or a CTA, polygon refined or not,
members passed over grid-wide): straight walls (near-ties all along), noisy ones, arcs (every point a
vertex), boxes with repeated points. Equal to the oracle's, boxes included."""
import numpy as np
import pytest

import lp_testlib as T

lp = T.lp
pytestmark = pytest.mark.gpu

# (points, width in metres): cluster sizes follow from the pixels they fall into
THINGS = [(20, 0.5), (40, 1), (80, 1), (120, 1.5), (180, 2), (350, 2), (600, 3), (800, 3), (2500, 4), (60000, 11)]
CLASSES = [(1, 32), (33, 64), (65, 256), (257, 512), (513, 8192), (8193, 1 << 30)]
ROWS, COLUMNS, UP, DOWN = 128, 4096, 15.0, -25.0


def thing(kind, n, rng):
    """n points (x, y) of a thing about 4 units wide around the origin."""
    t = rng.random(n)
    if kind == "wall":
        return np.stack([4 * t - 2, 1.5 * t - 0.75], 1)
    if kind == "noisy":
        return np.stack([4 * t - 2, 1.5 * t - 0.75], 1) + rng.normal(0, 0.02, (n, 2))
    if kind == "arc":
        return np.stack([2 * np.cos(3 * t), 1.2 * np.sin(3 * t)], 1)
    if kind == "repeats":  # two sides of a box on a 5 cm grid: corners and edges many times over
        p = np.where((t < 0.6)[:, None], np.stack([5 * t - 1.5, 0 * t], 1), np.stack([0 * t + 1.5, 5 * (t - 0.6)], 1))
        return np.round(p * 20) / 20
    raise ValueError(kind)


def scene(kind):
    """Flat ground with the things standing on it, 9 m away and apart."""
    rng = np.random.default_rng(len(kind))
    r, a = rng.uniform(3, 60, 60000), rng.uniform(-np.pi, np.pi, 60000)
    parts = [np.stack([r * np.cos(a), r * np.sin(a), -1.73 + rng.normal(0, 0.01, len(r))], 1)]
    at = np.cumsum([0.0] + [0.5 * (v[1] + w[1]) + 2.5 for v, w in zip(THINGS, THINGS[1:])])
    for (n, width), s in zip(THINGS, at):
        t = s / 9 - np.pi
        xy = thing(kind, n, rng) * (width / 4) @ np.array([[-np.sin(t), np.cos(t)], [-np.cos(t), -np.sin(t)]])
        parts.append(np.concatenate([xy + 9 * np.array([np.cos(t), np.sin(t)]), rng.uniform(-1.0, 0.8, (n, 1))], 1))
    x = np.zeros((sum(map(len, parts)), 4), np.float32)
    x[:, :3] = np.concatenate(parts)
    el = np.degrees(np.arctan2(x[:, 2], np.hypot(x[:, 0], x[:, 1])))
    ring = np.clip(np.round((el - DOWN) / (UP - DOWN) * (ROWS - 1)), 0, ROWS - 1).astype(np.uint16)
    cfg = lp.SegmenterConfig.default(image_height=ROWS, image_width=COLUMNS, elevation_up_deg=UP, elevation_down_deg=DOWN)
    return x, ring, cfg


@pytest.mark.parametrize("kind", ["wall", "noisy", "arc", "repeats"])
def test_cluster_hull_paths(ctx, kind):
    x, ring, cfg = scene(kind)
    pipe = lp.PipelineConfig.default()
    want = T.o_process(x, ring, cfg, pipe)
    sizes = np.bincount(want.cluster_labels[want.cluster_labels >= 0])
    for lo, hi in CLASSES[:5] if kind == "repeats" else CLASSES:  # (few pixels see the repeats)
        assert ((sizes >= lo) & (sizes <= hi)).any(), (lo, sizes)
    got = lp.process_batch(ctx, [x], pipe, [cfg], [ring])[0]
    assert np.array_equal(got.cluster_labels, want.cluster_labels)
    assert np.array_equal(got.hull_offsets, want.hull_offsets)
    assert np.array_equal(got.hull_indices, want.hull_indices)
    for k in range(want.n_clusters):
        assert T.boxes_identical(got.obb_calipers[k], want.obb_calipers[k]), k
        assert T.pca_boxes_equal(got.obb_pca[k], want.obb_pca[k]), k


@pytest.mark.parametrize("rings,columns", [(3, 1400), (7, 1301), (6, 4096)])
def test_hull_of_more_vertices_than_shared_memory(ctx, rings, columns):
    """A wall all around the sensor: one cluster, most of its outermost points hull vertices."""
    rng = np.random.default_rng(columns)
    ring, col = np.meshgrid(np.arange(rings), np.arange(columns), indexing="ij")
    r, az = 20 - 0.02 * ring, (col + 0.5) * 2 * np.pi / columns
    x = np.stack([r * np.cos(az), r * np.sin(az), 0.5 - 0.3 * ring, 0 * r], -1).reshape(-1, 4).astype(np.float32)
    order = rng.permutation(len(x))
    x, ring = np.ascontiguousarray(x[order]), np.ascontiguousarray(ring.ravel()[order].astype(np.uint16))
    cfg = lp.SegmenterConfig.default(image_height=rings, image_width=columns)
    pipe = lp.PipelineConfig.default()
    want = T.o_process(x, ring, cfg, pipe)
    assert want.n_clusters == 1 and len(want.hull_indices) > 1024
    got = lp.process_batch(ctx, [x], pipe, [cfg], [ring])[0]
    assert np.array_equal(got.cluster_labels, want.cluster_labels)
    assert np.array_equal(got.hull_indices, want.hull_indices)
    assert T.boxes_identical(got.obb_calipers[0], want.obb_calipers[0])
    assert T.pca_boxes_equal(got.obb_pca[0], want.obb_pca[0])
