"""Segmentation of scans of few points an azimuth slice (a warp per slice): slices of no, one, 32, 33 and many points, heights
that tie, lie half a metre apart or are NaN, cells near the sensor, long slices; many such scans in one batch.
Labels equal the oracle's."""
import numpy as np
import pytest

import lp_testlib as T

lp = T.lp
pytestmark = pytest.mark.gpu


def scan(n, seed, spacing=2.0, resolution=1.0, nan=False):
    rng = np.random.default_rng([n, seed])
    az = rng.uniform(0, 2 * np.pi, n)
    crowd = rng.random(n) < 0.4  # crowded slices, up to some hundred points each
    az[crowd] = (rng.integers(0, 40, crowd.sum()) * 9 + rng.uniform(0.1, 0.9, crowd.sum())) * np.pi / 180
    k = np.arange(n) < 65  # one of 32 and one of 33
    az[k] = (np.where(np.arange(n)[k] < 32, 100, 203) + rng.uniform(0.2, 0.8, k.sum())) * np.pi / 180
    d = np.where(rng.random(n) < 0.4, rng.uniform(2, 8, n), rng.uniform(2, 90, n))
    z = np.where(rng.random(n) < 0.5, rng.choice([-1.73, -1.5, -1.23, -0.73, -0.5, 0.0, 0.5, 1.0], n), rng.uniform(-2.2, 1.5, n))
    if nan:  # all points of a polar cell, so that the oracle's order of heights is defined
        cell = np.floor(d / spacing).astype(int) * 1000 + np.floor(az * 180 / np.pi / resolution).astype(int)
        z = np.where(cell % 13 == 0, np.nan, z)
    x = np.stack([d * np.cos(az), d * np.sin(az), z, rng.random(n)], 1).astype(np.float32)
    cfg = lp.SegmenterConfig.default(grid_radial_spacing_m=spacing, grid_slice_resolution_deg=resolution, image_height=32,
                                     image_width=512)
    return np.ascontiguousarray(x), rng.integers(0, 32, n).astype(np.uint16), cfg


@pytest.mark.parametrize("n", [1, 2, 33, 300, 3000, 5700, 5761])  # 5,760: a CTA per slice from there on
@pytest.mark.parametrize("spacing", [0.3, 2.0, 10.0])
def test_sparse_scan(ctx, n, spacing):
    for seed in range(6):
        x, ring, cfg = scan(n, seed, spacing)
        assert np.array_equal(lp.Segmenter(ctx, cfg).segment(x, ring), T.o_segment(x, ring, cfg)), seed


@pytest.mark.parametrize("n", [300, 5700])
@pytest.mark.parametrize("resolution", [0.25, 1.0])
def test_sparse_scan_with_nan_heights(ctx, n, resolution):
    for seed in range(6):
        x, ring, cfg = scan(n, seed, 2.0, resolution, nan=True)
        # cells of the device's own slice arithmetic may hold both: the labels of those depend on the order of heights
        az = np.arctan2(x[:, 1].astype(np.float64), x[:, 0]) % (2 * np.pi) / np.radians(resolution)
        edge = np.abs(az - np.round(az)) < 0.02
        x, ring = np.ascontiguousarray(x[~edge]), np.ascontiguousarray(ring[~edge])
        assert np.array_equal(lp.Segmenter(ctx, cfg).segment(x, ring), T.o_segment(x, ring, cfg)), seed


@pytest.mark.parametrize("nscans", [9, 300])
def test_batch_of_sparse_scans(ctx, nscans):
    scans = [scan(int(5 + 37 * (k % 17)), k, [0.5, 2.0, 5.0][k % 3], [1.0, 2.0][k % 2]) for k in range(nscans)]
    pipe = lp.PipelineConfig.default()
    got = lp.process_batch(ctx, [s[0] for s in scans], pipe, [s[2] for s in scans], [s[1] for s in scans])
    for r, (x, ring, cfg) in zip(got, scans):
        assert np.array_equal(r.seg_labels, T.o_segment(x, ring, cfg))
