"""Points whose height is NaN (invalid returns) pass the polar grid's comparisons. Polar cells that hold nothing else,
few and many of them in one azimuth slice, with up to and more than 256 points each, leave every label as the
oracle gives it, on both ways the cells' heights are taken (one bucket table per slice, or a warp per cell)."""
import numpy as np
import pytest

import lidar_gb300 as lp
import lp_testlib as T

pytestmark = pytest.mark.gpu

# (slice, radial bin, points) of the cells that hold NaN heights only
FEW = [(10, 12, 5)]
SLICE = [(40, r, n) for r, n in ((1, 3), (3, 40), (5, 256), (7, 257), (12, 300), (13, 9), (20, 700), (31, 64))]
MANY = SLICE + [(s, 6 + s % 9, 1 + 37 * (s % 8)) for s in range(50, 350, 3)]


@pytest.mark.parametrize("spacing", [2.0, 0.5])  # 50 x 15 and 200 x 15 buckets in a slice (the table holds 2,048)
@pytest.mark.parametrize("cells", [FEW, SLICE, MANY], ids=["few", "slice", "many"])
def test_cells_of_nan_heights(ctx, cells, spacing):
    x, ring, cfg = T.synth_scan(1, 3)
    cfg.grid_radial_spacing_m = spacing
    step = np.radians(cfg.grid_slice_resolution_deg)
    rng = np.random.default_rng(len(cells))
    az, d = np.arctan2(x[:, 1], x[:, 0]) % (2 * np.pi), np.hypot(x[:, 0], x[:, 1])
    keep, bad = np.ones(len(x), bool), []
    for s, r, n in cells:
        lo, hi = max(r * spacing, cfg.min_distance_m), (r + 1) * spacing
        if lo >= hi:
            continue
        keep &= ~((np.abs(az / step - (s + 0.5)) < 0.6) & (d > lo - 0.1) & (d < hi + 0.1))
        a, q = (s + rng.uniform(0.1, 0.9, n)) * step, rng.uniform(lo + 0.1 * (hi - lo), hi - 0.1 * (hi - lo), n)
        bad.append(np.stack([q * np.cos(a), q * np.sin(a), np.full(n, np.nan), np.zeros(n)], 1))
    bad = np.concatenate(bad).astype(np.float32)
    x = np.ascontiguousarray(np.concatenate([x[keep], bad]))
    ring = np.concatenate([ring[keep], rng.integers(0, cfg.image_height, len(bad)).astype(np.uint16)])
    order = rng.permutation(len(x))
    x, ring = np.ascontiguousarray(x[order]), np.ascontiguousarray(ring[order])
    want = T.o_segment(x, ring, cfg)
    for _ in range(10):
        assert np.array_equal(lp.Segmenter(ctx, cfg).segment(x, ring), want)
