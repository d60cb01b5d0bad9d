"""The jump-convolution vote at the edges of its dispatch: images narrower than the 5 x 5 window (every
pixel a border pixel), queues that fit one thread per pixel, need rounds over the list, and outgrow the
shared-memory states; equal weights (ties everywhere), no open neighbour, no queued pixel at all; batches
on both cluster sizes. Labels and the colour image equal the oracle's."""
import numpy as np
import pytest

import lidar_gb300 as lp
import lp_testlib as T

pytestmark = pytest.mark.gpu


def scan(H, W, fill, seed, obstacles=0.5):
    """One point per range-image pixel (a share `fill` of them), ground or 1.7 m above it at random."""
    rng = np.random.default_rng(seed)
    ring, col = np.nonzero(rng.random((H, W)) < fill)
    n = len(ring)
    az = (col + 0.5) * (2 * np.pi / max(W - 1, 1)) if W > 1 else rng.uniform(0, 2 * np.pi, n)
    r = 6.0 + 0.05 * ring + rng.uniform(0, 0.3, n)
    high = rng.random(n) < obstacles
    z = np.where(high, 0.0, -1.73) + rng.normal(0, 0.01, n)
    x = np.stack([r * np.cos(az), r * np.sin(az), z, rng.random(n)], 1).astype(np.float32)
    cfg = lp.SegmenterConfig.default(image_height=H, image_width=W)
    return np.ascontiguousarray(x), ring.astype(np.uint16), cfg


def check(ctx, x, ring, cfg):
    seg = lp.Segmenter(ctx, cfg)
    got = seg.segment(x, ring, want_image=True)
    want, img = T.o_segment(x, ring, cfg, image=True)
    assert np.array_equal(got, want)
    assert np.array_equal(seg.image(), img)


@pytest.mark.parametrize("H,W", [(1, 1), (1, 7), (2, 3), (3, 2), (4, 4), (5, 5), (6, 33), (64, 1), (64, 4), (16, 129)])
def test_narrow_images(ctx, H, W):
    for seed in range(4):
        check(ctx, *scan(H, W, 0.9, seed))


@pytest.mark.parametrize("H,W,fill,obstacles", [(32, 512, 1.0, 0.05), (64, 1024, 0.9, 0.1), (64, 4096, 1.0, 0.3),
                                                (128, 2048, 1.0, 0.02), (16, 2048, 1.0, 0.0), (16, 2048, 1.0, 1.0)])
@pytest.mark.parametrize("amp,reach", [(5.0, 1.0), (0.0, 1.0), (0.5, 30.0), (400.0, 1.0)])
def test_queue_sizes(ctx, H, W, fill, obstacles, amp, reach):
    x, ring, cfg = scan(H, W, fill, H + W, obstacles)
    cfg.amplification_factor = amp
    cfg.kernel_threshold_distance_m = reach
    check(ctx, x, ring, cfg)


@pytest.mark.parametrize("nscans", [1, 7, 8, 15])
def test_batches_on_both_cluster_sizes(ctx, nscans):
    scans = [scan(8 + 5 * k, 200 + 31 * k, 0.7, k, 0.1) for k in range(nscans)]
    pipe = lp.PipelineConfig.default()
    got = lp.process_batch(ctx, [s[0] for s in scans], pipe, [s[2] for s in scans], [s[1] for s in scans])
    for r, (x, ring, cfg) in zip(got, scans):
        assert np.array_equal(r.seg_labels, T.o_segment(x, ring, cfg))


def stripes(H, W, kind, seed=1):
    """Flat ground on whose returns every n-th pixel of a row, a column or a diagonal stands 0.6 m above it: nearly
    every ground pixel is queued and hangs on its left and upper neighbours, in chains as long as the image."""
    h, w = np.meshgrid(np.arange(H), np.arange(W), indexing="ij")
    el, az = np.radians(2.0 - 26.8 * (h + 0.5) / H), (w + 0.5) * 2 * np.pi / W
    seen = el < -0.03
    r = 1.73 / np.tan(np.where(seen, -el, 1.0))
    high = {"rows": h % 4 == 0, "columns": w % 4 == 0, "diagonals": (w + 2 * h) % 5 == 0,
            "noise": np.random.default_rng(seed).random((H, W)) < 0.15}[kind]
    x = np.stack([r * np.cos(az), r * np.sin(az), np.where(high, -1.13, -1.73), 0 * r], -1)[seen].astype(np.float32)
    cfg = lp.SegmenterConfig.default(image_height=H, image_width=W)
    return np.ascontiguousarray(x), np.ascontiguousarray(h[seen].astype(np.uint16)), cfg


@pytest.mark.parametrize("H,W", [(24, 900), (64, 300), (64, 2048), (128, 4096), (20, 20000), (2000, 64)])
@pytest.mark.parametrize("kind", ["rows", "columns", "diagonals", "noise"])
def test_long_chains(ctx, H, W, kind):
    check(ctx, *stripes(H, W, kind))


def test_long_chains_of_many_scans(ctx):
    scans = [stripes(16 + 5 * k, 700 + 131 * k, kind, k) for k, kind in enumerate(["rows", "columns", "diagonals", "noise"] * 3)]
    pipe = lp.PipelineConfig.default()
    got = lp.process_batch(ctx, [s[0] for s in scans], pipe, [s[2] for s in scans], [s[1] for s in scans])
    for r, (x, ring, cfg) in zip(got, scans):
        assert np.array_equal(r.seg_labels, T.o_segment(x, ring, cfg))
