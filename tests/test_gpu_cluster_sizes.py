"""Clustering and the hull bookkeeping at the edges of their layouts: clouds around a scan tile and the
smallest hash slice, both tile sizes of the device-wide scans, batches of more scans than a warp lays out
at once with empty and obstacle-free scans among them. Labels, offsets and hulls equal the oracle's."""
import numpy as np
import pytest

import lidar_gb300 as lp
import lp_testlib as T

pytestmark = pytest.mark.gpu


def blobs(n, seed, spread=0.3):
    rng = np.random.default_rng(seed)
    k = max(1, n // 40)
    c = rng.uniform(-40, 40, (k, 3)) * [1, 1, 0.05]
    return np.ascontiguousarray((c[rng.integers(0, k, n)] + rng.normal(0, spread, (n, 3))).astype(np.float32))


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 1023, 1024, 1025, 8193, 70000, 1048575, 1048577])
def test_cluster_sizes(ctx, n):
    x = blobs(n, n) if n < 1 << 20 else blobs(n, n, spread=0.15)[:, :3]
    cfg = lp.ClustererConfig.default()
    try:
        want = T.o_cluster(x, cfg)
    except OverflowError:  # more than 200,000 occupied voxels: the reference throws
        with pytest.raises(OverflowError):
            lp.Clusterer(ctx, cfg).cluster(x)
        return
    assert np.array_equal(lp.Clusterer(ctx, cfg).cluster(x), want)


@pytest.mark.parametrize("n", [1, 1022, 1023, 1024, 5000, 1048575, 1048576])
def test_split_clouds_sizes(ctx, n):
    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, 4)).astype(np.float32)
    lab = rng.integers(0, 3, n).astype(np.uint32)
    clouds = lp.split_clouds(ctx, x, lab)
    for got, keep in zip(clouds, (lab == lp.GROUND, lab == lp.OBSTACLE, lab == lp.UNKNOWN)):
        assert np.array_equal(np.stack([got["x"], got["y"], got["z"]], 1), x[keep, :3])


def test_batch_of_many_small_scans(ctx):
    """45 scans: empty, ground only, obstacles only, mixed; concurrent parts and one launch sequence."""
    rng = np.random.default_rng(3)
    scans = []
    for k in range(45):
        n = [0, 60, 700, 3000, 1][k % 5]
        a, r = rng.uniform(0, 2 * np.pi, n), rng.uniform(4, 30, n)
        z = np.full(n, -1.73) if k % 3 == 0 else rng.choice([-1.73, 0.2], n)
        x = np.stack([r * np.cos(a), r * np.sin(a), z + rng.normal(0, 0.01, n), rng.random(n)], 1).astype(np.float32)
        scans.append((np.ascontiguousarray(x), rng.integers(0, 16, n).astype(np.uint16),
                      lp.SegmenterConfig.default(image_height=16, image_width=128)))
    pipe = lp.PipelineConfig.default()
    xs, rings, cfgs = [s[0] for s in scans], [s[1] for s in scans], [s[2] for s in scans]
    unsplit = lp.process_batch(ctx, xs, pipe, cfgs, rings)
    batch = lp.PreparedBatch(ctx, xs, pipe, cfgs, rings)
    batch.execute()
    split = batch.download()
    batch.close()
    for res in (unsplit, split):
        for r, (x, ring, cfg) in zip(res, scans):
            if len(x) == 0:
                assert r.n_clusters == 0
                continue
            want = T.o_process(x, ring, cfg, pipe)
            assert np.array_equal(r.seg_labels, want.seg_labels)
            assert np.array_equal(r.cluster_labels, want.cluster_labels)
            assert np.array_equal(r.hull_offsets, want.hull_offsets)
            assert np.array_equal(r.hull_indices, want.hull_indices)
