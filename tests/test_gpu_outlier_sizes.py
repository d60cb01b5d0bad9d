"""The outlier filter about the sizes where its tree build changes hands (ranges finished by one warp, in shared memory,
by a CTA, by a cluster of CTAs) and on clouds whose searches leave much on the stack: the tree equals the
reference's node for node, the mask its sequential search's. Batches of scans of very different size."""
import numpy as np
import pytest

import lp_testlib as T

lp = T.lp
pytestmark = pytest.mark.gpu

EDGES = [16, 512, 2048, 4096, 6144, 12288, 65536]


def cloud(kind, n, seed):
    rng = np.random.default_rng([n, seed])
    if kind == "random":
        p = rng.normal(size=(n, 3)) * [20, 20, 0.5]
    elif kind == "grid":  # ties on every axis, neighbours at exactly the radius
        p = np.round(rng.uniform(-12, 12, (n, 3)) * 2) / 2
    elif kind == "sorted":  # ascending on the first axis
        p = np.sort(rng.uniform(-50, 50, (n, 3)), axis=0)
    else:  # dense things in a sparse cloud: stops and short points alternate
        p = np.where((rng.random(n) < 0.7)[:, None], rng.normal(size=(n, 3)) * 0.4 + rng.uniform(-30, 30, (16, 3))[rng.integers(0, 16, n)],
                     rng.uniform(-40, 40, (n, 3)))
    return np.ascontiguousarray(p.astype(np.float32))


@pytest.mark.parametrize("edge", EDGES)
@pytest.mark.parametrize("kind", ["random", "grid", "sorted"])
def test_tree_at_the_edges(ctx, kind, edge):
    for n in (edge - 1, edge, edge + 1, 2 * edge + 1):
        pts = cloud(kind, n, 0)
        assert np.array_equal(lp.debug_kdtree(ctx, pts)[0], T.o_kdtree_positions(pts)), n


@pytest.mark.parametrize("neighbours,radius", [(2, 0.1), (4, 0.5), (9, 1.0)])
@pytest.mark.parametrize("kind", ["random", "grid", "things"])
@pytest.mark.parametrize("n", [513, 4097, 6145, 20000, 65537])
def test_mask_at_the_edges(ctx, kind, n, neighbours, radius):
    pts = cloud(kind, n, 1)
    cfg = lp.NoiseRemoverConfig(0.02, radius, neighbours)
    assert np.array_equal(lp.NoiseRemover(ctx, cfg).filter(pts), T.o_noise(pts, cfg, T.DROR_KDTREE))


@pytest.mark.parametrize("sizes", [[70000, 5, 4097, 1, 900, 20000], [1, 1], [3, 66000], [2049] * 9])
def test_masks_of_a_mixed_batch(ctx, sizes):
    pts = [np.ascontiguousarray(np.c_[cloud("things", n, 2 + k), np.zeros(n, np.float32)]) for k, n in enumerate(sizes)]
    cfg = lp.SegmenterConfig.default(image_height=64, image_width=2048, assume_unorganized_cloud=1)
    pipe = lp.PipelineConfig.default()
    pipe.enable_noise_removal, pipe.noise = 1, lp.NoiseRemoverConfig(0.02, 0.3, 4)
    got = lp.process_batch(ctx, pts, pipe, [cfg] * len(pts), [None] * len(pts))
    for r, p in zip(got, pts):
        assert np.array_equal(r.noise_labels, T.o_noise(p, pipe.noise, T.DROR_KDTREE))
