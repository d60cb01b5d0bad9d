"""Range-image projection with the keys in one word and, where they need more than 63 bits, in two passes: from
a least distance of zero on and with fine grids, scans small and large, points of equal distance in one
pixel. Labels equal the oracle's."""
import numpy as np
import pytest

import lp_testlib as T

lp = T.lp
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("least", [0.0, 2.0])
@pytest.mark.parametrize("slices", [2.0, 0.05])
@pytest.mark.parametrize("scan,repeat", [(8, 1), (12, 4)])
def test_projection_keys(ctx, least, slices, scan, repeat):
    x, ring, cfg = T.synth_scan(3, scan)[:3]
    cfg.min_distance_m, cfg.grid_slice_resolution_deg = least, slices
    rng = np.random.default_rng(scan)
    far = x.copy()  # the same directions farther away, and points of exactly equal distance
    far[:, :3] *= 1.25
    x = np.concatenate([x, far, x[::3]] * repeat)
    ring = np.concatenate([ring, ring, ring[::3]] * repeat)
    order = rng.permutation(len(x))
    x, ring = np.ascontiguousarray(x[order]), np.ascontiguousarray(ring[order])
    want = T.o_segment(x, ring, cfg)
    got = lp.Segmenter(ctx, cfg).segment(x, ring)
    assert np.array_equal(got, want)
