"""A prepared batch takes no more device memory than before the vote kept a record per open pixel: a serving loop reserves
its memory once and refuses a scan whose batch is larger, so growth would refuse scans that fitted. Sizes in bytes, of
batches of one scan, with all results, of the layout before."""
import numpy as np
import pytest

import lp_testlib as T

lp = T.lp
pytestmark = pytest.mark.gpu

# points, rows, columns, outlier filter, rings given: bytes
BEFORE = [((20000, 32, 1024, 0, 1), 16012008), ((131072, 64, 2048, 0, 1), 94567032), ((131072, 64, 2048, 0, 0), 94271832),
          ((300001, 128, 4096, 0, 1), 236800971), ((524288, 128, 4096, 0, 0), 375665400), ((60000, 64, 2048, 1, 1), 60864363)]


@pytest.mark.parametrize("shape,before", BEFORE)
def test_batch_takes_no_more_memory(ctx, shape, before):
    n, rows, columns, noise, rings = shape
    pipe = lp.PipelineConfig.default()
    pipe.enable_noise_removal = noise
    cfg = lp.SegmenterConfig.default(image_height=rows, image_width=columns)
    b = lp.PreparedBatch(ctx, [np.zeros((n, 4), np.float32)], pipe, [cfg], [np.zeros(n, np.uint16) if rings else None])
    try:
        assert b.device_bytes <= before
    finally:
        b.close()
