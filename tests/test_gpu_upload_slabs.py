"""Uploads from host memory at the sizes where the slabs change: one slab,
a last slab of one layer, a ring that is used again, and one layer of more
than a kept ring's third; bricks, the four majorant levels and the maximum
against the oracle, bit for bit."""
import numpy as np
import pytest

import vcr
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

# 8 MB of brick layers (8 planes of FP32) a slab, three slabs
SIZES = [(9, 8, 7),        # one slab, one ragged layer
         (256, 256, 72),   # 4 + 4 + 1 layers
         (512, 256, 61),   # 2 layers a slab, four slabs: the first one's room is used again
         (1024, 768, 20)]  # a layer is 25 MB: the ring is the call's own


def _check(ctx, size, prec, seed):
    rng = np.random.default_rng(seed)
    dense = rng.random(size[::-1], dtype=np.float32)
    dense[rng.random(size[::-1]) < 0.3] = 0.0
    ctx.grid_upload(vcr.grid_desc(size, (1.0 / max(size),) * 3), dense, prec)
    og = orc.Grid(dense, prec)
    np.testing.assert_array_equal(ctx.grid_read_dense(), og.decoded())
    for level in range(4):
        np.testing.assert_array_equal(ctx.majorants(level), og.majorants(level), err_msg=f"level {level}")


@pytest.mark.parametrize("prec", [vcr.PREC_FP32, vcr.PREC_FP16, vcr.PREC_BF16])
def test_upload_is_the_oracles_grid(cuda, prec):
    with vcr.Context() as ctx:  # one context: streams, events and ring are used again
        for k, size in enumerate(SIZES + SIZES[:1]):
            _check(ctx, size, prec, k)


def test_refused_grid_leaves_the_next_upload_alone(cuda):
    dense = np.ones((40, 256, 256), np.float32)
    dense[39, 255, 255] = np.inf
    with vcr.Context() as ctx:
        with pytest.raises(vcr.VcrError):
            ctx.grid_upload(vcr.grid_desc((256, 256, 40), (1 / 256,) * 3), dense, vcr.PREC_FP32)
        _check(ctx, (256, 256, 40), vcr.PREC_FP32, 9)
