"""Beams through grids with texels below zero (a filtered cloud's undershoot)
or without a number: their majorants are zero at least and bound no lookup
there, so the gather may leave no segment and no part of a ray out."""
import numpy as np
import pytest

import vcr
from oracle import oracle as orc
from vcr import configs

pytestmark = pytest.mark.gpu

SIZE = (40, 33, 48)


def _grid(kind):
    dense = orc.fbm_fill(SIZE, seed=4, octaves=4)
    rng = np.random.default_rng(1)
    if kind == "undershoot":
        dense[dense == 0.0] = -0.01
    elif kind == "hollow":  # nothing but texels below zero in half of the grid
        dense[:, :, :32] = 0.0
        dense[12:36, 8:24, 4:24] = -2.0
    else:
        dense.reshape(-1)[rng.integers(0, dense.size, 40)] = np.nan
    return dense


@pytest.mark.parametrize("precision", [vcr.PREC_FP32, vcr.PREC_FP16])
@pytest.mark.parametrize("kind", ["undershoot", "hollow", "no number"])
def test_image_is_the_oracles(cuda, kind, precision):
    W, H, photons, cap, radius = 64, 43, 300, 1 << 16, 0.05
    dense = _grid(kind)
    g = orc.Grid(dense, precision)
    desc = vcr.grid_desc(SIZE, (1 / 48,) * 3)
    cloud = vcr.cloud_from_grid(desc, 1.0, 16.0)
    cloud.max_extinction = max(g.max_density(), 0.01)
    cam, prm = configs.C3_PPB.camera(W, H), configs.C3_PPB.params(vcr.TRACKER_DDA)
    with vcr.Context() as ctx:
        ctx.grid_upload(desc, dense, precision)
        ctx.set_cloud(cloud)
        ctx.set_camera(cam)
        ctx.set_params(prm)
        ctx.set_frame(W, H)
        ctx.ppb_setup(photons, cap, radius, 0.8)
        images = []
        for _ in range(2):
            ctx.reset()
            ctx.ppb_pass(seed=5, pass_index=0)
            images.append(ctx.image_sum())
            # the next grid has none of them, and is gathered as before
            plain = np.maximum(np.nan_to_num(dense), 0.0)
            if len(images) == 1:
                ctx.grid_upload(desc, plain, precision)
    for got, grid in ((images[0], g), (images[1], orc.Grid(plain, precision))):
        want, _ = orc.ppb_pass(grid, cloud, cam, prm, photons, cap, radius, 0.8, W, H, seed=5, pass_index=0)
        np.testing.assert_array_equal(got, want)
    assert precision != vcr.PREC_FP32 or not np.array_equal(images[0], images[1])
