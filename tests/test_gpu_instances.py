"""The path tracer's instances (with and without corner blocks, staged and
unstaged majorants, both CTA sizes; passes, batches and cached passes): each
kind of launch gives one image whichever instance ran it, and the plain
pass's is the oracle's."""
import itertools

import numpy as np
import pytest

import vcr
from oracle import oracle as orc
from vcr import configs

pytestmark = pytest.mark.gpu

SIZE, W, H = (44, 37, 50), 53, 47


@pytest.mark.parametrize("precision", [vcr.PREC_FP32, vcr.PREC_FP16, vcr.PREC_BF16])
def test_every_instance_gives_the_launch_its_image(cuda, precision):
    dense = orc.fbm_fill(SIZE, seed=6, octaves=4)
    g = orc.Grid(dense, precision)
    desc = vcr.grid_desc(SIZE, (1 / 50,) * 3)
    cloud = vcr.cloud_from_grid(desc, 1.0, 20.0)
    cloud.max_extinction = max(g.max_density(), 0.01)
    cam, prm = configs.C1_PT.camera(W, H), configs.C1_PT.params(vcr.TRACKER_DDA)
    cached = configs.C1_PT.params(vcr.TRACKER_DDA)
    cached.nrc_events = 2
    views = [(cam, W, H, configs.sun_travel_dir(20.0)), (configs.C1_PT.camera(31, 29), 31, 29,
                                                        configs.sun_travel_dir(60.0))]
    first = None
    for corners, stage, threads in itertools.product((1, 0), (1, 0), (256, 128)):
        with vcr.Context() as ctx:
            ctx.set_tuning(majorant_level=1, dda_steps=3, stage_majorants=stage, block_threads=threads,
                           corner_blocks=corners)
            ctx.grid_upload(desc, dense, precision)
            ctx.set_cloud(cloud)
            ctx.set_camera(cam)
            ctx.set_params(prm)
            ctx.set_frame(W, H)
            ctx.pt_pass(seed=9, pass_index=2)
            images = [ctx.image_sum()]
            ctx.batch_setup(views)
            ctx.batch_pass(seed=11, pass_index=1)
            ctx.synchronize()
            images += [ctx.batch_read(v) for v in range(len(views))]
            ctx.set_params(cached)
            ctx.nrc_setup(train_samples=512, query_capacity=W * H, seed=2)
            ctx.reset()
            ctx.pt_pass(seed=6, pass_index=0)  # paths that end in the cache, with its initial weights
            ctx.synchronize()
            images.append(ctx.image_sum())
            queries = ctx.nrc_info()["queries"]
        if first is None:
            og, _ = g.pt_pass(cloud, cam, prm, W, H, seed=9, pass_index=2, level=1)
            np.testing.assert_array_equal(images[0], og)
            first = images, queries
            assert queries > 50
            continue
        for k in range(3):
            np.testing.assert_array_equal(images[k], first[0][k])
        # a pixel's one query adds to its one path's radiance: the same two terms in either order
        np.testing.assert_allclose(images[3], first[0][3], rtol=1e-15, atol=0)
        assert queries == first[1]
