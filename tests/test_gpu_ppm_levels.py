"""The photon gather's way back up its levels: spheres that meet more than
four boxes of a level, so that the others wait while the first four are
opened, on three levels and more."""
import numpy as np
import pytest

import vcr
from oracle import oracle as orc
from oracle import oracle_ppm as opm
from vcr import configs

pytestmark = pytest.mark.gpu

SIZE = (32, 32, 32)


@pytest.mark.parametrize("photons,radius", [(3500, 0.5), (3500, 0.15), (700, 2.0)])
def test_levels_taken_up_again_match_the_oracle(cuda, photons, radius):
    dense = orc.fbm_fill(SIZE, seed=5, octaves=4)
    g = orc.Grid(dense, 0)
    desc = vcr.grid_desc(SIZE, (1 / 32,) * 3)
    cloud = vcr.cloud_from_grid(desc, 1.0, 24.0)
    cloud.max_extinction = max(g.max_density(), 0.01)
    W, H = 41, 23
    cam, prm = configs.C2_PPM.camera(W, H), configs.C2_PPM.params(vcr.TRACKER_DDA)
    st = opm.init_stats(W, H, radius)
    with vcr.Context() as ctx:
        ctx.grid_upload(desc, dense)
        ctx.set_cloud(cloud)
        ctx.set_camera(cam)
        ctx.set_params(prm)
        ctx.set_frame(W, H)
        ctx.ppm_setup(photons, 1 << 17, radius, 0.8)
        ctx.ppm_pass(seed=7, pass_index=0)
        n, levels = ctx.ppm_info()["photons_stored"], 0
        while n > 8:  # boxes of 8 up to a level of at most 8
            n, levels = -(-n // 8), levels + 1
        assert levels >= 3
        want, _ = opm.ppm_pass(g, cloud, cam, prm, photons, 1 << 17, 0.8, W, H, st, seed=7, pass_index=0)
        np.testing.assert_array_equal(ctx.ppm_read("stats"), st)
        np.testing.assert_array_equal(ctx.image_sum(), want)
        if radius == 2.0:  # every sphere holds the whole map, and so opens every box
            stored = ctx.ppm_info()["photons_stored"]
            assert ctx.gather_stats("ppm")[0] == stored * int((st[..., 0] > 0).sum())
