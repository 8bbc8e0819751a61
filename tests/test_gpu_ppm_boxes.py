"""The photon gather's boxes of 8: photon counts at the edges of their levels
(1 to several thousand stored photons), radii from a few photons to all of
them, against the oracle's tree walk bit for bit."""
import numpy as np
import pytest

import vcr
from oracle import oracle as orc
from oracle import oracle_ppm as opm
from vcr import configs

pytestmark = pytest.mark.gpu

SIZE = (32, 32, 32)


@pytest.mark.parametrize("photons,radius", [(1, 0.5), (2, 0.5), (5, 0.1), (40, 2.0), (40, 0.05), (300, 0.3),
                                            (2500, 0.02), (2500, 2.0)])
def test_gather_matches_the_oracle(cuda, photons, radius):
    dense = orc.fbm_fill(SIZE, seed=3, octaves=4)
    g = orc.Grid(dense, 0)
    desc = vcr.grid_desc(SIZE, (1 / 32,) * 3)
    cloud = vcr.cloud_from_grid(desc, 1.0, 24.0)
    cloud.max_extinction = max(g.max_density(), 0.01)
    W, H = 33, 17
    cam, prm = configs.C2_PPM.camera(W, H), configs.C2_PPM.params(vcr.TRACKER_DDA)
    st = opm.init_stats(W, H, radius)
    with vcr.Context() as ctx:
        ctx.grid_upload(desc, dense)
        ctx.set_cloud(cloud)
        ctx.set_camera(cam)
        ctx.set_params(prm)
        ctx.set_frame(W, H)
        ctx.ppm_setup(photons, 1 << 17, radius, 0.8)
        for k in range(2):
            ctx.ppm_pass(seed=4, pass_index=k)
            want, o = opm.ppm_pass(g, cloud, cam, prm, photons, 1 << 17, 0.8, W, H, st, seed=4, pass_index=k)
            assert ctx.ppm_info()["photons_stored"] == o["info"]["photons_stored"]
            np.testing.assert_array_equal(ctx.ppm_read("stats"), st)
            np.testing.assert_array_equal(ctx.image_sum(), want)
            # every photon found is counted
            assert ctx.counters()[2] >= int((st[..., 0] > 0).sum())
