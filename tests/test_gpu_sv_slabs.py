"""Shadow volumes of one slab, a part of one and several, with column counts
that are no multiple of a CTA's 32: bit-exact against the oracle's march."""
import numpy as np
import pytest

import vcr
from oracle import oracle as orc
from vcr import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 31, 64, 65, 129])
def test_shadow_volume_sizes(cuda, n):
    size = (24, 40, 32)
    dense = orc.fbm_fill(size, seed=8, octaves=4)
    og = orc.Grid(dense, 0)
    desc = vcr.grid_desc(size, (1 / 40,) * 3)
    cloud = vcr.cloud_from_grid(desc, 1.0, 6.0)
    cloud.max_extinction = max(og.max_density(), 0.01)
    sv = vcr.shadow_volume_setup(configs.sun_travel_dir(35.0, 120.0), cloud.bounds_min, cloud.bounds_max, n)
    with vcr.Context() as ctx:
        ctx.grid_upload(desc, dense)
        ctx.set_cloud(cloud)
        ctx.shadow_volume_build(sv)
        ctx.synchronize()
        got = ctx.shadow_volume(n)
    np.testing.assert_array_equal(got, og.sv_build(cloud, sv))
