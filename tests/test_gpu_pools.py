"""The path tracer's warp pools: launches of one path to many per warp give
each pixel the oracle's sum, and the logarithm's division is the rounded one
for every operand it can meet."""
import os
import subprocess

import numpy as np
import pytest

import vcr
from oracle import oracle as orc
from vcr import configs

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "cloudrendering-vulkan_gb300", "csrc")


def test_vlog_division_is_rounded_for_every_mantissa(cuda, tmp_path):
    exe = str(tmp_path / "vlog_all")
    subprocess.run([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-gencode", "arch=compute_103a,code=sm_103a",
                    "-O3", "-std=c++17", "-fmad=false", "-I", CSRC, "-o", exe,
                    os.path.join(HERE, "cpp", "vlog_all.cu")], check=True, capture_output=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    assert int(out) == 0


# one path a warp, a few, a pool's worth and several pools' worth; one pixel and one row; both CTA sizes and a
# level too large to stage beside the pools
@pytest.mark.parametrize("W,H,spp,threads,level", [(2, 2, 1, 256, 1), (61, 59, 1, 128, 2), (301, 2, 1, 256, 0),
                                                   (233, 177, 1, 256, 1), (401, 307, 2, 128, 0),
                                                   (640, 361, 2, 256, 2)])
def test_pool_sizes_match_the_oracle(cuda, W, H, spp, threads, level):
    size = (140, 70, 150)  # level 0: 18 x 9 x 19 cells, 12 KB
    dense = orc.fbm_fill(size, seed=6, octaves=4)
    g = orc.Grid(dense, 0)
    desc = vcr.grid_desc(size, (1 / 150,) * 3)
    cloud = vcr.cloud_from_grid(desc, 1.0, 20.0)
    cloud.max_extinction = max(g.max_density(), 0.01)
    cam, prm = configs.C1_PT.camera(W, H), configs.C1_PT.params(vcr.TRACKER_DDA)
    with vcr.Context() as ctx:
        ctx.set_tuning(majorant_level=level, dda_steps=3, block_threads=threads)
        ctx.grid_upload(desc, dense)
        ctx.set_cloud(cloud)
        ctx.set_camera(cam)
        ctx.set_params(prm)
        ctx.set_frame(W, H)
        ctx.pt_pass(seed=9, pass_index=2, spp=spp)
        got, counters = ctx.image_sum(), ctx.counters()
    og, stats = g.pt_pass(cloud, cam, prm, W, H, seed=9, pass_index=2, spp=spp, level=level,
                          flags=vcr.PASS_RECORD_STATS)
    if spp == 1:
        np.testing.assert_array_equal(got, og)
        assert counters[0] == W * H and counters[2] == int(stats[..., 0].sum())
        assert counters[1] == int(stats[..., 1].sum()) and counters[3] == int(stats[..., 3].sum())
    else:  # float64 sums of a pixel's samples in another order
        np.testing.assert_allclose(got, og, rtol=1e-12, atol=0)
        assert counters[0] == W * H * spp
