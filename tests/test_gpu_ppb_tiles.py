"""The beam gather's tile shapes: the launch picks 32, 16, 8, 4 or 2 pixels a
tile from the crop's size, and a pixel's sum is the same float whichever it
was (the order of its contributions is the leaf order)."""
import numpy as np
import pytest

import vcr
from oracle import oracle as orc
from vcr import configs

pytestmark = pytest.mark.gpu

SIZE = (40, 33, 48)


def _context(W, H, cam=None):
    desc = vcr.grid_desc(SIZE, (1 / 48,) * 3)
    cloud = vcr.cloud_from_grid(desc, 1.0, 16.0)
    dense = orc.fbm_fill(SIZE, seed=4, octaves=4)
    g = orc.Grid(dense, 0)
    cloud.max_extinction = max(g.max_density(), 0.01)
    prm = configs.C3_PPB.params(vcr.TRACKER_DDA)
    cam = cam or configs.C3_PPB.camera(W, H)
    ctx = vcr.Context()
    ctx.grid_upload(desc, dense)
    ctx.set_cloud(cloud)
    ctx.set_camera(cam)
    ctx.set_params(prm)
    ctx.set_frame(W, H)
    return ctx, g, cloud, cam, prm


# frames whose whole pass takes 32, 16, 8 and 4 pixels a tile on 152 SMs, with ragged tiles at both edges
@pytest.mark.parametrize("W,H", [(1283, 421), (601, 403), (403, 301), (265, 251)])
def test_a_frame_equals_its_crops_and_the_oracle(cuda, W, H):
    photons, cap, r0 = 150, 1 << 16, 0.04
    ctx, g, cloud, cam, prm = _context(W, H)
    with ctx:
        ctx.ppb_setup(photons, cap, r0, 0.8)
        ctx.ppb_pass(seed=3, pass_index=1)
        whole = ctx.image_sum()
        for crop in ((W // 2 - 9, H // 2 - 7, 19, 13), (W - 5, H - 3, 5, 3), (0, H // 3, 1, 1)):
            ctx.reset()
            ctx.ppb_pass(seed=3, pass_index=1, crop=crop)
            part = ctx.image_sum()
            x0, y0, cw, ch = crop
            np.testing.assert_array_equal(part[y0:y0 + ch, x0:x0 + cw], whole[y0:y0 + ch, x0:x0 + cw])
    crop = (W // 2 - 9, H // 2 - 7, 19, 13)
    o_sum, _ = orc.ppb_pass(g, cloud, cam, prm, photons, cap, r0, 0.8, W, H, seed=3, pass_index=1, crop=crop)
    x0, y0, cw, ch = crop
    np.testing.assert_array_equal(whole[y0:y0 + ch, x0:x0 + cw], o_sum[y0:y0 + ch, x0:x0 + cw])


# cameras for which the tile's pixel ranges need their margins: inside the cloud, far away with a narrow frame,
# looking along a face
@pytest.mark.parametrize("pos,fwd", [((0.02, 0.0, 0.45), (0.3, 0.1, 1.0)), ((0.0, 0.0, -30.0), (0.0, 0.0, 1.0)),
                                     ((-0.5, 0.0, -0.4), (0.05, 0.0, 1.0)), ((0.0, 1.2, 0.5), (0.0, -1.0, 0.0))])
def test_camera_poses_match_the_oracle(cuda, pos, fwd):
    W, H = 48, 41
    cam = vcr.camera_look(pos, fwd, 60.0, 0.1, W, H)
    if pos[2] == -30.0:  # a frame of the cloud alone
        cam.pixel_size_x *= 0.035
        cam.pixel_size_y *= 0.035
    ctx, g, cloud, cam, prm = _context(W, H, cam)
    with ctx:
        ctx.ppb_setup(300, 1 << 16, 0.05, 0.8)
        ctx.ppb_pass(seed=5, pass_index=0)
        got = ctx.image_sum()
    want, _ = orc.ppb_pass(g, cloud, cam, prm, 300, 1 << 16, 0.05, 0.8, W, H, seed=5, pass_index=0)
    np.testing.assert_array_equal(got, want)
    assert (want > 0.0).any()


# the pixels of a segment's own range: the sun along the view (rays nearly parallel to the beams), across it along an
# axis (segment ends on planes of rays), thin and thick beams, every tile shape's rounding far off the axis
@pytest.mark.parametrize("radius", [0.004, 0.11])
@pytest.mark.parametrize("sun", [(0.0, 0.0, 1.0), (0.0, -1.0, 0.0), (1.0, 0.0, 0.0), (0.6, 0.0, 0.8)])
def test_segment_ranges_match_the_oracle(cuda, sun, radius):
    W, H = 71, 43
    cam = vcr.camera_look((0.0, 0.0, -0.4), (0.0, 0.0, 1.0), 100.0, 0.1, W, H)
    ctx, g, cloud, cam, prm = _context(W, H, cam)
    for i in range(3):
        prm.sun_dir[i] = sun[i]
    with ctx:
        ctx.set_params(prm)
        ctx.ppb_setup(300, 1 << 17, radius, 0.8)
        ctx.ppb_pass(seed=8, pass_index=0)
        got = ctx.image_sum()
        for crop in ((3, 2, 8, 4), (W - 9, H - 6, 9, 6)):  # other tile shapes, other tile corners
            ctx.reset()
            ctx.ppb_pass(seed=8, pass_index=0, crop=crop)
            x0, y0, cw, ch = crop
            np.testing.assert_array_equal(ctx.image_sum()[y0:y0 + ch, x0:x0 + cw], got[y0:y0 + ch, x0:x0 + cw])
    want, _ = orc.ppb_pass(g, cloud, cam, prm, 300, 1 << 17, radius, 0.8, W, H, seed=8, pass_index=0)
    np.testing.assert_array_equal(got, want)
    assert (want > 0.0).any()


# photons a warp: 1 up to 20 warps an SM of 152, then 2 .. 32; a ragged last warp
@pytest.mark.parametrize("photons", [3040, 3041, 6083, 48643])
def test_emission_matches_the_oracle_at_every_share_of_a_warp(cuda, photons):
    W, H, cap = 24, 17, 1 << 14
    ctx, g, cloud, cam, prm = _context(W, H)
    prm.max_events = 3
    with ctx:
        ctx.set_params(prm)
        ctx.ppb_setup(photons, cap, 0.5, 0.8)
        ctx.ppb_pass(seed=6, pass_index=0, crop=(W // 2, H // 2, 2, 2))
        info = ctx.ppb_info()
        nbeams = ctx.ppb_read("nbeams", photons)
        slots = ctx.ppb_read("slots", photons)
    _, ob = orc.ppb_pass(g, cloud, cam, prm, photons, cap, 0.5, 0.8, W, H, seed=6, pass_index=0,
                         crop=(W // 2, H // 2, 2, 2))
    assert info["segments"] == ob["info"]["segments"] and info["dropped"] == ob["info"]["dropped"]
    np.testing.assert_array_equal(nbeams, ob["nbeams"])
    k = slots.size // (photons * 28)
    mine, want = slots.reshape(photons, k, 28), ob["slots"].reshape(photons, -1, 28)
    for b in range(k):
        has = nbeams > b
        np.testing.assert_array_equal(mine[has, b], want[has, b])
