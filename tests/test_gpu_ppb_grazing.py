"""Beams that graze a column of camera rays: a beam in a plane x = const beside
the plane x = 0 of the image's middle column, with the radius the float just
below their distance.  The closest points of such a pair pass the gather's
first comparison (which has a margin) while the ray misses the segment's box,
so the pair is queued and then turned away.  The image is the oracle's at
every tile shape."""
import numpy as np
import pytest

import vcr
from oracle import oracle as orc
from vcr import configs

pytestmark = pytest.mark.gpu

SIZE = (40, 33, 48)
F = np.float32


def _dot(a, b):
    return (a[..., 0] * b[..., 0] + a[..., 1] * b[..., 1]) + a[..., 2] * b[..., 2]


def _turned_away(cam, cloud, H, a, b, lo, hi, reach):
    """Pairs of the middle column's rays and the segments (start a, end b with
    the distance from the beam's origin, box lo .. hi) that the gather queues
    and whose ray misses the box: its float operations, one by one."""
    f = lambda v: np.array(list(v), F)  # noqa: E731
    rows = np.arange(H, dtype=F) - F(cam.half_height)
    d = (f(cam.forward) * F(cam.near_plane) + (f(cam.right) * F(cam.pixel_size_x)) * F(0)) - \
        (f(cam.up) * F(cam.pixel_size_y)) * rows[:, None]
    o = (d + f(cam.position))[:, None]
    rd = (d / np.sqrt(_dot(d, d))[:, None])[:, None]
    with np.errstate(divide="ignore", invalid="ignore"):
        inv = F(1) / rd
        s0, s1 = (f(cloud.bounds_min) - o) * inv, (f(cloud.bounds_max) - o) * inv
        t_in = np.nanmax(np.minimum(s0, s1), axis=-1)
        t_out = np.nanmin(np.maximum(s0, s1), axis=-1)
        ax = b[:, :3] - a[:, :3]
        length = np.sqrt(_dot(ax, ax))
        bd = ax / length[:, None]
        c = _dot(rd, bd)
        den = F(1) - c * c
        w0 = o - a[:, :3]
        dw, ew = _dot(rd, w0), _dot(bd, w0)
        t = (c * ew - dw) / den
        sb = ew + t * c
        e = (o + t[..., None] * rd) - (a[:, :3] + sb[..., None] * bd)
        r = a[0, 3]
        queued = (den > F(1e-6)) & (t >= t_in) & (t <= t_out) & (sb >= 0) & (sb <= length) & \
            (_dot(e, e) < (r * r) * F(1.000001)) & (b[:, 3] <= reach)
        q0, q1 = (lo[:, :3] - o) * inv, (hi[:, :3] - o) * inv
        tn = np.maximum(np.nanmax(np.minimum(q0, q1), axis=-1), t_in)
        tf = np.minimum(np.nanmin(np.maximum(q0, q1), axis=-1), t_out)
    return int((queued & ~(tn <= tf)).sum())


# frames whose whole pass takes 32, 16, 8, 4 and 2 pixels a tile on 152 SMs
@pytest.mark.parametrize("sun", [(0.0, -1.0, 0.0), (0.0, -0.6, 0.8)])
@pytest.mark.parametrize("W,H", [(1283, 421), (601, 403), (403, 301), (265, 251), (61, 45)])
def test_pairs_that_miss_the_box_leave_the_image_alone(cuda, W, H, sun):
    photons, cap, seed = 150, 1 << 17, 3
    desc = vcr.grid_desc(SIZE, (1 / 48,) * 3)
    # thin, so that flights get through, and without empty cells, so that every leaf is live
    cloud = vcr.cloud_from_grid(desc, 1.0, 0.5)
    dense = orc.fbm_fill(SIZE, seed=4, octaves=4) + F(0.05)
    g = orc.Grid(dense, 0)
    cloud.max_extinction = g.max_density()
    prm = configs.C3_PPB.params(vcr.TRACKER_DDA)
    for i in range(3):
        prm.sun_dir[i] = sun[i]
    cam = vcr.camera_look((0.0, 0.0, -0.4), (0.0, 0.0, 1.0), 90.0, 0.1, W, H)
    with vcr.Context() as ctx:
        ctx.grid_upload(desc, dense)
        ctx.set_cloud(cloud)
        ctx.set_camera(cam)
        ctx.set_params(prm)
        ctx.set_frame(W, H)
        ctx.ppb_setup(photons, cap, 0.5, 0.8)  # the photons' paths do not depend on the radius
        ctx.ppb_pass(seed=seed, pass_index=0, crop=(0, 0, 1, 1))
        K = ctx.ppb_info()["beam_slots"]
        first = ctx.ppb_read("slots", photons).reshape(photons, K, 28)[:, 0]
        away = np.abs(first[:, 0])
        away[(first[:, 3:6] != np.array(list(prm.sun_dir), F)).any(axis=1) | (away < 0.015)] = np.inf
        beam = int(np.argmin(away)) * K
        radius = float(np.nextafter(F(away.min()), F(0)))
        assert radius < 0.05
        ctx.reset()
        ctx.ppb_setup(photons, cap, radius, 0.8)
        ctx.ppb_pass(seed=seed, pass_index=0)
        got = ctx.image_sum()
        assert ctx.ppb_info()["dropped"] == 0
        order = ctx.ppb_read("order")
        mine = np.flatnonzero(ctx.ppb_read("seg_beam")[order] == beam)  # in leaf order, as the boxes are
        a, b = ctx.ppb_read("seg_a")[order][mine], ctx.ppb_read("seg_b")[order][mine]
        lo, hi = ctx.ppb_read("leaf_lo")[mine], ctx.ppb_read("leaf_hi")[mine]
    turned_away = _turned_away(cam, cloud, H, a, b, lo, hi, first[beam // K, 10:26].max())
    assert turned_away >= 5, turned_away
    x0, cw = W // 2 - 6, 13
    want, _ = orc.ppb_pass(g, cloud, cam, prm, photons, cap, radius, 0.8, W, H, seed=seed, pass_index=0,
                           crop=(x0, 0, cw, H))
    np.testing.assert_array_equal(got[:, x0:x0 + cw], want[:, x0:x0 + cw])
