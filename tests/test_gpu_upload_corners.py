"""Density lookups through the corner blocks right after an upload of several
slabs: the values a context without corner blocks gives, at points all over
the grid and around the planes where the slabs meet."""
import numpy as np
import pytest

import vcr

pytestmark = pytest.mark.gpu

# (size, z planes of a slab): one slab, three, four (the ring's first room is used again), a ring of the call's own
SIZES = [((9, 8, 7), 8), ((256, 256, 72), 32), ((512, 256, 61), 16), ((1024, 768, 20), 8), ((256, 256, 72), 32)]


def _points(size, planes, bounds, rng):
    """World positions: uniform, and within a voxel and a half of the slabs' planes and of the grid's faces."""
    n = np.array(size, np.float64)
    p = rng.uniform(-0.02, 1.02, (20000, 3))
    edges = np.append(np.arange(0, size[2] + planes, planes), size[2]).astype(np.float64)
    p[:14000, 2] = (edges[rng.integers(0, len(edges), 14000)] + rng.uniform(-1.5, 1.5, 14000)) / n[2]
    for a in range(2):
        face = slice(10000 + 2000 * a, 12000 + 2000 * a)
        p[face, a] = (rng.integers(0, 2, 2000) * n[a] + rng.uniform(-1.5, 1.5, 2000)) / n[a]
    lo, hi = (np.array(list(b), np.float64) for b in bounds)
    return (lo + p * (hi - lo)).astype(np.float32)


@pytest.mark.parametrize("prec", [vcr.PREC_FP32, vcr.PREC_FP16, vcr.PREC_BF16])
def test_lookups_after_an_upload_in_slabs(cuda, prec):
    import torch
    with vcr.Context() as ctx, vcr.Context() as plain:
        plain.set_tuning(corner_blocks=0)
        for k, (size, planes) in enumerate(SIZES):  # one context: streams, events and ring are used again
            rng = np.random.default_rng(20 + k)
            dense = rng.random(size[::-1], dtype=np.float32)
            desc = vcr.grid_desc(size, (1.0 / max(size),) * 3)
            cloud = vcr.cloud_from_grid(desc, 1.0, 8.0)
            points = torch.from_numpy(_points(size, planes, (cloud.bounds_min, cloud.bounds_max), rng)).to(cuda)
            out = []
            for c in (ctx, plain):
                got = torch.full((len(points),), -1.0, device=cuda)
                torch.cuda.synchronize()
                c.grid_upload(desc, dense, prec)
                c.set_cloud(cloud)
                c.grid_sample(points.data_ptr(), got.data_ptr(), len(points))
                c.synchronize()
                out.append(got.cpu().numpy())
            np.testing.assert_array_equal(out[0], out[1], err_msg=f"{size}")
            assert out[0].min() >= 0.0 and out[0].max() > 0.5
