"""Majorant-grid walks of rays that meet the cloud's box at an edge: moved to
the box, such a ray may miss it by a rounding, and the walk then goes as far as
the box test had got.  Cells and distances equal the oracle's."""
import numpy as np
import pytest

import vcr
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

SIZE = (48, 38, 36)


@pytest.mark.parametrize("level", [0, 2])
def test_rays_at_the_boxs_edges(cuda, level):
    import torch
    desc = vcr.grid_desc(SIZE, (1 / 48,) * 3)
    cloud = vcr.cloud_from_grid(desc, 1.0, 8.0)
    dense = orc.fbm_fill(SIZE, seed=2, octaves=4)
    og = orc.Grid(dense, 0)
    rng = np.random.default_rng(5)
    n, mc = 40000, 64
    lo, hi = np.array(list(cloud.bounds_min)), np.array(list(cloud.bounds_max))
    along_edge = np.arange(3)[None] == rng.integers(0, 3, n)[:, None]
    p = lo + (hi - lo) * np.where(along_edge, rng.random((n, 3)), rng.integers(0, 2, (n, 3)))
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o = (p - d * rng.uniform(0.5, 3.0, (n, 1))).astype(np.float32)
    d = d.astype(np.float32)
    with vcr.Context() as ctx:
        ctx.grid_upload(desc, dense)
        ctx.set_cloud(cloud)
        ctx.set_tuning(majorant_level=level)
        d_o, d_d = torch.from_numpy(o).to(cuda), torch.from_numpy(d).to(cuda)
        cells = torch.zeros((n, mc), dtype=torch.int32, device=cuda)
        tt = torch.zeros((n, mc, 2), dtype=torch.float32, device=cuda)
        cnt = torch.zeros(n, dtype=torch.int32, device=cuda)
        ctx.dda_trace(d_o.data_ptr(), d_d.data_ptr(), n, mc, cells.data_ptr(), tt.data_ptr(), cnt.data_ptr())
        ctx.synchronize()
    oc, ot, on = og.dda_trace(cloud, o, d, mc, level)
    assert (on > 0).sum() > n // 8
    np.testing.assert_array_equal(cnt.cpu().numpy().view(np.uint32), on)
    mask = np.arange(mc)[None, :] < on[:, None]
    np.testing.assert_array_equal(cells.cpu().numpy().view(np.uint32)[mask], oc[mask])
    np.testing.assert_array_equal(tt.cpu().numpy()[mask], ot[mask])
