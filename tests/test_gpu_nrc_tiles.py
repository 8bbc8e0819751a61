"""The training kernel's gradient at the record counts where its tiles and
buffers change: a single record, the edges of the 32-record fragments and the
128-record tiles, and two, three and four tiles on some CTAs (the inputs have
two buffers, the gradients of the layers two, taken in turn)."""
import numpy as np
import pytest

import vcr
from oracle import oracle as orc
from oracle import oracle_nrc as onrc

pytestmark = pytest.mark.gpu

SMS = 152


@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, SMS * 128 + 1, 2 * SMS * 128 + 17, 3 * SMS * 128 + 100])
def test_gradient_at_tile_edges(cuda, n):
    # the oracle rounds to BF16 where the GPU does; what is left is the order
    # of the FP32 sums and the roundings it tips: far below one BF16 step (2^-8)
    # of the whole gradient, allowed 2^-6
    desc = vcr.grid_desc((64, 32, 64), (1 / 64,) * 3)
    cloud = vcr.cloud_from_grid(desc, 1.0, 16.0)
    recs = onrc.random_records(n, cloud, np.random.default_rng(n))
    import torch
    with vcr.Context() as ctx:
        ctx.grid_upload(desc, orc.fbm_fill((64, 32, 64), seed=3, octaves=4))
        ctx.set_cloud(cloud)
        ctx.nrc_setup(train_samples=4096, seed=11)
        w = ctx.nrc_get_weights()
        dr = torch.from_numpy(recs.view(np.uint8).copy()).to(cuda)
        g, loss = ctx.nrc_gradient(dr.data_ptr(), n)
    gref, lref = onrc.gradient(w, recs, cloud)
    assert abs(loss - lref) <= 1e-2 * abs(lref)
    assert np.linalg.norm(g - gref) <= 2.0 ** -6 * np.linalg.norm(gref)
    out = g[5 * 64 * 64:].reshape(64, 16)
    assert np.all(out[:, 3:] == 0)
