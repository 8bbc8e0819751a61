"""The training kernel's last, ragged tile: with targets that make its records
nearly all of the gradient, so that the gradient is theirs."""
import numpy as np
import pytest

import vcr
from oracle import oracle as orc
from oracle import oracle_nrc as onrc

pytestmark = pytest.mark.gpu

SMS = 152


# (records, of which in the last tile): it is a CTA's only, second, third and fourth tile
@pytest.mark.parametrize("n,tail", [(1, 1), (33, 33), (SMS * 128 + 1, 1), (2 * SMS * 128 + 17, 17),
                                    (3 * SMS * 128 + 100, 100)])
def test_gradient_of_the_last_tile(cuda, n, tail):
    # the loss's gradient is 2 (y - t) / (y^2 + 0.01): linear in the target, so records with targets of 1e6 outweigh
    # the others, of order 1, by more than their number; as at the other sizes 2^-6 of the whole gradient and 1e-2 of
    # the loss are allowed for the rounding to BF16 and the order of the FP32 sums
    desc = vcr.grid_desc((64, 32, 64), (1 / 64,) * 3)
    cloud = vcr.cloud_from_grid(desc, 1.0, 16.0)
    recs = onrc.random_records(n, cloud, np.random.default_rng(n))
    recs["w"][n - tail:] *= 1e6
    import torch
    with vcr.Context() as ctx:
        ctx.grid_upload(desc, orc.fbm_fill((64, 32, 64), seed=3, octaves=4))
        ctx.set_cloud(cloud)
        ctx.nrc_setup(train_samples=4096, seed=11)
        w = ctx.nrc_get_weights()
        dr = torch.from_numpy(recs.view(np.uint8).copy()).to(cuda)
        g, loss = ctx.nrc_gradient(dr.data_ptr(), n)
    gref, lref = onrc.gradient(w, recs, cloud)
    rest, _ = onrc.gradient(w, recs[:n - tail], cloud) if n > tail else (np.zeros_like(gref), 0.0)
    # the others are no more than a tenth: without the tail, or with another tile's inputs under it, the gradient
    # would be another one altogether
    assert np.linalg.norm(rest) * (n - tail) / n < 0.1 * np.linalg.norm(gref)
    assert abs(loss - lref) <= 1e-2 * abs(lref)
    assert np.linalg.norm(g - gref) <= 2.0 ** -6 * np.linalg.norm(gref)
