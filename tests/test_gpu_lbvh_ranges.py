"""The tree's boxes at the sizes where a node's range is read another way:
leaf by leaf up to 32 leaves, by a warp above, with clusters of 32, 32^2 and
32^3 leaves from 65 leaves on; equal keys (long one-sided ranges) included."""
import numpy as np
import pytest

import vcr
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [31, 33, 34, 64, 65, 97, 1025, 2049, 33 * 1024 + 1, 70000])
@pytest.mark.parametrize("bits", [30, 3, 0])  # bits of the key that differ
def test_node_boxes_are_the_unions_of_their_ranges(cuda, n, bits):
    import torch
    rng = np.random.default_rng(n + bits)
    codes = np.sort(rng.integers(0, 1 << bits, n) << (30 - bits)).astype(np.uint32)
    order = rng.permutation(n).astype(np.uint32)
    a, b = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    a[:, :3] = rng.random((n, 3), dtype=np.float32) - 0.5
    a[:, 3] = 0.01
    b[:, :3] = a[:, :3] + 0.05 * (rng.random((n, 3), dtype=np.float32) - 0.5)
    ref = orc.lbvh(codes, order, a, b)
    dev = [torch.from_numpy(x.view(np.int32) if x.dtype == np.uint32 else x).to(cuda) for x in (codes, order, a, b)]
    out = {k: torch.zeros(s, dtype=t, device=cuda) for k, s, t in
           [("left", n - 1, torch.int32), ("right", n - 1, torch.int32), ("node_lo", (n - 1, 4), torch.float32),
            ("node_hi", (n - 1, 4), torch.float32), ("leaf_lo", (n, 4), torch.float32),
            ("leaf_hi", (n, 4), torch.float32)]}
    with vcr.Context() as ctx:
        ctx.lbvh_build(*[d.data_ptr() for d in dev], n, *[out[k].data_ptr() for k in (
            "left", "right", "node_lo", "node_hi", "leaf_lo", "leaf_hi")])
        ctx.synchronize()
    for k, v in out.items():
        got = v.cpu().numpy()
        np.testing.assert_array_equal(got.view(np.uint32) if k in ("left", "right") else got, ref[k][:len(got)], err_msg=k)
