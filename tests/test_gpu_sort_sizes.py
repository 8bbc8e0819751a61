"""The radix sort's dispatch: one CTA up to 8,192 pairs, then tiles of 4,096,
6,144 and 8,192 keys.  Sizes at the edges of each, keys at an address that is
not a multiple of 16 bytes, in place, and few distinct digits."""
import numpy as np
import pytest

import vcr

pytestmark = pytest.mark.gpu

SIZES = [1, 33, 1023, 1024, 1025, 2049, 4095, 4097, 8191, 8192, 8193, 12288, 12289, (1 << 20) - 1, 1 << 20,
         (1 << 20) + 1, 6144 * 200 + 1, 1 << 23, (1 << 23) + 1, 8192 * 1100 - 1]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("bits,kind", [((0, 32), "random"), ((5, 30), "random"), ((0, 32), "few")])
def test_sizes_at_the_edges(cuda, n, bits, kind):
    import torch
    g = torch.Generator(device=cuda).manual_seed(n % 1000)
    buf = torch.randint(-(1 << 31), (1 << 31) - 1, (n + 3,), dtype=torch.int32, device=cuda, generator=g)
    if kind == "few":
        buf = (buf % 3) * 0x01000100
    keys = buf[3:]  # 12 bytes past a 16-byte boundary
    vals = torch.randint(-(1 << 31), (1 << 31) - 1, (n,), dtype=torch.int32, device=cuda, generator=g)
    k0 = keys.cpu().numpy().view(np.uint32).copy()
    v0 = vals.cpu().numpy().view(np.uint32).copy()
    mask = np.uint32(((1 << (bits[1] - bits[0])) - 1) << bits[0])
    perm = np.argsort(k0 & mask, kind="stable")
    ko, vo = torch.empty_like(vals), torch.empty_like(vals)
    with vcr.Context() as ctx:
        ctx.radix_sort_pairs(keys.data_ptr(), vals.data_ptr(), ko.data_ptr(), vo.data_ptr(), n, *bits)
        ctx.radix_sort_pairs(keys.data_ptr(), vals.data_ptr(), keys.data_ptr(), vals.data_ptr(), n, *bits)
        ctx.synchronize()
    for k, v in ((ko, vo), (keys, vals)):
        np.testing.assert_array_equal(k.cpu().numpy().view(np.uint32), k0[perm])
        np.testing.assert_array_equal(v.cpu().numpy().view(np.uint32), v0[perm])
