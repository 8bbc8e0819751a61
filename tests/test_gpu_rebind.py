"""A cloud bound while passes that were queued before are still running on a
stream of the caller's: what is bound is the cloud, whatever the passes do
(each clears the words it counts in when it starts)."""
import numpy as np
import pytest

import vcr
from vcr import configs

pytestmark = pytest.mark.gpu


def test_a_cloud_bound_among_running_passes_is_whole(cuda):
    import torch
    sc, W, H = configs.C1_PT, 256, 256
    stream = torch.cuda.Stream()  # does not synchronise with the default stream
    with vcr.Context() as ctx:
        configs.setup_context(ctx, sc, width=W, height=H)
        want_max, levels = ctx.grid_info()[0], [ctx.majorants(k) for k in range(4)]
        ctx.pt_pass(seed=3, pass_index=0)
        ctx.synchronize()
        want = ctx.image_sum()
        for _ in range(5):
            for k in range(40):
                ctx.pt_pass(seed=1, pass_index=k, stream=stream.cuda_stream)
            ctx.grid_generate(sc.grid_desc(), sc.fbm(), sc.precision)
            assert ctx.grid_info()[0] == want_max
        ctx.synchronize()
        for k in range(4):
            np.testing.assert_array_equal(ctx.majorants(k), levels[k])
        ctx.reset()
        ctx.pt_pass(seed=3, pass_index=0)
        ctx.synchronize()
        np.testing.assert_array_equal(ctx.image_sum(), want)
