"""Frames with warps that start on training paths: with enough camera paths
to fill every warp, the training paths have a cursor of their own, the camera
paths' ids start behind them, and a warp goes over to camera paths when its
training paths are done.  Such a frame traces the paths of a pass and a
training step, each once."""
import numpy as np
import pytest

import vcr
from vcr import configs

pytestmark = pytest.mark.gpu

WARPS = 152 * 24  # that the launch has


# a few warps that start on training paths; more of them than the launch has warps
@pytest.mark.parametrize("samples", [2048, 393216])
def test_large_frame_equals_pass_and_train_step(cuda, samples):
    sc = configs.C1_PT
    W, H, spp = 640, 361, 2
    prm = sc.params(vcr.TRACKER_DDA)
    prm.nrc_events = 2
    res = []
    for mode in ("sequential", "frame"):
        with vcr.Context() as ctx:
            configs.setup_context(ctx, sc, width=W, height=H)
            ctx.set_params(prm)
            ctx.nrc_setup(train_samples=samples, learning_rate=3e-3, query_capacity=W * H * spp, seed=2)
            for k in range(3):  # the first calibrates the number of training paths
                if mode == "frame":
                    ctx.nrc_frame(seed=4, pass_index=k, spp=spp)
                    counters = np.array(ctx.counters())
                    queries = ctx.nrc_info()["queries"]
                else:
                    ctx.pt_pass(seed=4, pass_index=k, spp=spp)
                    camera, queries = np.array(ctx.counters()), ctx.nrc_info()["queries"]
                    ctx.nrc_train_step(seed=4, pass_index=k)
                    training = np.array(ctx.counters())
                    counters = camera + training
            ctx.synchronize()
            res.append((ctx.image_sum(), ctx.nrc_get_weights(), ctx.nrc_info(), counters, queries))
    assert camera[0] == W * H * spp >= 31 * WARPS
    assert training[0] >= 32 and (samples == 2048) == (training[0] < WARPS) and \
        (samples > 2048) == (training[0] > 16 * WARPS)
    (ia, wa, na, ca, qa), (ib, wb, nb, cb, qb) = res
    np.testing.assert_array_equal(cb, ca)  # paths, lookups, events and cells: every path once
    assert qa == qb and na["train_records"] == nb["train_records"] and na["steps"] == nb["steps"] == 3
    # the records come in another order, and with them the last bits of the gradient's FP32 sums: a
    # weight whose gradient is nothing but those moves by a step either way
    assert (np.abs(wb - wa) <= 1e-5).mean() > 0.999
    np.testing.assert_allclose(ib, ia, rtol=1e-4, atol=1e-7)
