"""The int8 CNN as one kernel on clusters (fused_cnn_few.cuh) at every number of images a cluster, and the four kernels just above its last batch."""
import numpy as np
import pytest

import graph_oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def models(zb):
    from zant_b200 import models
    return models


@pytest.fixture(scope="module")
def scales(zb, ctx, models):
    return models.calibrate_on_gpu(ctx, models.small_cnn_fp32(64), models.small_cnn_input(64))


def _check(zb, ctx, oracle, g, x, steps):
    want = graph_oracle.run(oracle, g, x)[g.output]
    plan = zb.Plan(ctx, g, fuse=True)
    assert len(plan.step_names()) == steps
    for graph in (False, True):
        plan.use_graph(graph)
        for _ in range(2):
            assert np.array_equal(plan.run(x).view(np.uint32), want.view(np.uint32))
    plan.close()
    assert len(np.unique(want)) > 8


@pytest.mark.parametrize("batch", [3, 15, 16, 29, 30, 31, 59, 60, 61, 119, 120, 121, 127, 240, 241, 480])
def test_images_of_a_cluster(zb, ctx, oracle, models, scales, batch):
    g = models.small_cnn_int8(batch, act_scales=scales, bias_amplitude=(100, 1000, 5000, 300))
    _check(zb, ctx, oracle, g, models.small_cnn_input(batch, batch), 1)


@pytest.mark.parametrize("batch", [481, 513, 640])
def test_four_kernels_above(zb, ctx, oracle, models, scales, batch):
    g = models.small_cnn_int8(batch, act_scales=scales, bias_amplitude=(100, 1000, 5000, 300))
    x = models.small_cnn_input(batch, batch)
    x.reshape(-1)[::97] = np.resize(np.array([np.nan, np.inf, -np.inf, -0.0, 1.0e-30], np.float32), x.reshape(-1)[::97].size)
    _check(zb, ctx, oracle, g, x, 4)


@pytest.mark.parametrize("batch,steps", [(4, 1), (500, 4)])
def test_device_input_of_any_address(zb, ctx, oracle, models, scales, batch, steps):
    """Images are read 16 bytes at a time: a caller's device buffer at another address is refused, in a replayed graph, which copies it, it is not."""
    import torch
    g = models.small_cnn_int8(batch, act_scales=scales)
    x = models.small_cnn_input(batch, batch)
    want = graph_oracle.run(oracle, g, x)[g.output]
    plan = zb.Plan(ctx, g, fuse=True)
    assert len(plan.step_names()) == steps
    buf = torch.zeros(x.size + 8, device="cuda")
    y = torch.empty(want.shape, device="cuda")
    for graph in (False, True):
        plan.use_graph(graph)
        for offset in (0, 1, 2, 4):
            xd = buf[offset:offset + x.size].view(x.shape)
            xd.copy_(torch.from_numpy(x))
            y.fill_(99.0)
            torch.cuda.synchronize()
            if offset % 4 and not graph:
                with pytest.raises(zb.ZantError, match="InvalidInput"):
                    plan.run(xd, y)
                continue
            plan.run(xd, y)
            ctx.synchronize()
            assert np.array_equal(y.cpu().numpy().view(np.uint32), want.view(np.uint32))
    plan.close()
