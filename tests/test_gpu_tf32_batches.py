"""TF32 plans: an image's result does not depend on the batch it is run in, so that a sharded batch equals the whole one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("net,batches", [("yolo160", (6, 7, 8, 33)), ("yolo224", (3, 8, 20)), ("cnn", (128, 200, 512, 4096))])
def test_rows_of_different_batches(zb, mode, net, batches):
    from zant_b200 import models
    ctx = zb.Context(0)
    ctx.set_tf32(mode)
    make = models.small_cnn_fp32 if net == "cnn" else (lambda b: models.tiny_yolo_fp32(b, res=int(net[4:])))
    full = zb.Plan(ctx, make(batches[-1]))
    x = np.random.default_rng(0).random(full.in_shape, dtype=np.float32)
    want = full.run(x)
    full.close()
    for b in batches[:-1]:
        plan = zb.Plan(ctx, make(b))
        got = plan.run(x[:b])
        plan.close()
        assert np.array_equal(got.view(np.uint32), want[:b].view(np.uint32)), b
    ctx.close()
