"""Pointwise QLinearConv layers with so few pixels that the tiles are cut smaller to fill the SMs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [(1, 192, 28, 28, 32), (1, 96, 56, 56, 24), (3, 32, 20, 20, 64), (1, 16, 20, 28, 200), (37, 32, 20, 20, 32), (1, 24, 72, 40, 130)])
def test_pixel_tiles(zb, ctx, oracle, case):
    N, C, H, W, M = case
    rng = np.random.default_rng(M)
    x = rng.integers(-128, 128, (N, C, H, W)).astype(np.int8)
    w = rng.integers(-127, 128, (M, C, 1, 1), dtype=np.int8)
    ws = rng.uniform(0.5, 1.5, M).astype(np.float32)
    args = (x, 0.02, 0, w, ws, None, float(0.02 * 73.0 * 74.0 * np.sqrt(C) / 50.0), 0)
    kw = dict(bias=rng.integers(-2000, 2000, M).astype(np.int32), y_dtype=zb.I8, stride=(1, 1), pads=(0,) * 4, dilations=(1, 1), group=1, activation=None)
    assert np.array_equal(ctx.qlinearconv(*args, **kw), oracle.qlinearconv(*args, **kw))
