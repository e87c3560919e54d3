"""Pointwise QLinearConv in a plan whose filters leave their last tile partly empty: the whole tiles and the rest as parts.

Integer results: they have to equal the oracle's exactly."""
import numpy as np
import pytest

import graph_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [96, 90, 144, 192, 160, 224, 250])       # 64 + 32, 64 + 26, 128 + 16, 128 + 64, 128 + 32; one launch
@pytest.mark.parametrize("u8,act", [(False, "relu6"), (True, "relu"), (False, None)])
def test_parts(zb, ctx, oracle, M, u8, act):
    N, C, H, W = 320 if M < 128 else 160, 4, 48, 52                                         # 2496 pixels: ragged groups and chunks
    rng = np.random.default_rng(M)
    g = zb.Graph("parts")
    x = g.tensor("x", zb.U8 if u8 else zb.I8, (N, C, H, W))
    w = g.tensor("w", zb.I8, (M, C, 1, 1), rng.integers(-127, 128, (M, C, 1, 1), dtype=np.int8))
    ws = g.tensor("s", zb.F32, (M,), (rng.random(M, dtype=np.float32) * 0.01 + 0.002).astype(np.float32))
    b = g.tensor("b", zb.I32, (M,), rng.integers(-3000, 3000, M).astype(np.int32))
    y = g.tensor("y", zb.I8, (N, M, H, W))
    g.node("QLinearConv", [x, w, ws, -1, b], [y], x_scale=0.05, x_zp=100 if u8 else 0, y_scale=0.1, y_zp=0, pads=(0,) * 4, strides=(1, 1), dilations=(1, 1), group=1,
           auto_pad="NOTSET", activation=act)
    g.input, g.output = x, y
    xv = (rng.integers(0, 256, (N, C, H, W)).astype(np.uint8) if u8 else rng.integers(-128, 128, (N, C, H, W)).astype(np.int8))
    want = graph_oracle.run(oracle, g, xv)
    plan = zb.Plan(ctx, g, fuse=True)
    assert np.array_equal(plan.run(xv), want[g.output])
    assert plan.launches_per_run == (1 if M > 192 else 2)
    assert len(np.unique(want[g.output])) > 16
    plan.close()
