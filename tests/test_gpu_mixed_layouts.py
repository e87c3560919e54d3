"""Plans with int8 and float parts on a context in TF32 mode: a dequantised tensor is float for every reader behind it.

Scales are powers of two and weights small integers, so that every product, sum and rounding to TF32 is exact."""
import numpy as np
import pytest

import graph_oracle

pytestmark = pytest.mark.gpu
CONV = dict(strides=(1, 1), dilations=(1, 1), group=1, auto_pad="NOTSET", pads=(1, 1, 1, 1))
POOL = dict(kernel_shape=(2, 2), strides=(2, 2), dilations=(1, 1), pads=(0, 0, 0, 0), auto_pad="NOTSET")


def quantized_branch(g, zb, rng, q, name, N, C, H, W, M):
    w = g.tensor("w" + name, zb.I8, (M, C, 3, 3), rng.integers(-127, 128, (M, C, 3, 3), dtype=np.int8))
    ws = g.tensor("s" + name, zb.F32, (1,), np.array([2.0 ** -7], np.float32))
    c = g.tensor("c" + name, zb.I8, (N, M, H, W))
    g.node("QLinearConv", [q, w, ws], [c], x_scale=0.5, x_zp=0, y_scale=32.0, y_zp=0, **CONV)
    d = g.tensor("d" + name, zb.F32, (N, M, H, W))
    g.node("DequantizeLinear", [c], [d], x_scale=0.25, x_zp=0)
    return d


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("behind", ["pool", "concat"])
def test_dequantised_tensor_in_front_of_float_convolutions(zb, oracle, mode, behind):
    rng = np.random.default_rng(mode)
    N, C, H, W, M = 2, 3, 24, 20, 16
    g = zb.Graph("mixed")
    x = g.tensor("x", zb.F32, (N, C, H, W))
    q = g.tensor("q", zb.U8, (N, C, H, W))
    g.node("QuantizeLinear", [x], [q], y_scale=0.5, y_zp=0)
    cur = quantized_branch(g, zb, rng, q, "a", N, C, H, W, M)
    cin = M
    if behind == "pool":
        H, W = H // 2, W // 2
        p = g.tensor("p", zb.F32, (N, M, H, W))
        g.node("MaxPool", [cur], [p], **POOL)
        cur = p
    else:
        m = g.tensor("m", zb.F32, (N, 2 * M, H, W))
        g.node("Concat", [cur, quantized_branch(g, zb, rng, q, "b", N, C, H, W, M)], [m], axis=1)
        cur, cin = m, 2 * M
    w = g.tensor("w", zb.F32, (32, cin, 3, 3), rng.integers(-2, 3, (32, cin, 3, 3)).astype(np.float32))
    f = g.tensor("f", zb.F32, (N, 32, H, W))
    g.node("Conv", [cur, w], [f], **CONV)
    y = g.tensor("y", zb.F32, (N, 32, H, W))
    g.node("Relu", [f], [y])
    g.input, g.output = x, y
    xin = rng.integers(0, 128, (N, C, 24, 20)).astype(np.float32)
    want = graph_oracle.run(oracle, g, xin)[y]
    c = zb.Context(0)
    try:
        c.set_tf32(mode)
        plan = zb.Plan(c, g)
        names = plan.step_names()
        got = plan.run(xin)
        plan.close()
    finally:
        c.close()
    assert any("tf32" in n for n in names), names
    assert np.array_equal(got, want), names
    assert len(np.unique(want)) > 30
