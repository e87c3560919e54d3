"""Nodes that a plan takes together are held to the rules of the nodes on their own: what is refused one by one is refused fused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CONV = dict(strides=(1, 1), dilations=(1, 1), group=1, auto_pad="NOTSET", pads=(1, 1, 1, 1))


def int8_graph(zb, w_zp=1, resize=None, dequant_inputs=1):
    """QuantizeLinear -> two channels-last convolutions -> [Resize] -> DequantizeLinear."""
    rng = np.random.default_rng(0)
    N, H, W, M = 1, 20, 20, 16
    g = zb.Graph("checks")
    x, q = g.tensor("x", zb.F32, (N, 3, H, W)), g.tensor("q", zb.U8, (N, 3, H, W))
    g.node("QuantizeLinear", [x], [q], y_scale=0.5, y_zp=0)
    cur, cin = q, 3
    for i in range(2):
        w = g.tensor(f"w{i}", zb.I8, (M, cin, 3, 3), rng.integers(-127, 128, (M, cin, 3, 3), dtype=np.int8))
        s = g.tensor(f"s{i}", zb.F32, (1,), np.array([0.01], np.float32))
        z = g.tensor(f"z{i}", zb.I32, (w_zp,), np.zeros(w_zp, np.int32))
        y = g.tensor(f"y{i}", zb.I8, (N, M, H, W))
        g.node("QLinearConv", [cur, w, s, z], [y], x_scale=0.5, x_zp=0, y_scale=8.0, y_zp=0, **CONV)
        cur, cin = y, M
    if resize:
        u = g.tensor("u", zb.I8, (N, M, 2 * H, 2 * W))
        g.node("Resize", [cur], [u], scales=resize, coord_mode="half_pixel")
        w = g.tensor("w2", zb.I8, (M, M, 3, 3), rng.integers(-127, 128, (M, M, 3, 3), dtype=np.int8))
        cur2 = g.tensor("y2", zb.I8, (N, M, 2 * H, 2 * W))
        g.node("QLinearConv", [u, w, s], [cur2], x_scale=8.0, x_zp=0, y_scale=80.0, y_zp=0, **CONV)
        cur, H, W = cur2, 2 * H, 2 * W
    d = g.tensor("d", zb.F32, (N, M, H, W))
    g.node("DequantizeLinear", [cur] + [s] * (dequant_inputs - 1), [d], x_scale=1.0, x_zp=0)
    g.input, g.output = x, d
    return g


def dense_graph(zb, rank):
    g = zb.Graph("dense")
    one = (1,) * (rank - 2)
    x, w = g.tensor("x", zb.F32, one + (4, 8)), g.tensor("w", zb.F32, one + (8, 6), np.ones(one + (8, 6), np.float32))
    b = g.tensor("b", zb.F32, (6,), np.arange(6, dtype=np.float32))
    m, a = g.tensor("m", zb.F32, one + (4, 6)), g.tensor("a", zb.F32, one + (4, 6))
    g.node("MatMul", [x, w], [m])
    g.node("Add", [m, b], [a])
    g.input, g.output = x, a
    return g


@pytest.mark.parametrize("make,name", [
    (lambda zb: int8_graph(zb, w_zp=5), "InputTensorsWrongShape"),                                    # neither one zero point nor one per filter
    (lambda zb: int8_graph(zb, resize=(1.0, 1.0, 3.0, 3.0)), "OutputTensorDifferentSize"),            # scales that do not give the output's shape
    (lambda zb: int8_graph(zb, dequant_inputs=2), "InvalidInput"),
    (lambda zb: dense_graph(zb, 5), "Unsupported"),                                                   # broadcast Add above rank 4
])
def test_refused_alike(zb, ctx, make, name):
    for fuse in (False, True):
        with pytest.raises(zb.ZantError) as e:
            zb.Plan(ctx, make(zb), fuse=fuse).close()
        assert e.value.name == name, fuse


@pytest.mark.parametrize("make", [lambda zb: int8_graph(zb, w_zp=16), lambda zb: int8_graph(zb, resize=(1.0, 1.0, 2.0, 2.0)), lambda zb: dense_graph(zb, 4)])
def test_accepted_alike(zb, ctx, make):
    x = np.random.default_rng(1).integers(0, 100, 1200).astype(np.float32)
    outs = []
    for fuse in (False, True):
        plan = zb.Plan(ctx, make(zb), fuse=fuse)
        outs.append(plan.run(x[:int(np.prod(plan.in_shape))].reshape(plan.in_shape)))
        plan.close()
    assert np.array_equal(*outs)
