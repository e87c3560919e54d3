"""QLinearAdd: the division-free rounding against the oracle, on its own and in the epilogue of the convolution in front of it.

Integer results: they have to equal the oracle's exactly, ties included."""
import numpy as np
import pytest

import graph_oracle

pytestmark = pytest.mark.gpu
CONV = dict(dilations=(1, 1), auto_pad="NOTSET")


@pytest.mark.parametrize("u8", [False, True])
@pytest.mark.parametrize("scales", [(0.1, 0.1, 0.1), (0.5, 0.25, 1.0), (0.1, 0.05, 0.2), (0.0472441, 0.1, 0.1), (3.0, 1e-4, 0.7), (1.0, 1.0, 0.001), (1e-38, 0.1, 0.1)])
@pytest.mark.parametrize("act", [None, "relu6"])
def test_every_pair_of_codes(ctx, oracle, u8, scales, act):
    """all 65536 pairs: exact ties (scales that are powers of two apart), saturation, scales the fast form does not take"""
    dt = np.uint8 if u8 else np.int8
    codes = np.arange(256, dtype=np.uint8).view(dt)
    a, b = (np.ascontiguousarray(v) for v in np.meshgrid(codes, codes))
    for azp, bzp, yzp in ((0, 0, 0), (3, 9, 5)):
        args = (a, scales[0], azp, b, scales[1], bzp, scales[2], yzp)
        assert np.array_equal(ctx.qlinearadd(*args, activation=act), oracle.qlinearadd(*args, activation=act))


# N C H W M k (filters), y_zp of the sum, relu in front of the addition, residual first
CASES = [
    (64, 8, 64, 64, 32, 0, False, True),       # pointwise, four pixel groups of 32 lanes
    (8, 8, 212, 212, 24, 0, True, False),      # pointwise, ragged groups and chunks
    (24, 8, 64, 64, 96, 0, False, False),      # pointwise, one tile, no groups
    (40, 8, 40, 40, 132, -7, True, True),      # two filter tiles, chunks of 16 pixels
    (700, 8, 14, 14, 64, 5, False, True),      # 196-byte planes: staged output
    (2100, 8, 10, 10, 40, 0, True, False),     # 100-byte planes
    (1, 96, 14, 14, 64, 3, False, True),       # few positions: whole words
    (2, 64, 7, 7, 33, 0, False, True),         # few positions: bytes, a ragged filter tile
    (7, 128, 1, 1, 48, -3, True, False),       # few positions: one pixel per image
    (2, 32, 20, 28, 24, 0, False, True),       # pointwise, little output: the addition stays a step of its own
]


@pytest.mark.parametrize("case", CASES, ids=[f"res{i}" for i in range(len(CASES))])
def test_fused(zb, ctx, oracle, case):
    N, C, H, W, M, yzp, relu, first = case
    rng = np.random.default_rng(C + H + M)
    g = zb.Graph("res")
    x = g.tensor("x", zb.I8, (N, C, H, W))
    def conv(src, cin, name, sy):
        w = g.tensor(f"w{name}", zb.I8, (M, cin, 1, 1), rng.integers(-127, 128, (M, cin, 1, 1), dtype=np.int8))
        ws = g.tensor(f"s{name}", zb.F32, (M,), (rng.random(M, dtype=np.float32) * 0.01 + 0.002).astype(np.float32))
        b = g.tensor(f"b{name}", zb.I32, (M,), rng.integers(-3000, 3000, M).astype(np.int32))
        y = g.tensor(f"c{name}", zb.I8, (N, M, H, W))
        g.node("QLinearConv", [src, w, ws, -1, b], [y], x_scale=0.05, x_zp=0, y_scale=sy, y_zp=0, pads=(0,) * 4, strides=(1, 1), group=1, **CONV)
        return y
    r = conv(x, C, "r", 0.3)
    cur = conv(r, M, "c", 0.25)
    if relu:
        a = g.tensor("relu", zb.I8, (N, M, H, W))
        g.node("Relu", [cur], [a], x_scale=0.25, x_zp=0, y_scale=0.25, y_zp=0)
        cur = a
    y = g.tensor("sum", zb.I8, (N, M, H, W))
    ins, at = ([r, cur], dict(x_scale=0.3, x_zp=0, b_scale=0.25, b_zp=0)) if first else ([cur, r], dict(x_scale=0.25, x_zp=0, b_scale=0.3, b_zp=0))
    g.node("QLinearAdd", ins, [y], y_scale=0.5, y_zp=yzp, **at)
    out = g.tensor("out", zb.F32, (N, M, H, W))
    g.node("DequantizeLinear", [y], [out], x_scale=0.5, x_zp=yzp)
    g.input, g.output = x, out
    xv = rng.integers(-128, 128, (N, C, H, W)).astype(np.int8)
    want = graph_oracle.run(oracle, g, xv)
    plan = zb.Plan(ctx, g, fuse=True)
    assert np.array_equal(plan.run(xv), want[g.output])
    assert len(np.unique(want[g.output])) > 30
    fused = any("+QLinearAdd" in n for n in plan.step_names())
    assert fused == (case != CASES[-1]), plan.step_names()
    plan.close()


def test_operand_that_is_the_output(zb, ctx, oracle):
    """A Reshape of the residual operand is the graph's output: the operand lies in the caller's buffer then, so the addition, whose
    loads in the convolution's epilogue are words, stays a step of its own."""
    rng = np.random.default_rng(3)
    g = zb.Graph("res")
    x = g.tensor("x", zb.I8, (64, 8, 64, 64))

    def conv(src, cin, name):
        w = g.tensor(f"w{name}", zb.I8, (32, cin, 1, 1), rng.integers(-127, 128, (32, cin, 1, 1), dtype=np.int8))
        ws = g.tensor(f"s{name}", zb.F32, (32,), (rng.random(32, dtype=np.float32) * 0.01 + 0.002).astype(np.float32))
        y = g.tensor(f"c{name}", zb.I8, (64, 32, 64, 64))
        g.node("QLinearConv", [src, w, ws, -1, -1], [y], x_scale=0.05, x_zp=0, y_scale=0.3, y_zp=0, pads=(0,) * 4, strides=(1, 1), group=1, **CONV)
        return y

    r = conv(x, 8, "r")
    cur = conv(r, 32, "c")
    y = g.tensor("sum", zb.I8, (64, 32, 64, 64))
    g.node("QLinearAdd", [r, cur], [y], x_scale=0.3, x_zp=0, b_scale=0.3, b_zp=0, y_scale=0.5, y_zp=0)
    flat = g.tensor("flat", zb.I8, (64, 32 * 64 * 64))
    g.node("Reshape", [r], [flat])
    g.input, g.output = x, flat
    xv = rng.integers(-128, 128, (64, 8, 64, 64)).astype(np.int8)
    want = graph_oracle.run(oracle, g, xv)
    plan = zb.Plan(ctx, g, fuse=True)
    assert not any("+QLinearAdd" in n for n in plan.step_names())
    assert np.array_equal(plan.run(xv), want[flat]) and np.array_equal(plan.read_tensor(y), want[y])
    plan.close()


@pytest.mark.parametrize("N,M,H,W,fused", [(16, 24, 32, 32, True), (15, 24, 32, 32, False), (28, 64, 20, 12, True), (11, 96, 32, 32, True), (10, 96, 32, 32, False), (33, 132, 16, 16, True)])
def test_short_form_in_the_epilogue(zb, ctx, oracle, N, M, H, W, fused):
    """Scales for which the rounding needs no division (proved when the plan is built): on either side of the sizes from which the addition is
    part of the convolution's step."""
    rng = np.random.default_rng(N + M)
    g = zb.Graph("res")
    x = g.tensor("x", zb.I8, (N, 8, H, W))
    sx, sr, sc, sy = 0.05, 0.0931, 0.1173, 0.2117

    def conv(src, cin, s_in, name, s_out):
        w = g.tensor(f"w{name}", zb.I8, (M, cin, 1, 1), rng.integers(-127, 128, (M, cin, 1, 1), dtype=np.int8))
        ws = g.tensor(f"s{name}", zb.F32, (M,), (rng.uniform(0.7, 1.3, M) * 60.0 * s_out / (s_in * 40.0 * 73.0 * np.sqrt(cin))).astype(np.float32))
        y = g.tensor(f"c{name}", zb.I8, (N, M, H, W))
        g.node("QLinearConv", [src, w, ws, -1, -1], [y], x_scale=s_in, x_zp=0, y_scale=s_out, y_zp=0, pads=(0,) * 4, strides=(1, 1), group=1, **CONV)
        return y

    r = conv(x, 8, sx, "r", sr)
    cur = conv(r, M, sr, "c", sc)
    y = g.tensor("sum", zb.I8, (N, M, H, W))
    g.node("QLinearAdd", [r, cur], [y], x_scale=sr, x_zp=0, b_scale=sc, b_zp=0, y_scale=sy, y_zp=0)
    out = g.tensor("out", zb.F32, (N, M, H, W))
    g.node("DequantizeLinear", [y], [out], x_scale=sy, x_zp=0)
    g.input, g.output = x, out
    xv = rng.integers(-128, 128, (N, 8, H, W)).astype(np.int8)
    want = graph_oracle.run(oracle, g, xv)
    plan = zb.Plan(ctx, g, fuse=True)
    assert any("+QLinearAdd" in n for n in plan.step_names()) == fused, plan.step_names()
    assert np.array_equal(plan.run(xv), want[g.output])
    assert len(np.unique(want[y])) > 100
    plan.close()
