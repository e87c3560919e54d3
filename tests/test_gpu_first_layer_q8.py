"""First layers of int8 networks whose input the convolution quantises itself (first_layer_q8.cuh): one to four channels, 16 to 64 filters, pooled widths
around the units of 16 pixels, bands with rows to spare, both code types, scales and zero points of either quantisation path, every kind of activation.  Bit for bit against the oracle: whole numbers throughout."""
import numpy as np
import pytest

import graph_oracle

pytestmark = pytest.mark.gpu

POOL = dict(kernel_shape=(2, 2), strides=(2, 2), dilations=(1, 1), pads=(0, 0, 0, 0), auto_pad="NOTSET")

CASES = [
    # N  C   H   W   M  type  zero point  scale  activation
    (2, 3, 64, 64, 16, "U8", 0, 1 / 255, "leaky"),
    (1, 3, 36, 70, 32, "U8", 0, 1 / 255, None),            # 35 pooled columns; floats one at a time, half a word at the end of a row
    (2, 1, 34, 66, 64, "I8", 0, 1 / 127, "relu"),          # one pooled column behind two units
    (3, 4, 48, 62, 48, "I8", 0, 1 / 127, "leaky"),         # 31 pooled columns
    (1, 2, 50, 96, 16, "U8", 7, 1 / 200, "clip"),          # a zero point of the quantisation
    (2, 3, 36, 72, 16, "I8", -3, 1 / 100, "relu6"),
    (2, 3, 40, 68, 32, "U8", 0, 2.0e30, "leaky"),          # a scale without the two-step quotient
    (230, 1, 28, 128, 16, "U8", 0, 1 / 255, "leaky"),      # bands of eight rows, the second with six
    (1, 1, 130, 520, 32, "U8", 0, 1 / 255, "relu"),        # two rounds of words a lane
    (2, 3, 2, 2, 16, "U8", 0, 1 / 255, "leaky"),           # one pooled pixel
    # bands whose rows and the activation's table just fill what a launch may have of shared memory, or would be above it
    (2, 3, 1200, 1600, 16, "U8", 0, 1 / 255, "leaky"),     # four pooled rows
    (1, 3, 1184, 2688, 16, "U8", 0, 1 / 255, "leaky"),     # two
    (1, 1, 4736, 2628, 16, "U8", 0, 1 / 255, None),        # eight
    (1, 1, 2368, 4804, 16, "I8", 0, 1 / 127, "relu"),      # four
    (1, 1, 1184, 8068, 16, "U8", 0, 1 / 255, "leaky"),     # two
    (1, 1, 2368, 4738, 16, "U8", 0, 1 / 255, "leaky"),     # four
    (4, 4, 1184, 640, 16, "U8", 0, 1 / 255, None),         # eight
    (2, 4, 600, 1924, 32, "U8", 0, 1 / 255, "leaky"),      # two
    (1, 2, 4, 6080, 16, "U8", 0, 1 / 255, "leaky"),        # one
    (1, 1, 4, 12160, 16, "U8", 0, 1 / 255, "leaky"),       # one
]


@pytest.mark.parametrize("case", CASES, ids=[f"first{i}" for i in range(len(CASES))])
def test_quantising_first_layer(zb, ctx, oracle, case):
    N, C, H, W, M, dt, zp, scale, act = case
    rng = np.random.default_rng(M + H)
    scale = float(np.float32(scale))
    g = zb.Graph("first")
    dtype = zb.U8 if dt == "U8" else zb.I8
    x = g.tensor("x", zb.F32, (N, C, H, W))
    q = g.tensor("xq", dtype, (N, C, H, W))
    g.node("QuantizeLinear", [x], [q], y_scale=scale, y_zp=zp)
    w = g.tensor("w", zb.I8, (M, C, 3, 3), rng.integers(-128, 128, (M, C, 3, 3), dtype=np.int8))
    sw = (rng.random(M, dtype=np.float32) * 0.01 + 0.002).astype(np.float32)
    b = g.tensor("b", zb.I32, (M,), rng.integers(-3000, 3000, M).astype(np.int32))
    y = g.tensor("c", zb.I8, (N, M, H, W))
    sx = float(np.float32(1 / 255))
    sy = float(np.float32(sx * 0.007 * 74 * 90 * np.sqrt(C * 9) / 40))
    ws = g.tensor("s", zb.F32, (M,), sw)
    extra = dict(activation="relu6") if act == "relu6" else {}
    conv = dict(strides=(1, 1), dilations=(1, 1), group=1, auto_pad="NOTSET")
    g.node("QLinearConv", [q, w, ws, -1, b], [y], x_scale=sx, x_zp=0, y_scale=sy, y_zp=0, pads=(1, 1, 1, 1), **conv, **extra)
    cur, s = y, sy
    if act in ("leaky", "relu", "clip"):
        a = g.tensor("a", zb.I8, (N, M, H, W))
        if act == "relu":
            g.node("Relu", [cur], [a], x_scale=s, x_zp=0, y_scale=s, y_zp=0)
        elif act == "leaky":
            g.node("LeakyRelu", [cur], [a], alpha=0.1, x_scale=s, x_zp=0, y_scale=s * 0.8, y_zp=0)
            s *= 0.8
        else:
            g.node("Clip", [cur], [a], alpha=0.0, beta=float(s * 60), x_scale=s, x_zp=0, y_scale=s, y_zp=0)
        cur = a
    PH, PW = H // 2, W // 2
    p = g.tensor("p", zb.I8, (N, M, PH, PW))
    g.node("MaxPool", [cur], [p], **POOL)
    # a reader of the channels-last result
    w1 = g.tensor("w1", zb.I8, (16, M, 1, 1), rng.integers(-127, 128, (16, M, 1, 1), dtype=np.int8))
    s1 = g.tensor("s1", zb.F32, (1,), np.array([0.01], np.float32))
    c1 = g.tensor("c1", zb.I8, (N, 16, PH, PW))
    sy1 = float(np.float32(s * 0.01 * 74 * 40 * np.sqrt(M) / 40))
    g.node("QLinearConv", [p, w1, s1], [c1], x_scale=s, x_zp=0, y_scale=sy1, y_zp=0, pads=(0, 0, 0, 0), **conv)
    out = g.tensor("y", zb.F32, (N, 16, PH, PW))
    g.node("DequantizeLinear", [c1], [out], x_scale=sy1, x_zp=0)
    g.input, g.output = x, out
    xin = ((rng.random((N, C, H, W), dtype=np.float32) * 1.2 - (0.1 if dt == "U8" else 0.6)) * np.float32(scale * 255)).astype(np.float32)
    xin.reshape(-1)[:3] = [np.nan, np.inf, -np.inf]
    want = graph_oracle.run(oracle, g, xin)
    plan = zb.Plan(ctx, g)
    assert plan.step_names()[0].startswith("Fused[QuantizeLinear+QLinearConv"), plan.step_names()
    got = plan.run(xin)
    assert np.array_equal(plan.read_tensor(p), want[p])
    assert np.array_equal(got, want[out])
    assert len(np.unique(want[p])) > (16 if H > 2 else 4)
    plan.close()


@pytest.mark.parametrize("N,C,H,W,M,order,one", [
    (2, 3, 64, 64, 16, (0, 1), True),           # the result is the first part of a Concat's pixels, a convolution of it the other
    (2, 1, 34, 66, 48, (1, 0), True),           # it starts behind 16 channels
    (1, 4, 36, 70, 64, (1, 0), True),
    (230, 1, 28, 128, 32, (1, 0), True),
    (1, 1, 4, 12164, 16, (1, 0), False),        # a row is too wide: a conversion and the tcgen05 form
])
def test_result_inside_a_concat(zb, ctx, oracle, N, C, H, W, M, order, one):
    rng = np.random.default_rng(N + W)
    conv = dict(strides=(1, 1), dilations=(1, 1), group=1, auto_pad="NOTSET")
    g = zb.Graph("first")
    PH, PW = H // 2, W // 2
    x = g.tensor("x", zb.F32, (N, C, H, W))
    q = g.tensor("xq", zb.U8, (N, C, H, W))
    c = g.tensor("c", zb.I8, (N, M, H, W))
    a = g.tensor("a", zb.I8, (N, M, H, W))
    p = g.tensor("p", zb.I8, (N, M, PH, PW))
    c1 = g.tensor("c1", zb.I8, (N, 16, PH, PW))
    cat = g.tensor("cat", zb.I8, (N, M + 16, PH, PW))
    c2 = g.tensor("c2", zb.I8, (N, 16, PH, PW))
    out = g.tensor("y", zb.F32, (N, 16, PH, PW))
    sx = float(np.float32(1 / 255))
    sy, s1, s2 = (float(np.float32(v)) for v in (sx * 0.007 * 74 * 90 * np.sqrt(C * 9) / 40, 0.02 * np.sqrt(M), 0.05 * np.sqrt(M + 16)))

    def weights(name, m, k, r):
        return (g.tensor("w" + name, zb.I8, (m, k, r, r), rng.integers(-127, 128, (m, k, r, r), dtype=np.int8)),
                g.tensor("s" + name, zb.F32, (m,), (rng.random(m, dtype=np.float32) * 0.01 + 0.002).astype(np.float32)))

    g.node("QuantizeLinear", [x], [q], y_scale=sx, y_zp=0)
    g.node("QLinearConv", [q, *weights("0", M, C, 3)], [c], x_scale=sx, x_zp=0, y_scale=sy, y_zp=0, pads=(1, 1, 1, 1), **conv)
    g.node("LeakyRelu", [c], [a], alpha=0.1, x_scale=sy, x_zp=0, y_scale=sy, y_zp=0)
    g.node("MaxPool", [a], [p], **POOL)
    g.node("QLinearConv", [p, *weights("1", 16, M, 1)], [c1], x_scale=0.02, x_zp=0, y_scale=s1, y_zp=0, pads=(0, 0, 0, 0), **conv)
    g.node("Concat", [(p, c1)[i] for i in order], [cat], axis=1)
    g.node("QLinearConv", [cat, *weights("2", 16, M + 16, 1)], [c2], x_scale=0.02, x_zp=0, y_scale=s2, y_zp=0, pads=(0, 0, 0, 0), **conv)
    g.node("DequantizeLinear", [c2], [out], x_scale=s2, x_zp=0)
    g.input, g.output = x, out
    xin = (rng.random((N, C, H, W), dtype=np.float32) * 1.2 - 0.1).astype(np.float32)
    want = graph_oracle.run(oracle, g, xin)
    plan = zb.Plan(ctx, g)
    names = plan.step_names()
    assert names[0].startswith("Fused[QuantizeLinear+QLinearConv") == one and "Concat" not in names, names
    got = plan.run(xin)
    for t in (p, c1, cat):
        assert np.array_equal(plan.read_tensor(t), want[t]) and len(np.unique(want[t])) > 16
    assert np.array_equal(got, want[out])
    plan.close()
