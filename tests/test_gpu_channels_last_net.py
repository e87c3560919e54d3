"""Convolutions between channels-last activations of a plan (tc_nhwc_net.cuh): tile edges, filter and channel remainders, fused
pool, Resize by two, Concat written in place, first layers.  int8 bit for bit against the oracle; the TF32 forms on small
integers, for which every product, sum and rounding to TF32 is exact, so they too have to agree bit for bit."""
import numpy as np
import pytest

import graph_oracle

pytestmark = pytest.mark.gpu

CONV = dict(strides=(1, 1), dilations=(1, 1), group=1, auto_pad="NOTSET")
POOL = dict(kernel_shape=(2, 2), strides=(2, 2), dilations=(1, 1), pads=(0, 0, 0, 0), auto_pad="NOTSET")

CASES = [
    # N  C0  H   W   [layers: (filters, kernel, activation, pool)]; the last layer leaves as NCHW
    (2, 3, 20, 28, [(16, 3, "leaky", 2), (32, 3, "leaky", 2), (48, 3, None, 0)]),       # pooled views: 16 and 32 filters, 16-byte pixels
    (1, 1, 26, 26, [(64, 3, "relu", 2), (80, 1, "relu", 0), (7, 3, None, 0)]),          # pooled pairs; ragged filters out
    (1, 4, 13, 13, [(160, 3, "leaky", 0), (272, 3, "leaky", 1), (33, 1, None, 0)]),     # two and three filter tiles, stride-1 pool
    (2, 2, 6, 150, [(16, 5, None, 0), (16, 3, "relu", 2), (255, 1, None, 0)]),          # two column segments; 16 -> 16 (pairs of taps)
    (3, 3, 8, 4, [(32, 1, "relu", 0), (96, 3, None, 0)]),                               # tiny images, a tile of mostly dead rows
    (1, 3, 52, 52, [(128, 3, "leaky", 2), (512, 3, "leaky", 0), (64, 3, None, 0)]),     # streamed weights, several channel stages
    (2, 3, 18, 22, [(96, 3, "clip", 2), (24, 3, None, 0)]),                             # 96 filters: a pool in 64-filter tiles; 24 stay NCHW
]


def first_layer_int8(g, zb, N, C, H, W):
    x = g.tensor("x", zb.F32, (N, C, H, W))
    q = g.tensor("xq", zb.U8, (N, C, H, W))
    g.node("QuantizeLinear", [x], [q], y_scale=float(np.float32(1 / 255)), y_zp=0)
    return x, q


@pytest.mark.parametrize("case", CASES, ids=[f"net{i}" for i in range(len(CASES))])
def test_int8_chain(zb, ctx, oracle, case):
    N, C, H, W, layers = case
    rng = np.random.default_rng(C + H + W)
    g = zb.Graph("net")
    x, cur = first_layer_int8(g, zb, N, C, H, W)
    s = float(np.float32(1 / 255))
    cin = C
    for li, (M, k, act, pool) in enumerate(layers):
        w = g.tensor(f"w{li}", zb.I8, (M, cin, k, k), rng.integers(-127, 128, (M, cin, k, k), dtype=np.int8))
        ws = g.tensor(f"s{li}", zb.F32, (M,), (rng.random(M, dtype=np.float32) * 0.01 + 0.002).astype(np.float32))
        b = g.tensor(f"b{li}", zb.I32, (M,), rng.integers(-3000, 3000, M).astype(np.int32))
        y = g.tensor(f"c{li}", zb.I8, (N, M, H, W))
        sy = float(np.float32(s * 0.007 * 74 * (90 if li == 0 else 40) * np.sqrt(cin * k * k) / 40))
        p = k // 2
        g.node("QLinearConv", [cur, w, ws, -1, b], [y], x_scale=s, x_zp=0, y_scale=sy, y_zp=0, pads=(p,) * 4, **CONV)
        cur, s, cin = y, sy, M
        if act:
            a = g.tensor(f"a{li}", zb.I8, (N, M, H, W))
            if act == "relu":
                g.node("Relu", [cur], [a], x_scale=s, x_zp=0, y_scale=s, y_zp=0)
            elif act == "leaky":
                g.node("LeakyRelu", [cur], [a], alpha=0.1, x_scale=s, x_zp=0, y_scale=s * 0.8, y_zp=0)
                s *= 0.8
            else:
                g.node("Clip", [cur], [a], alpha=0.0, beta=float(s * 60), x_scale=s, x_zp=0, y_scale=s, y_zp=0)
            cur = a
        if pool == 2:
            H, W = H // 2, W // 2
            o = g.tensor(f"p{li}", zb.I8, (N, M, H, W))
            g.node("MaxPool", [cur], [o], **POOL)
            cur = o
        elif pool == 1:
            o = g.tensor(f"p{li}", zb.I8, (N, M, H, W))
            g.node("MaxPool", [cur], [o], kernel_shape=(2, 2), strides=(1, 1), dilations=(1, 1), pads=(0, 0, 0, 0), auto_pad="SAME_UPPER")
            cur = o
    y = g.tensor("y", zb.F32, (N, cin, H, W))
    g.node("DequantizeLinear", [cur], [y], x_scale=s, x_zp=0)
    g.input, g.output = x, y
    xin = rng.random((N, C, case[2], case[3]), dtype=np.float32)
    want = graph_oracle.run(oracle, g, xin)
    plan = zb.Plan(ctx, g)
    names = plan.step_names()
    got = plan.run(xin)
    assert np.array_equal(got, want[y]), names
    assert len(np.unique(want[y])) > 16
    # a tensor kept channels-last reads back in the graph's order
    for t in range(len(g.tensors)):
        if g.tensors[t]["data"] is None and g.tensors[t]["dtype"] == zb.I8:
            try:
                arr = plan.read_tensor(t)
            except zb.ZantError as e:
                assert e.name == "Unsupported"
                continue
            assert np.array_equal(arr, want[t]), g.tensors[t]["name"]
    plan.close()


def tf32_net(zb, rng, N, C, H, W, M1, M2, k, pool, up, cat):
    """Small integers throughout: |x| <= 2, |w| <= 1 on a few taps, so that layer 1 stays below 2048 in magnitude."""
    g = zb.Graph("tf32")
    F32 = zb.F32

    def weights(m, c):
        w = np.zeros((m, c, k, k), np.float32)
        for i in range(m):
            for _ in range(40):
                w[i, rng.integers(c), rng.integers(k), rng.integers(k)] = rng.integers(-2, 3)
        return w
    x = g.tensor("x", F32, (N, C, H, W))
    w1 = g.tensor("w1", F32, (M1, C, k, k), weights(M1, C)); b1 = g.tensor("b1", F32, (M1,), rng.integers(-9, 10, M1).astype(np.float32))
    c1 = g.tensor("c1", F32, (N, M1, H, W)); r1 = g.tensor("r1", F32, (N, M1, H, W))
    p = k // 2
    g.node("Conv", [x, w1, b1], [c1], pads=(p,) * 4, **CONV)
    g.node("Relu", [c1], [r1])
    cur = r1
    if pool:
        H, W = H // 2, W // 2
        o = g.tensor("p1", F32, (N, M1, H, W))
        g.node("MaxPool", [cur], [o], **POOL)
        cur = o
    cin = M1
    if cat:
        w3 = g.tensor("w3", F32, (M2, M1, k, k), np.sign(weights(M2, M1)) * 0.25)
        c3 = g.tensor("c3", F32, (N, M2, H, W)); r3 = g.tensor("r3", F32, (N, M2, H, W))
        g.node("Conv", [cur, w3], [c3], pads=(p,) * 4, **CONV)
        g.node("LeakyRelu", [c3], [r3], alpha=0.5)
        side = r3
        if up:
            H, W = 2 * H, 2 * W
            u = g.tensor("u", F32, (N, M2, H, W))
            g.node("Resize", [r3], [u], scales=(1.0, 1.0, 2.0, 2.0), coord_mode="half_pixel")
            side, main = u, r1
        else:
            main = cur
        m = g.tensor("m", F32, (N, M2 + M1, H, W))
        g.node("Concat", [side, main], [m], axis=1)
        cur, cin = m, M1 + M2
    w2 = g.tensor("w2", F32, (M2, cin, k, k), weights(M2, cin))
    y = g.tensor("y", F32, (N, M2, H, W))
    g.node("Conv", [cur, w2], [y], pads=(p,) * 4, **CONV)
    g.input, g.output = x, y
    return g, rng.integers(-2, 3, (N, C, case_h(g, x), case_w(g, x))).astype(np.float32)


def case_h(g, x):
    return g.tensors[x]["shape"][2]


def case_w(g, x):
    return g.tensors[x]["shape"][3]


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("N,C,H,W,M1,M2,k,pool,up,cat", [
    (2, 3, 20, 28, 16, 32, 3, True, False, False),
    (1, 4, 26, 26, 64, 48, 3, True, True, True),        # upsampled and concatenated in place
    (1, 3, 13, 17, 32, 144, 3, False, False, True),
    (1, 2, 30, 12, 48, 16, 1, False, False, False),
    (2, 1, 10, 140, 16, 16, 5, False, False, False),    # two column segments
])
def test_tf32_exact_on_integers(zb, oracle, mode, N, C, H, W, M1, M2, k, pool, up, cat):
    rng = np.random.default_rng(H + W + M1)
    g, xin = tf32_net(zb, rng, N, C, H, W, M1, M2, k, pool, up, cat)
    want = graph_oracle.run(oracle, g, xin)
    assert all(np.abs(want[g.id_of(n)]).max() < 2048 for n in ("r1",))
    c = zb.Context(0)
    c.set_tf32(mode)
    plan = zb.Plan(c, g)
    names = plan.step_names()
    assert any("tf32" in n for n in names) and "Resize" not in names and "Concat" not in names, names
    assert ("MaxPool" in names) == (pool and up), names          # with `up` the unpooled tensor has a second reader
    assert np.array_equal(plan.run(xin), want[g.output]), names
    plan.close()
    c.close()
