"""The quantisation that writes a first layer's pixels of 16 bytes (to_nhwc_small_k): inputs on both sides of every rounding step (the quotient is
computed without a division), both code types, zero points; planes that several images of a CTA share, and sizes that are multiples of nothing."""
import numpy as np
import pytest

import graph_oracle

pytestmark = pytest.mark.gpu


def _graph(zb, N, C, H, W, dtype, scale, zp):
    rng = np.random.default_rng(N + C + H + W)
    g = zb.Graph("first")
    x = g.tensor("x", zb.F32, (N, C, H, W))
    q = g.tensor("q", dtype, (N, C, H, W))
    g.node("QuantizeLinear", [x], [q], y_scale=scale, y_zp=zp)
    cur, cin, s, z = q, C, scale, zp
    for i, M in enumerate((16, 16)):                   # a first layer pays for the conversion in front of another channels-last layer
        w = g.tensor(f"w{i}", zb.I8, (M, cin, 1, 1), rng.integers(-127, 128, (M, cin, 1, 1), dtype=np.int8))
        ws = g.tensor(f"s{i}", zb.F32, (M,), rng.uniform(0.008, 0.012, M).astype(np.float32))
        y = g.tensor(f"y{i}", zb.I8, (N, M, H, W))
        sy = float(np.float32(s * 0.01 * 74 * 74 * np.sqrt(cin) / 40))
        g.node("QLinearConv", [cur, w, ws, -1, -1], [y], x_scale=s, x_zp=z, y_scale=sy, y_zp=0, pads=(0,) * 4, strides=(1, 1), dilations=(1, 1), group=1, auto_pad="NOTSET")
        cur, cin, s, z = y, M, sy, 0
    g.input, g.output = x, cur
    return g, q


@pytest.mark.parametrize("N,C,H,W", [(3, 3, 8, 8), (37, 1, 5, 7), (5, 4, 22, 23), (3, 2, 27, 19), (2, 3, 32, 32), (1, 3, 33, 31), (2, 2, 41, 25), (700, 1, 2, 3)])
@pytest.mark.parametrize("code,zp", [("U8", 0), ("U8", 131), ("I8", 0), ("I8", -7)])
@pytest.mark.parametrize("scale", [1.0 / 255.0, 0.3, 1.0e-31])
def test_steps(zb, ctx, oracle, N, C, H, W, code, zp, scale):
    s = float(np.float32(scale))
    lo, hi = (0, 255) if code == "U8" else (-128, 127)
    g, q = _graph(zb, N, C, H, W, getattr(zb, code), s, zp)
    v = ((np.arange(lo - zp - 2, hi - zp + 3, dtype=np.float64) + 0.5) * s).astype(np.float32)
    around = [v]
    up, dn = v, v
    for _ in range(3):
        up, dn = np.nextafter(up, np.float32(np.inf)), np.nextafter(dn, np.float32(-np.inf))
        around += [up, dn]
    pool = np.concatenate([np.array([np.inf, -np.inf, np.nan, 0.0, -0.0, 3.0e38, -3.0e38, 1.0e-45], np.float32)] + around)
    count = N * C * H * W
    rng = np.random.default_rng(count)
    x = np.resize(rng.permutation(pool) if count < pool.size else np.concatenate([pool, rng.choice(pool, count - pool.size)]), count)
    x = rng.permutation(x).astype(np.float32).reshape(N, C, H, W)
    want = graph_oracle.run(oracle, g, x)
    plan = zb.Plan(ctx, g, fuse=True)
    assert "QuantizeLinear" in plan.step_names() and sum("tc-implicit" in n for n in plan.step_names()) == 2
    got = plan.run(x)
    assert np.array_equal(plan.read_tensor(q), want[q])
    assert np.array_equal(got, want[g.output])
    plan.close()
