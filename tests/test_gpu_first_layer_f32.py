"""FP32 first layers, 3x3 convolution of up to three channels with activation and 2x2 pool (conv3x3_pool_f32_lowc), bit for bit against the oracle."""
import numpy as np
import pytest

import graph_oracle

pytestmark = pytest.mark.gpu

CASES = [
    # N   C   H   W    M   pads          act
    (1, 1, 28, 28, 32, (0, 0, 0, 0), "Relu"),            # eight filters a thread
    (300, 1, 28, 28, 32, (0, 0, 0, 0), "Relu"),          # sixteen
    (1500, 1, 28, 28, 40, (0, 0, 0, 0), None),           # all
    (2, 3, 34, 30, 16, (1, 1, 1, 1), "LeakyRelu"),       # border of zeros
    (3, 2, 9, 13, 5, (1, 0, 0, 1), "Relu"),              # odd sizes, filters that are no whole eight, one-sided border
    (5, 3, 5, 5, 256, (0, 1, 1, 0), "LeakyRelu"),        # most filters
    (1, 1, 4, 4, 1, (0, 0, 0, 0), "Relu"),               # one pooled pixel, one filter
    (7, 3, 12, 300, 9, (1, 1, 1, 1), "Relu"),
]


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("case", CASES, ids=[f"first{i}" for i in range(len(CASES))])
def test_layer(zb, ctx, oracle, case, special):
    N, C, H, W, M, pads, act = case
    rng = np.random.default_rng(H + W + M)
    xin, wv, bv = (rng.standard_normal(s).astype(np.float32) for s in ((N, C, H, W), (M, C, 3, 3), (M,)))
    if special:                                          # zeros of both signs, infinities and NaNs, alone and together in a window
        flat = xin.reshape(-1)
        for i, v in enumerate((0.0, -0.0, np.inf, -np.inf, np.nan)):
            flat[rng.integers(0, flat.size, max(1, flat.size // 40))] = v
        wv.reshape(-1)[:2] = (0.0, -0.0)
        bv[0] = -0.0
    OH, OW = H + pads[0] + pads[2] - 2, W + pads[1] + pads[3] - 2
    g = zb.Graph("first")
    F32 = zb.F32
    x, w, b = g.tensor("x", F32, xin.shape), g.tensor("w", F32, wv.shape, wv), g.tensor("b", F32, (M,), bv)
    c = g.tensor("c", F32, (N, M, OH, OW))
    g.node("Conv", [x, w, b], [c], strides=(1, 1), pads=pads, dilations=(1, 1), group=1, auto_pad="NOTSET")
    if act:
        r = g.tensor("r", F32, (N, M, OH, OW))
        g.node(act, [c], [r], **(dict(alpha=0.1) if act == "LeakyRelu" else {}))
        c = r
    y = g.tensor("y", F32, (N, M, OH // 2, OW // 2))
    g.node("MaxPool", [c], [y], kernel_shape=(2, 2), strides=(2, 2), dilations=(1, 1), pads=(0, 0, 0, 0), auto_pad="NOTSET")
    g.input, g.output = x, y
    want = graph_oracle.run(oracle, g, xin)[y]
    plan = zb.Plan(ctx, g)
    assert len(plan.step_names()) == 1
    got = plan.run(xin)
    plan.close()
    assert np.array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    assert np.array_equal(got[ok].view(np.uint32), want[ok].view(np.uint32))
