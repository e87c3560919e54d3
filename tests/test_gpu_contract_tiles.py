"""Every tile shape of the FP32 contractions with ragged last tiles, bit for bit against the oracle: products and Gemm with transposed
operands, convolutions as calls, as plans (weights in slab order) and with the pool in the epilogue."""
import numpy as np
import pytest

import graph_oracle

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


MATS = [(4090, 70, 500), (2500, 9, 401), (5000, 13, 65), (40000, 9, 5), (2500, 17, 31), (700, 33, 130), (9, 63, 33), (2007, 129, 1)]


@pytest.mark.parametrize("M,K,N", MATS)
def test_products(ctx, oracle, M, K, N):
    rng = np.random.default_rng(M + N)
    a, b = rng.standard_normal((M, K)).astype(np.float32), rng.standard_normal((K, N)).astype(np.float32)
    want = oracle.mat_mul(a, b)
    assert np.array_equal(bits(ctx.mat_mul(a, b)), bits(want))
    for ta, tb in ((False, True), (True, False)):
        got = ctx.gemm((a.T if ta else a)[None, None].copy(), (b.T if tb else b)[None, None].copy(), None, 1.0, 1.0, ta, tb)
        assert np.array_equal(bits(got[0, 0]), bits(want)), (ta, tb)


CONVS = [
    # N   C   H   W   M   k
    (21, 17, 30, 30, 127, 3),       # 128 x 128
    (30, 9, 18, 15, 123, 3),        # 128 x 64
    (40, 16, 13, 13, 130, 1),       # 128 x 64 with the pool
    (12, 2, 22, 22, 66, 3),         # 128 x 32
    (40, 1, 20, 21, 6, 3),          # 128 x 16
    (11, 1, 43, 20, 131, 3),
    (50, 3, 16, 17, 19, 3),         # 32 x 32
    (7, 4, 13, 11, 5, 3),           # few outputs
]


@pytest.mark.parametrize("case", CONVS, ids=[f"conv{i}" for i in range(len(CONVS))])
@pytest.mark.parametrize("pool", [False, True])
def test_convolutions(zb, ctx, oracle, case, pool):
    N, C, H, W, M, k = case
    rng = np.random.default_rng(C + M)
    OH, OW = H - k + 1, W - k + 1
    attrs = dict(strides=(1, 1), pads=(0, 0, 0, 0), dilations=(1, 1), group=1, auto_pad="NOTSET")
    g = zb.Graph("tiles")
    F32 = zb.F32
    xin, wv, bv = (rng.standard_normal(s).astype(np.float32) for s in ((N, C, H, W), (M, C, k, k), (M,)))
    x, w, b = g.tensor("x", F32, xin.shape), g.tensor("w", F32, wv.shape, wv), g.tensor("b", F32, (M,), bv)
    c = y = g.tensor("c", F32, (N, M, OH, OW))
    g.node("Conv", [x, w, b], [c], **attrs)
    if pool:
        y = g.tensor("p", F32, (N, M, OH // 2, OW // 2))
        g.node("MaxPool", [c], [y], kernel_shape=(2, 2), strides=(2, 2), dilations=(1, 1), pads=(0, 0, 0, 0), auto_pad="NOTSET")
    g.input, g.output = x, y
    want = graph_oracle.run(oracle, g, xin)
    plan = zb.Plan(ctx, g)
    assert len(plan.step_names()) == 1
    got = plan.run(xin)
    plan.close()
    assert np.array_equal(bits(got), bits(want[y]))
    if not pool:
        got = ctx.conv_lean(xin, wv, (N, M, OH, OW), bias=bv, stride=(1, 1), pads=(0, 0, 0, 0), dilations=(1, 1), group=1, auto_pad="NOTSET")
        assert np.array_equal(bits(got), bits(want[c]))
