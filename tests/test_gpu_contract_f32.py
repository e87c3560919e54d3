"""FP32 contractions at the edges of their tiles, bit for bit against the oracle (one thread per sum, ascending k, separately
rounded multiply and add), alone and with what a plan fuses behind them."""
import numpy as np
import pytest

import graph_oracle

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


# few outputs; 32 x 32; 128 x {16, 32, 64, 128} tiles; K around a slab (16, 64)
@pytest.mark.parametrize("M,K,N", [(1, 1600, 512), (8, 64, 33), (9, 63, 31), (300, 17, 40), (4000, 9, 16), (4000, 15, 32), (5000, 33, 64),
                                   (2500, 48, 1030), (129, 1, 129), (1, 1, 1), (20000, 16, 3)])
def test_mat_mul(ctx, oracle, M, K, N):
    rng = np.random.default_rng(M + K + N)
    a, b = rng.standard_normal((M, K)).astype(np.float32), rng.standard_normal((K, N)).astype(np.float32)
    a[0, 0] = -0.0
    assert np.array_equal(bits(ctx.mat_mul(a, b)), bits(oracle.mat_mul(a, b)))


@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True), (True, True)])
def test_gemm_operand_orders(ctx, oracle, ta, tb):
    rng = np.random.default_rng(3)
    M, K, N = 260, 50, 70
    a = rng.standard_normal((1, 1, K, M) if ta else (1, 1, M, K)).astype(np.float32)
    b = rng.standard_normal((1, 1, N, K) if tb else (1, 1, K, N)).astype(np.float32)
    c = rng.standard_normal((1, 1, M, N)).astype(np.float32)
    assert np.array_equal(bits(ctx.gemm(a, b, c, 0.5, 1.5, ta, tb)), bits(oracle.gemm(a, b, c, 0.5, 1.5, ta, tb)))


CHAIN = [
    # N  C   H   W   M   k  pad act      pool
    (3, 1, 28, 28, 32, 3, 0, "Relu", True),        # K = 9: less than a slab; window members in one thread
    (2, 5, 11, 13, 64, 3, 1, "LeakyRelu", True),   # odd sizes: the last row and column are in no window
    (1, 7, 9, 9, 10, 3, 1, "Relu", True),          # few outputs: window members in four warps
    (40, 16, 13, 13, 130, 1, 0, None, True),
    (2, 3, 40, 37, 16, 5, 2, "Relu", False),
    (60, 8, 20, 20, 48, 3, 1, "LeakyRelu", False),
]


@pytest.mark.parametrize("case", CHAIN, ids=[f"chain{i}" for i in range(len(CHAIN))])
def test_conv_groups(zb, ctx, oracle, case):
    N, C, H, W, M, k, pad, act, pool = case
    rng = np.random.default_rng(C + M)
    g = zb.Graph("conv")
    F32 = zb.F32
    OH, OW = H + 2 * pad - k + 1, W + 2 * pad - k + 1
    x = g.tensor("x", F32, (N, C, H, W))
    w = g.tensor("w", F32, (M, C, k, k), rng.standard_normal((M, C, k, k)).astype(np.float32))
    b = g.tensor("b", F32, (M,), rng.standard_normal(M).astype(np.float32))
    cur = g.tensor("conv", F32, (N, M, OH, OW))
    g.node("Conv", [x, w, b], [cur], strides=(1, 1), pads=(pad,) * 4, dilations=(1, 1), group=1, auto_pad="NOTSET")
    if act:
        a = g.tensor("act", F32, (N, M, OH, OW))
        g.node(act, [cur], [a], alpha=0.1)
        cur = a
    if pool:
        p = g.tensor("pool", F32, (N, M, OH // 2, OW // 2))
        g.node("MaxPool", [cur], [p], kernel_shape=(2, 2), strides=(2, 2), dilations=(1, 1), pads=(0, 0, 0, 0), auto_pad="NOTSET")
        cur = p
    g.input, g.output = x, cur
    xin = rng.standard_normal((N, C, H, W)).astype(np.float32)
    want = graph_oracle.run(oracle, g, xin)[cur]
    plan = zb.Plan(ctx, g)
    assert len(plan.step_names()) == 1
    got = plan.run(xin)
    plan.close()
    assert np.array_equal(bits(got), bits(want))


@pytest.mark.parametrize("M,relu", [(1, True), (5, False), (700, True)])
def test_dense_group(zb, ctx, oracle, M, relu):
    rng = np.random.default_rng(M)
    g = zb.Graph("dense")
    F32 = zb.F32
    x = g.tensor("x", F32, (M, 50))
    w = g.tensor("w", F32, (50, 36), rng.standard_normal((50, 36)).astype(np.float32))
    b = g.tensor("b", F32, (36,), rng.standard_normal(36).astype(np.float32))
    m, a, r = (g.tensor(n, F32, (M, 36)) for n in ("m", "a", "r"))
    g.node("MatMul", [x, w], [m])
    g.node("Add", [m, b], [a])
    if relu:
        g.node("Relu", [a], [r])
    g.input, g.output = x, r if relu else a
    xin = rng.standard_normal((M, 50)).astype(np.float32)
    plan = zb.Plan(ctx, g)
    assert len(plan.step_names()) == 1
    got = plan.run(xin)
    plan.close()
    assert np.array_equal(bits(got), bits(graph_oracle.run(oracle, g, xin)[g.output]))
