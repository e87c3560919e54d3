"""Weights of few-position QLinearConv / QLinearMatMul: put in fragment order on the device, in calls and in plans."""
import time

import numpy as np
import pytest

import graph_oracle

pytestmark = pytest.mark.gpu
CONV = dict(strides=(1, 1), dilations=(1, 1), group=1, auto_pad="NOTSET")


def test_call_does_not_pay_for_a_shuffle_on_the_host(ctx):
    """8 rows against 256 (whose weights another kernel blocks): about the same time, the upload of the matrix.  The host took 10
    times as long to shuffle it."""
    rng = np.random.default_rng(0)
    b = rng.integers(-127, 128, (4096, 4096), dtype=np.int8)

    def best(M):
        a = rng.integers(-128, 128, (M, 4096), dtype=np.int8)
        t = []
        for _ in range(8):
            t0 = time.perf_counter()
            ctx.qlinearmatmul(a, 0.02, 0, b, [0.01], None, 1.0, 0)
            t.append(time.perf_counter() - t0)
        return min(t)
    many = best(256)
    assert best(8) < 4 * many


# channels, filters and plane around the 32-channel steps, 16-filter tiles and load paths; K of the product behind the convolution
@pytest.mark.parametrize("N,C,H,M,k,xzp,NC,bias", [(1, 33, 7, 17, 3, 5, 10, True), (1, 64, 14, 48, 1, -3, 33, False), (7, 31, 3, 16, 1, 128, 100, True), (2, 3, 9, 40, 5, 0, 7, False)])
def test_plan(zb, ctx, oracle, N, C, H, M, k, xzp, NC, bias):
    rng = np.random.default_rng(C + M)
    U8 = xzp == 128
    g = zb.Graph("few")
    x = g.tensor("x", zb.U8 if U8 else zb.I8, (N, C, H, H))
    w = g.tensor("w", zb.I8, (M, C, k, k), rng.integers(-127, 128, (M, C, k, k), dtype=np.int8))
    ws = g.tensor("ws", zb.F32, (M,), (rng.random(M, dtype=np.float32) * 0.01 + 0.002).astype(np.float32))
    b = g.tensor("b", zb.I32, (M,), rng.integers(-3000, 3000, M).astype(np.int32)) if bias else -1
    c = g.tensor("c", zb.I8, (N, M, H, H))
    sy = float(np.float32(0.02 * 0.007 * 74 * 74 * np.sqrt(C * k * k) / 45))
    g.node("QLinearConv", [x, w, ws, -1, b], [c], x_scale=0.02, x_zp=xzp, y_scale=sy, y_zp=xzp // 4, pads=(k // 2,) * 4, **CONV)
    K = M * H * H
    f = g.tensor("f", zb.I8, (N, K))
    g.node("Reshape", [c], [f])
    w2 = g.tensor("w2", zb.I8, (K, NC), rng.integers(-127, 128, (K, NC), dtype=np.int8))
    ws2 = g.tensor("ws2", zb.F32, (1,), np.array([0.01], np.float32))
    b2 = g.tensor("b2", zb.I32, (NC,), rng.integers(-3000, 3000, NC).astype(np.int32)) if bias else -1
    m = g.tensor("m", zb.I8, (N, NC))
    g.node("QLinearMatMul", [f, w2, ws2, -1, b2], [m], x_scale=sy, x_zp=xzp // 4, y_scale=float(np.float32(sy * 0.01 * 74 * np.sqrt(K))), y_zp=1)
    g.input, g.output = x, m
    xin = rng.integers(0, 256, (N, C, H, H)).astype(np.uint8) if U8 else rng.integers(-128, 128, (N, C, H, H)).astype(np.int8)
    want = graph_oracle.run(oracle, g, xin)
    plan = zb.Plan(ctx, g)
    assert np.array_equal(plan.run(xin), want[m])
    assert np.array_equal(plan.read_tensor(c), want[c])
    plan.close()
