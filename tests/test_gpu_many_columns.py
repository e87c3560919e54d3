"""FP32 contractions with more columns than 65535 blocks of the narrow tiles cover (32 columns: 2 097 120)."""
import numpy as np
import pytest

import graph_oracle

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


@pytest.mark.parametrize("M,K,N", [(1, 2, 2097120), (1, 2, 2097121), (3, 1, 4194240), (40, 1, 2097121)])
def test_mat_mul(ctx, oracle, M, K, N):
    rng = np.random.default_rng(N)
    a, b = rng.standard_normal((M, K)).astype(np.float32), rng.standard_normal((K, N)).astype(np.float32)
    assert np.array_equal(bits(ctx.mat_mul(a, b)), bits(oracle.mat_mul(a, b)))


def test_conv_in_a_plan(zb, ctx, oracle):
    M = 2097121
    rng = np.random.default_rng(0)
    g = zb.Graph("wide")
    x = g.tensor("x", zb.F32, (1, 1, 1, 2))
    w = g.tensor("w", zb.F32, (M, 1, 1, 1), rng.standard_normal((M, 1, 1, 1)).astype(np.float32))
    y = g.tensor("y", zb.F32, (1, M, 1, 2))
    g.node("Conv", [x, w], [y], strides=(1, 1), pads=(0, 0, 0, 0), dilations=(1, 1), group=1, auto_pad="NOTSET")
    g.input, g.output = x, y
    xin = rng.standard_normal((1, 1, 1, 2)).astype(np.float32)
    plan = zb.Plan(ctx, g)
    got = plan.run(xin)
    plan.close()
    assert np.array_equal(bits(got), bits(graph_oracle.run(oracle, g, xin)[y]))
