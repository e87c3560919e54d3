"""zant_b200_plan_tensor_ptr: the buffer holds the tensor in the graph's order, whatever layout the plan keeps it in."""
import ctypes as C

import numpy as np
import pytest

import graph_oracle
from test_gpu_channels_last_net import CONV, first_layer_int8, tf32_net

pytestmark = pytest.mark.gpu


def contents(zb, plan, tid):
    import torch
    t = plan.graph.tensors[tid]
    p = zb.lib().zant_b200_plan_tensor_ptr(plan._h, C.c_int32(tid))
    if p is None:
        return None
    plan.ctx.synchronize()

    class Buffer:
        __cuda_array_interface__ = dict(shape=tuple(t["shape"]), typestr=np.dtype(zb.NP_DTYPE[t["dtype"]]).str, data=(p, False), version=3)
    return torch.as_tensor(Buffer(), device="cuda").cpu().numpy()


@pytest.mark.parametrize("graph", [False, True])
def test_int8(zb, ctx, oracle, graph):
    rng = np.random.default_rng(0)
    g = zb.Graph("net")
    N, H, W = 2, 20, 28
    x, q = first_layer_int8(g, zb, N, 3, H, W)

    def conv(src, cin, M, name, sx, sy):
        w = g.tensor("w" + name, zb.I8, (M, cin, 3, 3), rng.integers(-127, 128, (M, cin, 3, 3), dtype=np.int8))
        s = g.tensor("s" + name, zb.F32, (1,), np.array([0.01], np.float32))
        c = g.tensor("c" + name, zb.I8, (N, M, H, W))
        g.node("QLinearConv", [src, w, s], [c], x_scale=sx, x_zp=0, y_scale=sy, y_zp=0, pads=(1,) * 4, **CONV)
        return c
    a, b = conv(q, 3, 16, "a", 1 / 255, 0.05), conv(q, 3, 32, "b", 1 / 255, 0.05)
    m = g.tensor("m", zb.I8, (N, 48, H, W))
    g.node("Concat", [a, b], [m], axis=1)
    c = conv(m, 48, 16, "c", 0.05, 1.0)
    y = g.tensor("y", zb.F32, (N, 16, H, W))
    g.node("DequantizeLinear", [c], [y], x_scale=1.0, x_zp=0)
    g.input, g.output = x, y
    plan = zb.Plan(ctx, g)
    if graph:
        plan.use_graph()
    launches = plan.launches_per_run
    for i in range(3):
        xin = rng.random((N, 3, H, W), dtype=np.float32)
        want = graph_oracle.run(oracle, g, xin)
        assert np.array_equal(plan.run(xin), want[y])
        for t in (q, a, b, m):
            assert np.array_equal(contents(zb, plan, t), want[t]), (i, g.tensors[t]["name"])
        assert contents(zb, plan, c) is None                    # dequantised in the convolution's own step
    assert plan.launches_per_run == launches
    plan.close()


@pytest.mark.parametrize("mode", [1, 2])
def test_tf32(zb, oracle, mode):
    rng = np.random.default_rng(mode)
    g, xin = tf32_net(zb, rng, 1, 4, 26, 26, 64, 48, 3, True, True, True)
    want = graph_oracle.run(oracle, g, xin)
    ctx = zb.Context(0)
    ctx.set_tf32(mode)
    plan = zb.Plan(ctx, g)
    plan.run(xin)
    for name in ("r1", "p1", "m"):
        t = g.id_of(name)
        got = contents(zb, plan, t)
        assert np.array_equal(got, want[t]) and np.array_equal(got, plan.read_tensor(t)), name
    plan.close()
    ctx.close()
