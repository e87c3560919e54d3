"""A plan whose finalize failed can be finalized again, with or without fusion."""
import ctypes as C

import numpy as np
import pytest

import graph_oracle

pytestmark = pytest.mark.gpu
CONV = dict(strides=(1, 1), dilations=(1, 1), group=1, auto_pad="NOTSET", pads=(1, 1, 1, 1))


def declared(zb, ctx, graph):
    """A Plan before its finalize."""
    L = zb.lib()
    plan = zb.Plan.__new__(zb.Plan)
    plan.ctx, plan.graph, plan._h = ctx, graph, C.c_void_p(None)
    zb.check(L.zant_b200_plan_create(ctx._h, C.byref(plan._h)))
    for t in graph.tensors:
        sh, r = zb._sz(t["shape"])
        tid = C.c_int32(-1)
        zb.check(L.zant_b200_plan_tensor(plan._h, C.c_int32(t["dtype"]), sh, C.c_size_t(r), zb._ptr(t["data"]), C.byref(tid)))
    for n in graph.nodes:
        ins, outs = (C.c_int32 * len(n["inputs"]))(*n["inputs"]), (C.c_int32 * len(n["outputs"]))(*n["outputs"])
        a = zb._fill_attrs(n["attrs"])
        zb.check(L.zant_b200_plan_node(plan._h, C.c_int32(zb.OP[n["op"]]), ins, C.c_size_t(len(ins)), outs, C.c_size_t(len(outs)), C.byref(a)))
    for side in ("in", "out"):
        t = graph.tensors[graph.input if side == "in" else graph.output]
        setattr(plan, side + "_shape", t["shape"])
        setattr(plan, side + "_dtype", t["dtype"])
    return plan


def finalize(zb, plan, fuse):
    return zb.lib().zant_b200_plan_finalize(plan._h, C.c_int32(plan.graph.input), C.c_int32(plan.graph.output), C.c_int32(int(fuse)))


@pytest.mark.parametrize("first,second", [(True, False), (True, True), (False, True)])
def test_second_attempt(zb, ctx, oracle, first, second):
    rng = np.random.default_rng(0)
    N, H, W = 2, 18, 22
    g = zb.Graph("again")
    x, q = g.tensor("x", zb.F32, (N, 3, H, W)), g.tensor("q", zb.U8, (N, 3, H, W))
    g.node("QuantizeLinear", [x], [q], y_scale=1 / 255, y_zp=0)

    def conv(src, cin, name, M, sx, sy):
        w = g.tensor("w" + name, zb.I8, (M, cin, 3, 3), rng.integers(-127, 128, (M, cin, 3, 3), dtype=np.int8))
        s = g.tensor("s" + name, zb.F32, (1,), np.array([0.01], np.float32))
        c, r = g.tensor("c" + name, zb.I8, (N, M, H, W)), g.tensor("r" + name, zb.I8, (N, M, H, W))
        g.node("QLinearConv", [src, w, s], [c], x_scale=sx, x_zp=0, y_scale=sy, y_zp=0, **CONV)
        g.node("Relu", [c], [r], x_scale=sy, x_zp=0, y_scale=sy, y_zp=0)
        return r
    a, b = conv(q, 3, "a", 16, 1 / 255, 0.05), conv(q, 3, "b", 32, 1 / 255, 0.05)
    m = g.tensor("m", zb.I8, (N, 48, H, W))
    g.node("Concat", [a, b], [m], axis=1)                       # channels-last: its operands live in it
    c = conv(m, 48, "c", 16, 0.05, 1.0)
    f = g.tensor("f", zb.I8, (N, 16 * H * W))
    g.node("Reshape", [c], [f])
    y = g.tensor("y", zb.F32, (N, 16 * H * W))
    g.node("DequantizeLinear", [f], [y], x_scale=1.0, x_zp=0)
    g.input, g.output = x, y
    xin = rng.random((N, 3, H, W), dtype=np.float32)
    want = graph_oracle.run(oracle, g, xin)
    plan = declared(zb, ctx, g)
    try:
        zb.debug_fail_alloc(1)
        assert finalize(zb, plan, first) == -2                  # MemError
        zb.debug_fail_alloc(0)
        assert finalize(zb, plan, second) == 0
        assert np.array_equal(plan.run(xin), want[y])
        assert len(np.unique(want[y])) > 16
        if not second:
            for t in (a, b, m, c):
                assert np.array_equal(plan.read_tensor(t), want[t])
        fresh = zb.Plan(ctx, g, fuse=second)
        assert fresh.arena_bytes == plan.arena_bytes and fresh.step_names() == plan.step_names()
        fresh.close()
    finally:
        zb.debug_fail_alloc(0)
        plan.close()
