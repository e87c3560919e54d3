"""Expand 1x1 -> depthwise 3x3 -> project 1x1 [-> residual addition] as one kernel (irb_q8.cuh) against the oracle, bit for bit."""
import numpy as np
import pytest

import graph_oracle

pytestmark = pytest.mark.gpu

CONV = dict(dilations=(1, 1), auto_pad="NOTSET")

# N C E M H W, input zero point, biases, residual addition: 0 none, 1 input first, 2 input second; stride; activation of the addition
CASES = [
    (9, 64, 384, 64, 14, 14, 0, True, 1, 1),        # whole chunks, one image a tile, both halves in one accumulator
    (160, 96, 576, 96, 14, 14, 0, False, 2, 1),     # half a chunk at the end, CTAs with two tiles
    (310, 32, 128, 32, 7, 7, 0, True, 1, 1),        # two images a tile, CTAs with two tiles, one chunk
    (17, 160, 960, 160, 7, 7, 0, True, 1, 1),       # two filter tiles, an odd image
    (16, 160, 960, 320, 7, 7, -3, True, 0, 1),      # three filter tiles, input zero point
    (8, 40, 200, 48, 14, 16, 2, True, 0, 1),
    (21, 24, 144, 24, 12, 9, 5, True, 1, 1),        # ragged width, K step partly empty
    (33, 40, 240, 112, 5, 16, -1, False, 0, 1),     # odd rows, halves apart
    (18, 32, 192, 32, 11, 13, 0, True, 2, 1),       # odd plane
    (40, 48, 288, 48, 3, 3, 0, True, 1, 1),
    (19, 64, 136, 16, 2, 5, 9, True, 0, 1),         # eight channels in the last chunk
    (150, 32, 256, 32, 10, 10, 0, True, 1, 1),
    (30, 64, 384, 64, 6, 8, 0, True, 1, 1),
    (17, 64, 384, 64, 8, 4, 0, True, 1, 1),
    (16, 32, 160, 32, 4, 6, 0, True, 1, 1),
    (12, 32, 160, 32, 8, 11, 0, True, 2, 1),
    (9, 16, 128, 16, 2, 12, 0, True, 1, 1),         # one output row a half
    (9, 96, 576, 160, 14, 14, 2, True, 0, 2),       # stride 2, two filter tiles
    (150, 32, 192, 64, 10, 10, 1, True, 0, 2),      # both halves in one accumulator, three and two output rows, CTAs with two tiles
    (20, 24, 144, 80, 12, 12, 3, False, 0, 2),      # the second half reads more rows than the first
    (11, 40, 130, 16, 4, 14, -4, True, 0, 2),
    (31, 48, 700, 48, 5, 5, 0, True, 1, 1),         # six chunks on six CTAs a tile, 60 channels in the last, an odd image
    (90, 64, 1100, 64, 4, 6, 0, True, 2, 1),        # nine chunks on three CTAs
    (160, 64, 384, 64, 14, 14, 0, True, 1, 1, "relu"),
    (31, 48, 700, 48, 5, 5, 0, True, 2, 1, "relu6"),
]

# Blocks that the kernel for many images takes (on 148 SMs): every width that it is instantiated for, images a tile, chunks, filter tiles.
ONE = [
    (53, 64, 384, 64, 14, 14, 0, True, 1, 1),       # whole chunks, one image a tile, both halves in one accumulator
    (160, 96, 576, 96, 14, 14, 0, False, 2, 1),     # half a chunk at the end, CTAs with two tiles
    (485, 32, 128, 32, 7, 7, 0, True, 1, 1),        # two images a tile, an odd image, CTAs with two tiles, one chunk
    (101, 160, 960, 160, 7, 7, 0, True, 1, 1),      # two filter tiles, an odd image
    (53, 160, 960, 320, 7, 7, -3, True, 0, 1),      # three filter tiles, input zero point
    (65, 40, 200, 48, 14, 16, 2, True, 0, 1),
    (61, 40, 240, 112, 5, 16, -1, False, 0, 1),     # odd rows, halves apart
    (1037, 64, 136, 16, 2, 5, 9, True, 0, 1),       # eight channels in the last chunk
    (179, 64, 384, 64, 6, 8, 0, True, 1, 1),
    (47, 96, 576, 160, 14, 14, 2, True, 0, 2),      # stride 2, two filter tiles
    (297, 24, 144, 160, 12, 12, 3, False, 0, 2),    # the second half reads more rows than the first
    (99, 24, 128, 16, 10, 10, 0, True, 0, 2),        # both halves in one accumulator
    (185, 48, 700, 48, 5, 5, 0, True, 1, 1),        # 60 channels in the last chunk, an odd image
    (221, 64, 1100, 64, 4, 6, 0, True, 2, 1),       # nine chunks
    (185, 48, 700, 48, 5, 5, 0, True, 2, 1, "relu6"),
    (1333, 40, 128, 8, 2, 4, 4, True, 0, 1),        # widths in the kernel's steps, without and with an addition
    (275, 8, 128, 8, 2, 3, 0, True, 1, 1),
    (221, 24, 128, 96, 3, 6, 0, True, 0, 1),
    (59, 80, 128, 80, 2, 5, 0, True, 2, 1),
    (445, 40, 128, 48, 2, 7, 0, True, 0, 1),
    (189, 12, 128, 12, 4, 7, 1, True, 1, 1),
    (445, 40, 128, 8, 3, 8, 0, False, 0, 1),
    (125, 8, 128, 8, 2, 8, 0, True, 1, 1),
    (115, 72, 128, 112, 6, 10, 0, True, 0, 1),
    (99, 80, 200, 80, 13, 9, 0, True, 1, 1),
    (125, 24, 384, 24, 13, 10, 0, True, 2, 1),
    (91, 24, 640, 256, 2, 12, 0, True, 0, 1),       # one output row a half
    (105, 32, 384, 32, 11, 12, 5, True, 1, 1),
    (75, 72, 128, 96, 4, 13, 0, True, 0, 1),
    (129, 80, 136, 80, 9, 14, 0, True, 1, 1),
    (125, 12, 128, 160, 2, 15, 0, True, 0, 1),
    (101, 80, 256, 80, 6, 15, 0, True, 1, 1),
    (127, 12, 256, 12, 11, 16, 0, True, 1, 1),      # an odd plane
]


def block(zb, case):
    """Graph up to the block's result `cur`, and the tensors t1, t2 between the convolutions."""
    N, C, E, M, H, W, xzp, bias, res, stride = case[:10]
    act = case[10] if len(case) > 10 else None
    OH, OW = (H + stride - 1) // stride, (W + stride - 1) // stride
    rng = np.random.default_rng(C + E + H * 16 + W)
    g = zb.Graph("irb")
    x0 = g.tensor("x", zb.I8, (N, 4, H, W))

    def conv(src, cin, cout, k, group, name, sx, zx, sy, zy, act, oh=H, ow=W, s=1):
        w = g.tensor("w" + name, zb.I8, (cout, cin // group, k, k), rng.integers(-127, 128, (cout, cin // group, k, k), dtype=np.int8))
        target = 60.0 * sy / (sx * 40.0 * 73.0 * np.sqrt(cin // group * k * k))        # outputs spread over the codes
        ws = g.tensor("s" + name, zb.F32, (cout,), (rng.uniform(0.7, 1.4, cout) * target).astype(np.float32))
        b = g.tensor("b" + name, zb.I32, (cout,), rng.integers(-3000, 3000, cout).astype(np.int32)) if bias else -1
        y = g.tensor("y" + name, zb.I8, (N, cout, oh, ow))
        g.node("QLinearConv", [src, w, ws, -1, b], [y], x_scale=sx, x_zp=zx, y_scale=sy, y_zp=zy, pads=(k // 2,) * 4, strides=(s, s), group=group, activation=act, **CONV)
        return y

    x = conv(x0, 4, C, 1, 1, "0", 0.05, 0, 0.1, xzp, None)
    six = float(np.float32(6.0) / np.float32(127.0))
    t1 = conv(x, C, E, 1, 1, "e", 0.1, xzp, six, 0, "relu6")
    t2 = conv(t1, E, E, 3, E, "d", six, 0, six, 0, "relu", OH, OW, stride)
    cur = conv(t2, E, M, 1, 1, "p", six, 0, 0.12, 0, None, OH, OW)
    if res:
        y = g.tensor("sum", zb.I8, (N, M, H, W))
        if res == 1:
            g.node("QLinearAdd", [x, cur], [y], x_scale=0.1, x_zp=xzp, b_scale=0.12, b_zp=0, y_scale=0.2, y_zp=2, activation=act)
        else:
            g.node("QLinearAdd", [cur, x], [y], x_scale=0.12, x_zp=0, b_scale=0.1, b_zp=xzp, y_scale=0.2, y_zp=0, activation=act)
        cur = y
    g.input = x0
    return g, t1, t2, cur, rng.integers(-128, 128, (N, 4, H, W)).astype(np.int8)


@pytest.mark.parametrize("case", CASES, ids=["x".join(map(str, c[:6] + c[9:])) for c in CASES])
def test_block(zb, ctx, oracle, case):
    g, t1, t2, cur, xv = block(zb, case)
    out = g.tensor("out", zb.F32, g.tensors[cur]["shape"])
    g.node("DequantizeLinear", [cur], [out], x_scale=0.2, x_zp=0)
    g.output = out
    want = graph_oracle.run(oracle, g, xv)
    plan = zb.Plan(ctx, g, fuse=True)
    assert any("expand+depthwise+project" in n for n in plan.step_names())
    for _ in range(2):
        assert np.array_equal(plan.run(xv), want[g.output])
    assert len(np.unique(want[t1])) > 30 and len(np.unique(want[t2])) > 20 and len(np.unique(want[cur])) > 30
    plan.close()


@pytest.mark.parametrize("case", ONE, ids=["x".join(map(str, c[:6] + c[9:])) for c in ONE])
def test_block_of_many_images(zb, ctx, oracle, case):
    g, t1, t2, cur, xv = block(zb, case)
    out = g.tensor("out", zb.F32, g.tensors[cur]["shape"])
    g.node("DequantizeLinear", [cur], [out], x_scale=0.2, x_zp=0)
    g.output = out
    want = graph_oracle.run(oracle, g, xv)
    plan = zb.Plan(ctx, g, fuse=True)
    assert any("expand+depthwise+project" in n for n in plan.step_names())
    ctx.selftest_give_up(0)                                  # (only the kernel on bands of rows would)
    for _ in range(2):
        assert np.array_equal(plan.run(xv), want[g.output])
    ctx.selftest_give_up(-1)
    assert len(np.unique(want[t1])) > 20 and len(np.unique(want[t2])) > 15 and len(np.unique(want[cur])) > 30
    plan.close()


@pytest.mark.parametrize("res", [0, 1])
def test_result_behind_a_reshape_is_the_output(zb, ctx, oracle, res):
    """The block's result is then the caller's buffer, which need not have the alignment that the kernel's stores want."""
    import torch
    case = (160, 64, 384, 64, 14, 14, 0, True, res, 1)
    g, t1, t2, cur, xv = block(zb, case)
    flat = g.tensor("flat", zb.I8, (160, 64 * 14 * 14))
    g.node("Reshape", [cur], [flat])
    g.output = flat
    want = graph_oracle.run(oracle, g, xv)[flat]
    plan = zb.Plan(ctx, g, fuse=True)
    steps = [n for n in plan.step_names() if "expand+depthwise+project" in n]
    assert not steps or (res and not steps[0].endswith("+QLinearAdd"))         # (the addition, a step of its own, takes any alignment)
    x = torch.from_numpy(xv).cuda()
    buf = torch.zeros(want.size + 64, dtype=torch.int8, device="cuda")
    for offset in (0, 32, 4, 1):
        y = buf[offset:offset + want.size].view(want.shape)
        try:
            plan.run(x, y)
        except zb.ZantError as e:
            assert e.name == "InvalidInput" and offset % 32 != 0
            continue
        ctx.synchronize()
        assert np.array_equal(y.cpu().numpy(), want)
    plan.close()


@pytest.mark.parametrize("case,ctas", [((31, 48, 700, 48, 5, 5, 0, True, 1, 1), 96), ((16, 160, 960, 320, 7, 7, -3, True, 0, 1), 64)])
@pytest.mark.parametrize("graph", [False, True])
def test_sums_are_clean_after_a_time_out(zb, oracle, case, ctas, graph):
    """A CTA that gives up half way through its additions reports a time-out in its run; the runs behind it are right."""
    ctx = zb.Context(0)
    g, t1, t2, cur, xv = block(zb, case)
    out = g.tensor("out", zb.F32, g.tensors[cur]["shape"])
    g.node("DequantizeLinear", [cur], [out], x_scale=0.2, x_zp=0)
    g.output = out
    want = graph_oracle.run(oracle, g, xv)[out]
    plan = zb.Plan(ctx, g, fuse=True)
    assert any("expand+depthwise+project" in n for n in plan.step_names())
    for cta in (0, 1, ctas // 2, ctas - 1):
        ctx.selftest_give_up(cta)
        if graph:
            plan.use_graph(True)                 # (the kernel that gives up is part of this graph)
        with pytest.raises(zb.ZantError) as e:
            plan.run(xv)
        assert e.value.name == "DeviceTimeout"
        if graph:
            plan.use_graph(True)
        for _ in range(2):
            assert np.array_equal(plan.run(xv), want)
    plan.close()
    ctx.close()


@pytest.mark.parametrize("case,ctas", [((64, 160, 960, 160, 7, 7, 0, True, 1, 1), 128),          # four chunks a CTA: weights that it stops fetching; pairs of CTAs
                                       ((148, 160, 960, 160, 4, 4, 0, True, 1, 1), 148)])        # four chunks, no cluster
@pytest.mark.parametrize("graph", [False, True])
def test_several_chunks_a_cta_and_a_time_out(zb, oracle, case, ctas, graph):
    """A CTA of the kernel on bands of rows gives up its first wait: a time-out in that run, once; the runs behind it are right."""
    test_sums_are_clean_after_a_time_out(zb, oracle, case, ctas, graph)
