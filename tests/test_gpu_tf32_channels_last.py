"""The TF32 forms of the channels-last kernel on real-valued data, against the same network in 64 bits.

Bound: an operand rounded to TF32 is off by at most 2^-11 of itself, independently of the others, so the output of a layer by about
2^-11 * sqrt(2 / 3) of its 2-norm (weights and activations), and what a layer in front of it brought; three layers: 2^-11 * sqrt(2) = 7e-4.
Split operands leave 2^-22 and the fp32 accumulation, whose truncated additions dominate: 1e-4 with a wide margin."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CONV = dict(strides=(1, 1), dilations=(1, 1), group=1, auto_pad="NOTSET")
POOL = dict(kernel_shape=(2, 2), strides=(2, 2), dilations=(1, 1), pads=(0, 0, 0, 0), auto_pad="NOTSET")


@pytest.mark.parametrize("mode,bound", [(1, 7e-4), (2, 1e-4)])
@pytest.mark.parametrize("N,C,H,W,M1,M2,M3,k", [(2, 3, 28, 20, 16, 48, 33, 3), (1, 4, 26, 34, 64, 256, 80, 3), (3, 2, 17, 19, 32, 512, 16, 1)])
def test_against_64_bits(zb, mode, bound, N, C, H, W, M1, M2, M3, k):
    import torch
    import torch.nn.functional as F
    rng = np.random.default_rng(M1 + M2)
    g = zb.Graph("real")
    x = g.tensor("x", zb.F32, (N, C, H, W))
    xin = rng.standard_normal((N, C, H, W)).astype(np.float32)
    cur, ref, cin = x, torch.from_numpy(xin).double(), C
    pool = H % 2 == 0 and W % 2 == 0
    for i, M in enumerate((M1, M2, M3)):
        wv = (rng.standard_normal((M, cin, k, k)) / np.sqrt(cin * k * k)).astype(np.float32)
        bv = rng.standard_normal(M).astype(np.float32)
        w, b = g.tensor(f"w{i}", zb.F32, wv.shape, wv), g.tensor(f"b{i}", zb.F32, (M,), bv)
        c = g.tensor(f"c{i}", zb.F32, (N, M, H, W))
        g.node("Conv", [cur, w, b], [c], pads=(k // 2,) * 4, **CONV)
        ref = F.conv2d(ref, torch.from_numpy(wv).double(), torch.from_numpy(bv).double(), padding=k // 2)
        cur, cin = c, M
        if i < 2:
            r = g.tensor(f"r{i}", zb.F32, (N, M, H, W))
            g.node("LeakyRelu", [cur], [r], alpha=0.125)
            ref = torch.where(ref <= 0, ref * 0.125, ref)
            cur = r
        if i == 0 and pool:
            H, W = H // 2, W // 2
            p = g.tensor("p", zb.F32, (N, M, H, W))
            g.node("MaxPool", [cur], [p], **POOL)
            ref = F.max_pool2d(ref, 2)
            cur = p
    g.input, g.output = x, cur
    ctx = zb.Context(0)
    ctx.set_tf32(mode)
    plan = zb.Plan(ctx, g)
    assert sum("tf32" in n for n in plan.step_names()) >= 3
    got = plan.run(xin)
    again = plan.run(xin)
    plan.close()
    ctx.close()
    err = float(np.linalg.norm(got - ref.numpy()) / ref.norm())
    assert 0 < err < bound
    assert np.array_equal(got.view(np.uint32), again.view(np.uint32))      # repeats itself exactly
