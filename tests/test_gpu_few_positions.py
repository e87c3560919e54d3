"""QLinearConv / QLinearMatMul with fewer than 256 output positions (warp-level MMAs, K split over warps), bit for bit against
the oracle: every load path, remainders of the 16-filter, 32-position and 32-channel tiles, both activation types."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
I8, U8 = 1, 2


def codes(rng, shape, dt):
    return rng.integers(0, 256, shape, dtype=np.uint8) if dt == U8 else rng.integers(-128, 128, shape, dtype=np.int8)


CONV = [
    # N  C    H   W   M    k  s  p  d  xdt ydt xzp yzp act
    (1, 960, 7, 7, 160, 1, 1, 0, 1, I8, I8, 0, 0, None),          # byte path, K deep enough for eight warps
    (1, 64, 14, 14, 384, 1, 1, 0, 1, I8, I8, 0, 0, "relu6"),      # word path
    (3, 33, 4, 5, 17, 1, 1, 0, 1, U8, I8, 128, 0, "relu"),        # ragged channels, filters and positions
    (1, 8, 15, 17, 600, 1, 1, 0, 1, I8, U8, -5, 9, None),         # 255 positions, 32 filters per CTA
    (2, 20, 9, 9, 12, 3, 2, 1, 1, U8, U8, 7, 3, "relu"),          # padding and stride
    (1, 5, 11, 13, 33, 5, 1, 2, 1, I8, I8, 3, 0, "relu"),         # 5x5
    (1, 40, 10, 10, 16, 3, 1, 2, 2, I8, I8, 0, 0, None),          # dilation
    (200, 70, 1, 1, 19, 1, 1, 0, 1, I8, I8, -4, 0, None),         # planes of one pixel
    (1, 1, 1, 1, 1, 1, 1, 0, 1, I8, I8, 0, 0, None),
]


@pytest.mark.parametrize("case", CONV, ids=[f"few{i}" for i in range(len(CONV))])
def test_qlinearconv_few_positions(zb, ctx, oracle, case):
    N, C, H, W, M, k, s, p, d, xdt, ydt, xzp, yzp, act = case
    rng = np.random.default_rng(C + M)
    x = codes(rng, (N, C, H, W), xdt)
    w = rng.integers(-127, 128, (M, C, k, k), dtype=np.int8)
    ws = (rng.random(M, dtype=np.float32) * 0.02 + 0.001).astype(np.float32)
    bias = rng.integers(-2000, 2000, M).astype(np.int32)
    args = (x, 0.02, xzp, w, ws, None, float(np.float32(0.02 * np.sqrt(C * k * k))), yzp)
    kw = dict(bias=bias, y_dtype=ydt, stride=(s, s), pads=(p,) * 4, dilations=(d, d), activation=act)
    want = oracle.qlinearconv(*args, **kw)
    assert np.array_equal(ctx.qlinearconv(*args, **kw), want)
    # device buffers that are not word aligned: the word path gives way to byte loads
    import torch
    xd = torch.empty(x.size + 1, dtype=torch.uint8 if xdt == U8 else torch.int8, device="cuda")[1:].view(x.shape)
    yd = torch.empty(want.size + 1, dtype=torch.uint8 if ydt == U8 else torch.int8, device="cuda")[1:].view(want.shape)
    xd.copy_(torch.from_numpy(x))
    torch.cuda.synchronize()
    ctx.qlinearconv(xd, *args[1:], out=yd, **kw)
    ctx.synchronize()
    assert np.array_equal(yd.cpu().numpy(), want)


@pytest.mark.parametrize("M,K,N,adt,azp", [(1, 1280, 1000, I8, 0), (37, 1280, 1000, I8, 0), (255, 63, 10, U8, 128), (33, 100, 65, I8, -3), (1, 1, 1, I8, 0)])
def test_qlinearmatmul_few_rows(ctx, oracle, M, K, N, adt, azp):
    rng = np.random.default_rng(M + K)
    a = codes(rng, (M, K), adt)
    b = rng.integers(-127, 128, (K, N), dtype=np.int8)
    bs = (rng.random(N, dtype=np.float32) * 0.02 + 0.001).astype(np.float32)
    bias = rng.integers(-2000, 2000, N).astype(np.int32)
    args = (a, 0.02, azp, b, bs, None, float(np.float32(0.02 * np.sqrt(K))), 0)
    assert np.array_equal(ctx.qlinearmatmul(*args, bias=bias), oracle.qlinearmatmul(*args, bias=bias))
