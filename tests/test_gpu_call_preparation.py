"""What a channels-last QLinearConv call prepares on the device in one launch (nh_prep_k): inputs on the device at any word, last words of a tensor that is
not whole words, channel tiles that end inside 16, pixel tiles of one pixel and more, folded biases."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
I8 = 1

# N C H W M k s pad, input zero point (uint8 where it is not 0), words in front of the input
CASES = [
    (1, 17, 3, 129, 20, 3, 1, 1, 0, 1),            # 387 pixels: three tiles and three pixels; an odd number of bytes
    (3, 1, 11, 13, 33, 3, 1, 1, 0, 3),             # one channel
    (2, 65, 16, 16, 40, 1, 2, 0, 128, 1),          # a second tile of one channel; bias folded
    (257, 129, 1, 1, 18, 1, 1, 0, 7, 2),           # planes of one pixel
    (5, 80, 9, 15, 512, 3, 2, 1, 0, 5),            # many blocks of weights
    (4, 48, 8, 16, 90, 3, 1, 0, 9, 0),             # whole words and tiles
]


@pytest.mark.parametrize("case", CASES, ids=[f"prep{i}" for i in range(len(CASES))])
def test_device_input(ctx, oracle, case):
    import torch
    N, C, H, W, M, k, s, pad, zp, words = case
    rng = np.random.default_rng(C + H + W + M)
    x = rng.integers(0, 256, (N, C, H, W)).astype(np.uint8) if zp else rng.integers(-128, 128, (N, C, H, W)).astype(np.int8)
    buf = torch.zeros(x.size + 4 * words, dtype=torch.uint8 if zp else torch.int8, device="cuda")
    xd = buf[4 * words:].view(x.shape)
    xd.copy_(torch.from_numpy(x))
    w = rng.integers(-127, 128, (M, C, k, k), dtype=np.int8)
    ws = rng.uniform(0.002, 0.012, M).astype(np.float32)
    bias = rng.integers(-3000, 3000, M).astype(np.int32)
    kw = dict(bias=bias, y_dtype=I8, stride=(s, s), pads=(pad,) * 4, dilations=(1, 1), group=1, activation=None)
    args = (0.02, zp, w, ws, None, float(0.02 * 0.007 * 74 * 74 * np.sqrt(C * k * k) / 45), 0)
    want = oracle.qlinearconv(x, *args, **kw)
    out = torch.empty(want.shape, dtype=torch.int8, device="cuda")
    for _ in range(2):
        out.fill_(99)
        ctx.qlinearconv(xd, *args, **kw, out=out)
        ctx.synchronize()
        assert np.array_equal(out.cpu().numpy(), want)
