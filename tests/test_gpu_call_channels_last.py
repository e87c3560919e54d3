"""QLinearConv calls that are put channels-last first: stride 2 as parity planes, odd sizes, channel and filter remainders.

Integer results: they have to equal the oracle's exactly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
I8, U8 = 1, 2

CASES = [
    # N   C   H   W    M  k  s  pads          xdt zp  act
    (5, 45, 27, 27, 85, 3, 1, (1, 1, 1, 1), U8, 0, "relu"),         # odd planes, channel and filter remainders
    (3, 70, 9, 31, 300, 3, 1, (1, 1, 1, 1), I8, 0, "relu6"),        # two channel stages, filter tiles
    (9, 64, 14, 14, 48, 3, 2, (1, 1, 1, 1), I8, 0, None),           # stride 2, even sizes
    (4, 40, 15, 21, 33, 3, 2, (1, 1, 1, 1), U8, 0, "relu"),         # stride 2, odd sizes
    (3, 20, 18, 27, 24, 3, 2, (0, 1, 1, 0), I8, 0, "relu6"),        # stride 2, even and odd first tap
    (2, 24, 33, 26, 70, 5, 2, (2, 2, 2, 2), U8, 0, None),           # 5 x 5, stride 2: shifts of both signs
    (2, 12, 30, 41, 16, 5, 2, (1, 1, 1, 1), I8, 0, "relu"),         # at most 16 channel bytes
    (6, 9, 20, 16, 40, 3, 2, (1, 1, 1, 1), I8, 0, None),
    (3, 50, 23, 17, 66, 1, 2, (0, 0, 0, 0), U8, 128, "relu"),       # 1 x 1, stride 2: every second pixel; zero point folded in
    (4, 31, 11, 13, 20, 1, 1, (0, 0, 0, 0), U8, 128, None),         # 1 x 1 on odd planes and channels
    (2, 16, 9, 200, 24, 3, 2, (1, 1, 1, 1), I8, 0, "relu6"),        # a row of 100 outputs
    (1, 130, 26, 300, 40, 3, 2, (1, 1, 1, 1), I8, 0, None),         # two column segments
    (40, 8, 3, 3, 9, 3, 1, (1, 1, 1, 1), I8, 0, "relu"),            # tiles of mostly dead rows
    (7, 256, 14, 14, 512, 3, 2, (1, 1, 1, 1), I8, 0, "relu"),       # streamed weights, two images per tile, an odd one
    (90, 40, 2, 5, 24, 3, 1, (1, 1, 1, 1), U8, 0, None),            # four images per tile
    (300, 70, 3, 3, 33, 1, 2, (0, 0, 0, 0), I8, 3, "relu"),         # 1 x 1 with stride 2 onto 2 x 2: 32 images per tile
]


@pytest.mark.parametrize("case", CASES, ids=[f"nhcall{i}" for i in range(len(CASES))])
def test_qlinearconv(ctx, oracle, case):
    N, C, H, W, M, k, s, pads, xdt, zp, act = case
    rng = np.random.default_rng(N + C + H + W + M)
    x = rng.integers(0, 256, (N, C, H, W)).astype(np.uint8) if xdt == U8 else rng.integers(-128, 128, (N, C, H, W)).astype(np.int8)
    w = rng.integers(-127, 128, (M, C, k, k), dtype=np.int8)
    ws = (rng.random(M, dtype=np.float32) * 0.01 + 0.002).astype(np.float32)
    bias = rng.integers(-3000, 3000, M).astype(np.int32) if M % 3 else None
    kw = dict(bias=bias, y_dtype=I8, stride=(s, s), pads=pads, dilations=(1, 1), group=1, activation=act)
    args = (x, 0.02, zp, w, ws, None, float(0.02 * 0.007 * 74 * 74 * np.sqrt(C * k * k) / 45), 0)
    got, want = ctx.qlinearconv(*args, **kw), oracle.qlinearconv(*args, **kw)
    assert np.array_equal(got, want)
    assert len(np.unique(want)) > (6 if act == "relu6" else 16)      # (relu6 leaves 6 / y_scale codes)
