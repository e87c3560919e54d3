"""Depthwise 3x3 QLinearConv on few planes: the rows of a plane are cut into bands for different warps.

Integer arithmetic and one rounding per output: the codes have to equal the oracle's exactly."""
import numpy as np
import pytest

I8 = 1
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W", [16, 12, 20, 13])                      # 8 columns per lane, 4 (narrow and wide), unaligned rows
@pytest.mark.parametrize("H", [1, 3, 4, 5, 7, 9, 13, 22, 64])         # one band; bands of two and three rows with last bands of one and two; many
@pytest.mark.parametrize("stride", [1, 2])
def test_bands(ctx, oracle, H, W, stride):
    if stride == 2 and (H % 2 or W % 2):
        H, W = H + H % 2, W + W % 2
    rng = np.random.default_rng(100 * H + W + stride)
    C, u8 = 5, H % 2 == 0
    x = rng.integers(0, 256, (2, C, H, W)).astype(np.uint8) if u8 else rng.integers(-128, 128, (2, C, H, W)).astype(np.int8)
    w = rng.integers(-127, 128, (C, 1, 3, 3), dtype=np.int8)
    ws = (rng.random(C, dtype=np.float32) * 0.02 + 0.001).astype(np.float32)
    bias = rng.integers(-3000, 3000, C).astype(np.int32)
    kw = dict(bias=bias, y_dtype=I8, stride=(stride, stride), pads=(1, 1, 1, 1), dilations=(1, 1), group=C, activation=["relu", None, "relu6"][W % 3])
    args = (x, 0.02, 7 if u8 else -5, w, ws, None, 0.045, 0)
    got, want = ctx.qlinearconv(*args, **kw), oracle.qlinearconv(*args, **kw)
    assert np.array_equal(got, want)
    assert len(np.unique(want)) > (16 if want.size > 400 else 2)


def test_bands_many_groups(ctx, oracle):
    """enough plane groups for bands of four rows and more, for two bands each, and for whole planes"""
    rng = np.random.default_rng(3)
    for C in (700, 3000, 5000):
        x = rng.integers(-128, 128, (1, C, 31, 128)).astype(np.int8)
        w = rng.integers(-127, 128, (C, 1, 3, 3), dtype=np.int8)
        ws = (rng.random(C, dtype=np.float32) * 0.02 + 0.001).astype(np.float32)
        kw = dict(bias=None, y_dtype=I8, stride=(1, 1), pads=(1, 1, 1, 1), dilations=(1, 1), group=C, activation=None)
        args = (x, 0.02, 0, w, ws, None, 0.045, 0)
        assert np.array_equal(ctx.qlinearconv(*args, **kw), oracle.qlinearconv(*args, **kw))
