"""Staging of single-operator calls: weights re-blocked on the device, pageable buffers through the page-locked ring."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
I8, U8 = 1, 2


def codes(rng, shape, dt):
    return rng.integers(0, 256, shape, dtype=np.uint8) if dt == U8 else rng.integers(-128, 128, shape, dtype=np.int8)


@pytest.mark.parametrize("N,C,H,W,M,k,s,xdt,xzp", [
    (2, 48, 28, 28, 40, 3, 1, I8, 0),        # implicit GEMM from NCHW
    (2, 64, 28, 28, 136, 1, 1, U8, 128),     # pointwise, two filter tiles
    (2, 96, 28, 28, 24, 1, 1, I8, -3),       # pointwise, block-diagonal weights
    (1, 3, 96, 96, 32, 3, 2, U8, 7),         # stem
    (2, 48, 27, 27, 72, 3, 2, I8, 5),        # im2col, K order (tap, channel)
    (2, 45, 27, 27, 72, 3, 1, I8, 5),        # im2col, K order (channel, tap)
])
def test_qlinearconv_weights_in_either_memory(ctx, oracle, N, C, H, W, M, k, s, xdt, xzp):
    """The weights of a call are re-blocked on the device; they may live in host or device memory."""
    import torch
    rng = np.random.default_rng(C + M)
    x = codes(rng, (N, C, H, W), xdt)
    w = rng.integers(-127, 128, (M, C, k, k), dtype=np.int8)
    ws = (rng.random(M, dtype=np.float32) * 0.02 + 0.001).astype(np.float32)
    args = (ws, None, float(np.float32(0.02 * np.sqrt(C * k * k))), 0)
    kw = dict(stride=(s, s), pads=(k // 2,) * 4)
    want = oracle.qlinearconv(x, 0.02, xzp, w, *args, **kw)
    assert np.array_equal(ctx.qlinearconv(x, 0.02, xzp, w, *args, **kw), want)
    assert np.array_equal(ctx.qlinearconv(x, 0.02, xzp, torch.from_numpy(w).cuda(), *args, **kw), want)


@pytest.mark.parametrize("n", [1, 131072, 131073, 700001, 9000001])
def test_pageable_transfers(ctx, n):
    """Host arrays around the slot size of the page-locked ring (131072 floats), and more than the whole ring."""
    x = np.random.default_rng(n).standard_normal(n).astype(np.float32)
    for _ in range(2):
        assert np.array_equal(ctx.ReLU(x), np.maximum(x, 0))


@pytest.mark.parametrize("N,C,H,W,M,k", [(1, 192, 18, 18, 160, 3),      # a 256-filter tile's weights leave no room for two stages
                                         (2, 64, 3, 3, 16, 3), (1, 64, 5, 100, 48, 1)])   # mostly empty row blocks
def test_channels_last_shapes_that_fill_tiles_badly(ctx, oracle, N, C, H, W, M, k):
    rng = np.random.default_rng(C)
    x = codes(rng, (N, C, H, W), I8)
    w = rng.integers(-127, 128, (M, C, k, k), dtype=np.int8)
    args = (np.array([0.01], np.float32), None, float(np.float32(0.02 * np.sqrt(C * k * k))), 0)
    kw = dict(pads=(k // 2,) * 4)
    want = oracle.qlinearconv(x, 0.02, 0, w, *args, **kw)
    got = ctx.qlinearconv_nhwc(np.ascontiguousarray(x.transpose(0, 2, 3, 1)), 0.02, 0, w, *args, **kw)
    assert np.array_equal(got.transpose(0, 3, 1, 2), want)
