"""Host arrays of a call: small ones leave as one copy, large weights on a stream of their own beside the kernels of the call before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def call(ctx, oracle, rng, N, C, H, W, M, k, s, zp=0):
    import torch
    x = rng.integers(-128, 128, (N, C, H, W)).astype(np.int8)
    w = rng.integers(-127, 128, (M, C, k, k), dtype=np.int8)
    ws = rng.uniform(0.002, 0.012, M).astype(np.float32)
    bias = rng.integers(-3000, 3000, M).astype(np.int32)
    pad = k // 2 if zp == 0 else 0
    kw = dict(bias=bias, stride=(s, s), pads=(pad,) * 4, dilations=(1, 1), group=1, activation="relu")
    args = (ws, None, float(0.02 * 0.007 * 74 * 74 * np.sqrt(C * k * k) / 45), 0)
    want = oracle.qlinearconv(x, 0.02, zp, w, *args, y_dtype=1, **kw)
    xd, y = torch.from_numpy(x).cuda(), torch.empty(want.shape, dtype=torch.int8, device="cuda")
    return want, y, lambda: ctx.qlinearconv(xd, 0.02, zp, w, *args, y_dtype=1, out=y, **kw), (w, ws, bias)


def test_weights_of_calls_in_a_row(zb, oracle):
    """No call waits for another: each one's weights, changed as soon as it returns, are its own, in any order of sizes and kernels."""
    ctx = zb.Context(0)
    rng = np.random.default_rng(0)
    shapes = [(4, 256, 14, 14, 512, 3, 2, 0),        # channels-last, 1.2 MB
              (4, 200, 14, 14, 208, 3, 2, 0),        # 374 KB: pieces of two sizes
              (2, 170, 27, 27, 180, 3, 1, 0),
              (3, 192, 28, 28, 256, 3, 1, 0),        # implicit GEMM from NCHW
              (4, 260, 14, 13, 120, 3, 2, 5),        # im2col (an input zero point), 281 KB
              (2, 300, 9, 9, 700, 4, 1, 0),          # 3.4 MB: whole slots
              (2, 16, 30, 30, 24, 3, 1, 0),          # small arrays only
              (4, 256, 14, 14, 114, 3, 2, 0)]        # 262656 bytes: just above the line
    cases = [call(ctx, oracle, rng, *s) for s in shapes]
    for order in (range(len(cases)), reversed(range(len(cases))), (0, 0, 1, 0, 3, 5, 0, 6, 0, 5, 5, 1)):
        want = {}
        for i in order:
            w, y, go, arrays = cases[i]
            keep = [a.copy() for a in arrays]
            go()
            for a in arrays:
                a[...] = 77                          # (the library has read them)
            for a, b in zip(arrays, keep):
                a[...] = b
            want[i] = (w, y)
        ctx.synchronize()
        for i, (w, y) in want.items():
            assert np.array_equal(y.cpu().numpy(), w), shapes[i]
            y.zero_()
    ctx.close()


def test_weights_under_a_limit_and_without_memory(zb, oracle):
    """Under an arena limit, or when the buffers cannot be had, the weights go through the arena as before."""
    rng = np.random.default_rng(1)
    ctx = zb.Context(0, arena_bytes=1 << 26)
    want, y, go, _ = call(ctx, oracle, rng, 4, 256, 14, 14, 512, 3, 2)
    zb.debug_fail_alloc(1)
    go()
    zb.debug_fail_alloc(0)
    ctx.synchronize()
    assert np.array_equal(y.cpu().numpy(), want)
    ctx.set_arena_limit(1 << 26)
    y.zero_()
    go()
    ctx.synchronize()
    assert np.array_equal(y.cpu().numpy(), want)
    ctx.close()


def test_small_arrays_of_one_call(ctx, oracle):
    """Inputs in host memory too, together around a quarter of a slot (256 KB) of the page-locked ring, and the gaps between the arrays."""
    rng = np.random.default_rng(2)
    for N, C, H, W, M in ((1, 3, 9, 29, 5), (2, 40, 30, 50, 33), (2, 40, 48, 64, 33), (1, 64, 64, 64, 16)):
        x = rng.integers(-128, 128, (N, C, H, W)).astype(np.int8)
        w = rng.integers(-127, 128, (M, C, 3, 3), dtype=np.int8)
        ws = rng.uniform(0.002, 0.012, M).astype(np.float32)
        bias = rng.integers(-3000, 3000, M).astype(np.int32)
        args = (0.02, 0, w, ws, None, float(0.02 * 0.007 * 74 * 74 * np.sqrt(C * 9) / 45), 0)
        kw = dict(bias=bias, y_dtype=1, stride=(1, 1), pads=(1,) * 4, dilations=(1, 1), group=1, activation=None)
        assert np.array_equal(ctx.qlinearconv(x, *args, **kw), oracle.qlinearconv(x, *args, **kw))


def test_stream_changed_between_calls(zb, oracle):
    """Calls return with copies under way; the context's own stream goes away, and the next call, whose arrays share the ring, runs on another."""
    import torch
    ctx = zb.Context(0)
    rng = np.random.default_rng(3)
    cases = [call(ctx, oracle, rng, *s) for s in ((2, 16, 30, 30, 24, 3, 1, 0), (4, 256, 14, 14, 512, 3, 2, 0), (2, 170, 27, 27, 180, 3, 1, 0))]
    streams = [torch.cuda.Stream() for _ in range(4)]
    for turn in range(5):
        if turn:                                         # the first of these destroys the context's own stream
            ctx.set_stream(streams[turn - 1].cuda_stream)
        for i in (turn % 3, (turn + 1) % 3, 0):
            want, y, go, _ = cases[i]
            y.zero_()
            torch.cuda.synchronize()
            go()
    ctx.synchronize()
    for want, y, _, _ in cases:
        assert np.array_equal(y.cpu().numpy(), want)
    ctx.close()
