"""Calls at a limit of the staging arena: a call whose own buffers fit runs, if need be on a kernel that wants less workspace."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
I8 = 1


class Limited:
    def __init__(self, zb, limit):
        self.ctx = zb.Context(0, arena_bytes=limit)
        self.ctx.set_arena_limit(limit)

    def __enter__(self):
        return self.ctx

    def __exit__(self, *a):
        self.ctx.close()


# N C H W M k s, weights on the device, limit: what the buffers of the call and the smallest workspace need
CONV = [
    (8, 64, 56, 56, 64, 3, 1, True, 64 << 10),       # implicit GEMM: blocked weights
    (8, 45, 27, 27, 85, 3, 1, True, 64 << 10),       # channels-last copy of the input
    (8, 64, 56, 56, 64, 1, 1, True, 8 << 10),        # pointwise
    (1, 3, 224, 224, 32, 3, 2, True, 3 << 10),       # stem
    (8, 64, 56, 56, 64, 1, 2, False, 1 << 20),       # a 1 x 1 filter with stride 2: the im2col matrix is smaller than the input
    (4, 512, 28, 28, 512, 1, 1, False, 300 << 10),   # pointwise, host weights: 256 KB of them
    (1, 1, 12, 12, 24, 5, 1, False, 2 << 10),        # few positions: weights padded to steps of 32 channels
]


@pytest.mark.parametrize("case", CONV, ids=[f"conv{i}" for i in range(len(CONV))])
def test_qlinearconv(zb, oracle, case):
    import torch
    N, C, H, W, M, k, s, dev, limit = case
    rng = np.random.default_rng(C + M)
    x = rng.integers(-128, 128, (N, C, H, W), dtype=np.int8)
    w = rng.integers(-127, 128, (M, C, k, k), dtype=np.int8)
    args = (np.array([0.01], np.float32), None, float(np.float32(0.02 * np.sqrt(C * k * k))), 0)
    kw = dict(stride=(s, s), pads=(k // 2,) * 4)
    want = oracle.qlinearconv(x, 0.02, 0, w, *args, **kw)
    y = torch.empty(want.shape, dtype=torch.int8, device="cuda")
    with Limited(zb, limit) as c:
        c.qlinearconv(torch.from_numpy(x).cuda(), 0.02, 0, torch.from_numpy(w).cuda() if dev else w, *args, out=y, **kw)
        c.synchronize()
    assert np.array_equal(y.cpu().numpy(), want)


@pytest.mark.parametrize("M,K,N,dev,limit", [(512, 256, 128, True, 8 << 10), (40, 3, 4000, False, 64 << 10)])
def test_qlinearmatmul(zb, oracle, M, K, N, dev, limit):
    import torch
    rng = np.random.default_rng(K)
    a, b = rng.integers(-128, 128, (M, K), dtype=np.int8), rng.integers(-127, 128, (K, N), dtype=np.int8)
    args = (np.array([0.01], np.float32), None, float(np.float32(0.02 * np.sqrt(K))), 0)
    want = oracle.qlinearmatmul(a, 0.02, 0, b, *args)
    y = torch.empty(want.shape, dtype=torch.int8, device="cuda")
    with Limited(zb, limit) as c:
        c.qlinearmatmul(torch.from_numpy(a).cuda(), 0.02, 0, torch.from_numpy(b).cuda() if dev else b, *args, out=y)
        c.synchronize()
    assert np.array_equal(y.cpu().numpy(), want)


def test_channels_last(zb, oracle):
    import torch
    rng = np.random.default_rng(1)
    N, C, H, W, M = 2, 128, 20, 20, 64
    x, w = rng.integers(-128, 128, (N, C, H, W), dtype=np.int8), rng.integers(-127, 128, (M, C, 3, 3), dtype=np.int8)
    bias = rng.integers(-2000, 2000, M).astype(np.int32)
    args = (np.array([0.01], np.float32), None, float(np.float32(0.02 * np.sqrt(C * 9))), 0)
    want = oracle.qlinearconv(x, 0.02, 0, w, *args, bias=bias, pads=(1, 1, 1, 1))
    y = torch.empty((N, H, W, M), dtype=torch.int8, device="cuda")
    with Limited(zb, 80 << 10) as c:                 # the weights are 72 KB
        c.qlinearconv_nhwc(torch.from_numpy(np.ascontiguousarray(x.transpose(0, 2, 3, 1))).cuda(), 0.02, 0, w, *args, bias=bias, pads=(1, 1, 1, 1), out=y)
        c.synchronize()
    assert np.array_equal(y.cpu().numpy().transpose(0, 3, 1, 2), want)
