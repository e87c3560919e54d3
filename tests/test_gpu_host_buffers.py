"""Host buffers of a call are read inside their bounds: arrays that end at an unmapped page."""
import ctypes
import mmap

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
I8 = 1


def before_unmapped_page(a):
    """A copy of `a` whose last byte is the last one of a mapped page."""
    page = mmap.PAGESIZE
    room = -(-a.nbytes // page) * page
    m = mmap.mmap(-1, room + page)
    start = ctypes.addressof(ctypes.c_char.from_buffer(m))
    assert ctypes.CDLL(None, use_errno=True).mprotect(ctypes.c_void_p(start + room), ctypes.c_size_t(page), 0) == 0
    out = np.frombuffer(m, dtype=a.dtype, count=a.size, offset=room - a.nbytes).reshape(a.shape)
    out[...] = a
    return out


# filters below and above a filter tile of 64, 128, 256
@pytest.mark.parametrize("M", [16, 48, 80, 320])
@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
def test_qlinearconv_bias_and_weights(ctx, oracle, layout, M):
    rng = np.random.default_rng(M)
    N, C, H, W = 2, 64, 24, 24
    x = rng.integers(-128, 128, (N, C, H, W), dtype=np.int8)
    w = before_unmapped_page(rng.integers(-127, 128, (M, C, 3, 3), dtype=np.int8))
    bias = before_unmapped_page(rng.integers(-3000, 3000, M).astype(np.int32))
    ws = before_unmapped_page((rng.random(M, dtype=np.float32) * 0.01 + 0.002).astype(np.float32))
    args = (0.02, 0, w, ws, None, float(np.float32(0.02 * np.sqrt(C * 9))), 0)
    kw = dict(bias=bias, pads=(1, 1, 1, 1))
    want = oracle.qlinearconv(x, *args, **kw)
    if layout == "nchw":
        got = ctx.qlinearconv(x, *args, **kw)
    else:
        got = ctx.qlinearconv_nhwc(np.ascontiguousarray(x.transpose(0, 2, 3, 1)), *args, **kw).transpose(0, 3, 1, 2)
    assert np.array_equal(got, want)
    assert len(np.unique(want)) > 16
