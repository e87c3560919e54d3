"""Depthwise 3x3 on planes 28 wide, where a thread takes two output rows: heights that leave a single row, partial batches, input zero points,
unsigned codes, activations and outputs of the general form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,C,H", [(9, 24, 28), (5, 40, 27), (31, 8, 5), (3, 33, 64), (40, 16, 1), (200, 12, 2)])
@pytest.mark.parametrize("x_dtype,y_dtype,act", [("int8", "I8", "relu6"), ("uint8", "I8", None), ("int8", "U8", "relu"), ("uint8", "I8", "relu")])
def test_pairs_of_rows(zb, ctx, oracle, N, C, H, x_dtype, y_dtype, act):
    rng = np.random.default_rng(N + C + H)
    lo, hi = (0, 256) if x_dtype == "uint8" else (-128, 128)
    x = rng.integers(lo, hi, (N, C, H, 28)).astype(x_dtype)
    w = rng.integers(-127, 128, (C, 1, 3, 3), dtype=np.int8)
    ws = rng.uniform(0.008, 0.012, C).astype(np.float32)
    args = (x, 0.02, 9 if x_dtype == "uint8" else -7, w, ws, None, float(0.02 * 0.01 * 74.0 * 74.0 * 3.0 / 40.0), 0 if y_dtype == "I8" else 60)
    kw = dict(bias=rng.integers(-2000, 2000, C).astype(np.int32), y_dtype=getattr(zb, y_dtype), stride=(1, 1), pads=(1,) * 4, dilations=(1, 1), group=C, activation=act)
    want = oracle.qlinearconv(*args, **kw)
    assert np.array_equal(ctx.qlinearconv(*args, **kw), want)
    assert len(np.unique(want)) > 20
