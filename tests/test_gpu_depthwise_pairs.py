"""Depthwise 3x3 on planes 28 wide, by batches of planes with a thread for one output row, or for two from two batches an SM on: heights that
leave a single row, partial batches, input zero points, unsigned codes, activations and outputs of the general form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def batch(H, threads):
    """planes of a batch: 256 threads, `threads` a plane, whole 16 bytes"""
    unit = 16
    while unit > 1 and H * 28 * (unit // 2) % 16 == 0:
        unit //= 2
    return 256 // threads // unit * unit


# planes on either side of two batches of two-row threads for each of 148 SMs, with a partial batch at the end; fewer than four of those batches
ONE_ROW = [(9, 24, 28), (5, 40, 27), (31, 8, 5), (3, 33, 64), (40, 16, 1), (200, 12, 2), (5, 8, 28), (80, 66, 28)]
TWO_ROWS = [(60, 89, 28), (59, 81, 27), (200, 125, 5), (43, 57, 64), (800, 95, 1), (777, 98, 2), (60, 106, 28)]


def test_shapes_reach_the_forms():
    for N, C, H in ONE_ROW:
        pair, row = batch(H, (H + 1) // 2), batch(H, H)
        assert N * C < 2 * 148 * pair
    for N, C, H in TWO_ROWS:
        pair = batch(H, (H + 1) // 2)
        assert N * C >= 2 * 148 * pair and N * C % pair != 0, (N, C, H, pair)


@pytest.mark.parametrize("N,C,H", ONE_ROW + TWO_ROWS)
@pytest.mark.parametrize("x_dtype,y_dtype,act", [("int8", "I8", "relu6"), ("uint8", "I8", None), ("int8", "U8", "relu"), ("uint8", "I8", "relu")])
def test_pairs_of_rows(zb, ctx, oracle, N, C, H, x_dtype, y_dtype, act):
    rng = np.random.default_rng(N + C + H)
    lo, hi = (0, 256) if x_dtype == "uint8" else (-128, 128)
    x = rng.integers(lo, hi, (N, C, H, 28)).astype(x_dtype)
    w = rng.integers(-127, 128, (C, 1, 3, 3), dtype=np.int8)
    ws = rng.uniform(0.008, 0.012, C).astype(np.float32)
    if N * C * H * 28 > 1 << 20 and (act, y_dtype) not in (("relu6", "I8"), ("relu", "U8")):
        pytest.skip("the large sizes with two of the four forms of codes")
    args = (x, 0.02, 9 if x_dtype == "uint8" else -7, w, ws, None, float(0.02 * 0.01 * 74.0 * 74.0 * 3.0 / 40.0), 0 if y_dtype == "I8" else 60)
    kw = dict(bias=rng.integers(-2000, 2000, C).astype(np.int32), y_dtype=getattr(zb, y_dtype), stride=(1, 1), pads=(1,) * 4, dilations=(1, 1), group=C, activation=act)
    want = oracle.qlinearconv(*args, **kw)
    assert np.array_equal(ctx.qlinearconv(*args, **kw), want)
    assert len(np.unique(want)) > 20
