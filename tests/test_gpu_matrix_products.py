"""QLinearMatMul on the tensor cores: rows that are runs of 16-byte chunks or not, results stored as words or bytes, column tiles of every width."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K,N", [(256, 1280, 1000), (300, 64, 30), (513, 40, 64), (1100, 80, 130), (2300, 128, 260), (256, 16, 1)])
@pytest.mark.parametrize("a_dtype,y_dtype,act", [("int8", "I8", "relu"), ("uint8", "I8", None), ("int8", "U8", "relu6")])
def test_qlinearmatmul(zb, ctx, oracle, M, K, N, a_dtype, y_dtype, act):
    rng = np.random.default_rng(M + K + N)
    lo, hi = (0, 256) if a_dtype == "uint8" else (-128, 128)
    a = rng.integers(lo, hi, (M, K)).astype(a_dtype)
    b = rng.integers(-127, 128, (K, N), dtype=np.int8)
    bs = rng.uniform(0.008, 0.012, N).astype(np.float32)
    yzp = 0 if y_dtype == "I8" else 100
    args = (a, 0.02, 0 if a_dtype == "int8" else 128, b, bs, None, float(0.02 * 0.01 * 74.0 * 74.0 * np.sqrt(K) / 50.0), yzp)
    kw = dict(bias=rng.integers(-500, 500, N).astype(np.int32), y_dtype=getattr(zb, y_dtype), activation=act)
    want = oracle.qlinearmatmul(*args, **kw)
    assert np.array_equal(ctx.qlinearmatmul(*args, **kw), want)
    assert len(np.unique(want)) > 5
