"""QLinearAdd with operand zero points outside the type's range: the entry point takes any int32."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("u8", [False, True])
@pytest.mark.parametrize("azp,bzp", [(256, 0), (0, -129), (300, -300), (5000, -4990), (16777217, -16777217)])
@pytest.mark.parametrize("scale", [0.1, 0.0472441])
def test_every_pair_of_codes(ctx, oracle, u8, azp, bzp, scale):
    """16 n + 5 values: the vector body and the rest of one call follow the same rule."""
    dt = np.uint8 if u8 else np.int8
    codes = np.arange(256, dtype=np.uint8).view(dt)
    a, b = (np.concatenate([v.reshape(-1), v.reshape(-1)[:5]]) for v in np.meshgrid(codes, codes))
    args = (a, scale, azp, b, scale, bzp, scale, 0)
    assert np.array_equal(ctx.qlinearadd(*args), oracle.qlinearadd(*args))
