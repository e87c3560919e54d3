"""Page-locked results come straight from the device; pageable ones of the same size pass the ring."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 1000, 200000, 262080, 262081, 300000])      # a result that fills a slot of the ring, and one more
def test_results(ctx, n):
    import torch
    x = np.random.default_rng(n).standard_normal(n).astype(np.float32)
    xp, yp = torch.from_numpy(x).pin_memory(), torch.zeros(n).pin_memory()
    for a in (x, xp):
        for out in (np.zeros(n, np.float32), yp):
            ctx.ReLU(a, out=out)
            assert np.array_equal(np.asarray(out), np.maximum(x, 0))
        yp.zero_()


def test_no_second_copy_on_the_host(ctx):
    """200000 floats: 54 us page-locked against 112 pageable; a detour through the ring made 88 of the 54."""
    import torch
    x = np.random.default_rng(0).standard_normal(200000).astype(np.float32)

    def best(a, out):
        t = []
        for _ in range(300):
            t0 = time.perf_counter()
            ctx.ReLU(a, out=out)
            t.append(time.perf_counter() - t0)
        return min(t)
    pageable = best(x, np.empty_like(x))
    assert best(torch.from_numpy(x).pin_memory(), torch.empty(200000).pin_memory()) < 0.65 * pageable
