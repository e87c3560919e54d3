"""Expand 1x1 -> depthwise 3x3 -> project 1x1 [-> residual addition] on bands of rows and clusters of CTAs (irb_band.cuh) against the oracle, bit for bit."""
import numpy as np
import pytest

import graph_oracle
from test_gpu_inverted_residual import block

pytestmark = pytest.mark.gpu

# N C E M H W, input zero point, biases, residual addition: 0 none, 1 input first, 2 input second; stride
CASES = [
    (1, 64, 384, 64, 14, 14, 0, True, 1, 1),        # one image
    (1, 16, 96, 24, 112, 112, 2, True, 0, 2),       # widest plane of the networks, stride 2
    (2, 24, 144, 24, 56, 56, 3, True, 2, 1),        # nine 16-channel tiles, K step partly empty
    (1, 160, 960, 320, 7, 7, -3, True, 0, 1),       # odd plane, twenty filter tiles
    (37, 160, 960, 160, 5, 5, 0, True, 1, 1),       # several chunks a CTA, an odd image
    (100, 96, 576, 96, 10, 10, 0, True, 2, 1),
    (3, 32, 192, 64, 13, 13, 1, True, 0, 2),        # stride 2 on an odd plane: no row below the last
    (2, 32, 192, 64, 9, 10, -1, False, 0, 2),
    (4, 24, 144, 32, 11, 15, 2, True, 0, 1),        # rows of odd length
    (5, 40, 200, 48, 20, 18, 0, True, 0, 1),        # half a channel tile at the end
    (3, 12, 40, 8, 30, 33, -7, True, 0, 1),         # half a filter tile, one channel tile a CTA
    (2, 8, 17, 8, 6, 61, 0, True, 1, 1),            # a tile of one channel
    (4, 4, 8, 4, 2, 3, 0, True, 1, 1),              # smallest plane, a quarter of a K step
    (2, 16, 64, 40, 3, 4, 5, True, 0, 2),
    (1, 8, 32, 8, 300, 6, 0, True, 1, 1),           # high and narrow
    (1, 8, 48, 16, 4, 256, 0, True, 0, 2),          # one band of wide rows
    (64, 32, 192, 32, 20, 20, 0, True, 1, 1),       # two rounds of the SMs
]


@pytest.mark.parametrize("case", CASES, ids=["x".join(map(str, c[:6] + c[9:])) for c in CASES])
def test_block(zb, ctx, oracle, case):
    g, t1, t2, cur, xv = block(zb, case)
    out = g.tensor("out", zb.F32, g.tensors[cur]["shape"])
    g.node("DequantizeLinear", [cur], [out], x_scale=0.2, x_zp=0)
    g.output = out
    want = graph_oracle.run(oracle, g, xv)
    plan = zb.Plan(ctx, g, fuse=True)
    assert any("expand+depthwise+project" in n for n in plan.step_names())
    for graph in (False, True):
        plan.use_graph(graph)
        for _ in range(2):
            assert np.array_equal(plan.run(xv), want[g.output])
    assert len(np.unique(want[t1])) > 20 and len(np.unique(want[cur])) > 20
    plan.close()
