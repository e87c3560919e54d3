"""First stages of the fused int8 CNN: inputs on both sides of every rounding step of the quantisation for several scales (the quotient is
computed without a division), biases that the float form of the accumulators does not take, batches around the blocks of 128 images."""
import numpy as np
import pytest

import graph_oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def models(zb):
    from zant_b200 import models
    return models


@pytest.fixture(scope="module")
def scales(zb, ctx, models):
    return models.calibrate_on_gpu(ctx, models.small_cnn_fp32(64), models.small_cnn_input(64))


def _run(zb, ctx, oracle, g, x):
    want = graph_oracle.run(oracle, g, x)
    plan = zb.Plan(ctx, g, fuse=True)
    assert any("Fused" in n for n in plan.step_names())
    got = plan.run(x)
    plan.close()
    assert np.array_equal(got.view(np.uint32), want[g.output].view(np.uint32))
    return want


@pytest.mark.parametrize("zp", [0, 131])
@pytest.mark.parametrize("scale", [1.0 / 255.0, 1.0 / 256.0, 0.007812501, 0.3, 3.1e-5, 17.0, 1.0e-31])
def test_quantisation_steps(zb, ctx, oracle, models, scales, scale, zp):
    s = np.float32(scale)
    g = models.small_cnn_int8(8, act_scales=scales)
    g.nodes[0]["attrs"].update(y_scale=float(s), y_zp=zp)
    g.nodes[1]["attrs"].update(x_scale=float(s), x_zp=zp, y_scale=float(s) * g.nodes[1]["attrs"]["y_scale"] * 255.0)
    for n in g.nodes[2:]:
        if n["op"] == "Relu" and n["inputs"][0] == g.nodes[1]["outputs"][0]:
            n["attrs"].update(x_scale=g.nodes[1]["attrs"]["y_scale"], y_scale=g.nodes[1]["attrs"]["y_scale"])
    g.nodes[4]["attrs"].update(x_scale=g.nodes[1]["attrs"]["y_scale"])
    # k + 0.5 steps of the code, a few floats to either side
    v = ((np.arange(-zp - 2, 258 - zp, dtype=np.float64) + 0.5) * float(s)).astype(np.float32)
    around = [v]
    up, dn = v, v
    for _ in range(3):
        up, dn = np.nextafter(up, np.float32(np.inf)), np.nextafter(dn, np.float32(-np.inf))
        around += [up, dn]
    pool = np.concatenate(around + [np.array([np.inf, -np.inf, np.nan, 0.0, -0.0, 3.0e38, -3.0e38, 1.0e-45], np.float32)])
    x = np.random.default_rng(zp).permutation(np.resize(pool, 8 * 784)).astype(np.float32).reshape(8, 1, 28, 28)
    want = _run(zb, ctx, oracle, g, x)
    assert len(np.unique(want[g.nodes[0]["outputs"][0]])) > 200


@pytest.mark.parametrize("layer", [1, 4])
def test_biases_beyond_the_float_form(zb, ctx, oracle, models, scales, layer):
    g = models.small_cnn_int8(5, act_scales=scales, bias_amplitude=(100, 1000, 5000, 300))
    t = g.tensors[g.nodes[layer]["inputs"][4]]
    t["data"] = t["data"].copy()
    t["data"][::3] = 5_000_000
    t["data"][1::3] = -4_500_000
    _run(zb, ctx, oracle, g, models.small_cnn_input(5, 9))


@pytest.mark.parametrize("batch", [1, 2, 127, 128, 129, 131, 260])
def test_blocks_of_images(zb, ctx, oracle, models, scales, batch):
    g = models.small_cnn_int8(batch, act_scales=scales, bias_amplitude=(100, 1000, 5000, 300))
    _run(zb, ctx, oracle, g, models.small_cnn_input(batch, batch))


@pytest.mark.parametrize("batch", [700, 1025])
def test_several_single_windows_a_cta(zb, ctx, oracle, models, scales, batch):
    g = models.small_cnn_int8(batch, act_scales=scales, bias_amplitude=(100, 1000, 5000, 300))
    _run(zb, ctx, oracle, g, models.small_cnn_input(batch, batch))


@pytest.mark.parametrize("batch", [384, 390, 512, 513])
def test_column_tiles_of_fc1(zb, ctx, oracle, models, scales, batch):
    """Around four blocks of 128 images, where fc1's column tiles are wider than the grid alone asks for."""
    g = models.small_cnn_int8(batch, act_scales=scales, bias_amplitude=(100, 1000, 5000, 300))
    _run(zb, ctx, oracle, g, models.small_cnn_input(batch, batch))
