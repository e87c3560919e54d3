"""The workloads that the back end is timed on.

`listed()` are the fixed ones, `draw(rng)` gives more of the same ranges, `prepare` builds what a program holds before the
call (plan or weights, input and output buffers), `run` makes one pass through the public entry points of the package,
`work` and `tolerance` state what a pass cannot do without and how far two correct results may lie apart.

Families
  cnn     the reference's example CNN on 1x28x28 inputs, FP32 (the reference's arithmetic) or QLinear int8, as a plan
  calls   the same FP32 CNN as a generated predict() runs it: one library call per graph node
  mbv2    MobileNetV2-style int8 classifier as a plan
  yolo    Tiny-YOLOv3-style detector as a plan: int8, FP32 (the reference's arithmetic), TF32 or split TF32
  qconv   one QLinearConv call (NCHW or channels-last), weights in host memory as a generated library holds them

`where`: "device" = the caller's buffers are CUDA tensors, "host" = numpy arrays.  `graph`: the plan replays a captured
CUDA graph (plan.use_graph), the library's form for single-image latency.
"""
import functools
import math

import numpy as np
import torch

import __graft_entry__ as entry

zb = entry.load_package()
from zant_b200 import models  # noqa: E402

TF32_MODE = {"tf32": 1, "tf32x3": 2}
TORCH_DTYPE = {zb.F32: torch.float32, zb.I8: torch.int8, zb.U8: torch.uint8, zb.I32: torch.int32}


def listed():
    return [
        # one digit at a time: launches and host work are all there is
        dict(name="cnn_int8_b1", family="cnn", dtype="int8", batch=1, where="device", graph=False),
        # the headline configuration: a full batch resident on the GPU
        dict(name="cnn_int8_b65536", family="cnn", dtype="int8", batch=65536, where="device", graph=False),
        # a caller whose arrays are ordinary host memory, batch of no particular size
        dict(name="cnn_int8_host_b3001", family="cnn", dtype="int8", batch=3001, where="host", graph=False),
        # the reference's own FP32 network at its large batch
        dict(name="cnn_fp32_b4096", family="cnn", dtype="fp32", batch=4096, where="device", graph=False),
        # generated code, one call per node, one image
        dict(name="cnn_fp32_calls_b1", family="calls", batch=1, where="device"),
        # camera-style classification: one image, captured graph
        dict(name="mbv2_b1", family="mbv2", batch=1, res=224, graph=True),
        # a service's remainder batch on a smaller input
        dict(name="mbv2_r160_b37", family="mbv2", batch=37, res=160, graph=False),
        # bulk classification
        dict(name="mbv2_b1024", family="mbv2", batch=1024, res=224, graph=False),
        # detector, quantized, one GPU's share of a batch of 256
        dict(name="yolo_int8_b32", family="yolo", dtype="int8", batch=32, res=416),
        # detector in floating point on the tensor cores
        dict(name="yolo_tf32_b8", family="yolo", dtype="tf32", batch=8, res=416),
        # stand-alone QLinearConv: the sweep's stride-2 layer
        dict(name="qconv_256x14_512_s2", family="qconv", N=256, C=256, H=14, W=14, K=512, k=3, s=2, p=1, group=1, layout="nchw", x="int8", act="none"),
        # stand-alone QLinearConv on sizes that are multiples of nothing
        dict(name="qconv_odd_45x27", family="qconv", N=33, C=45, H=27, W=27, K=85, k=3, s=1, p=1, group=1, layout="nchw", x="uint8", act="relu"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["cnn", "cnn", "calls", "mbv2", "mbv2", "yolo", "yolo", "qconv", "qconv", "qconv"])
    if family == "cnn":
        dtype = rng.choice(["int8", "int8", "fp32"])
        batch = _log_int(rng, 1, 65536 if dtype == "int8" else 4096)
        where = rng.choice(["device", "device", "host"])
        if where == "host":
            batch = min(batch, 8192 + rng.randrange(512))
        return dict(family="cnn", dtype=dtype, batch=batch, where=where, graph=batch <= 64 and rng.random() < 0.5)
    if family == "calls":
        return dict(family="calls", batch=_log_int(rng, 1, 256), where=rng.choice(["device", "device", "host"]))
    if family == "mbv2":
        res = rng.choice([96, 112, 128, 144, 160, 176, 192, 208, 224])
        batch = _log_int(rng, 1, 768)
        return dict(family="mbv2", batch=batch, res=res, graph=batch <= 8 and rng.random() < 0.7)
    if family == "yolo":
        dtype = rng.choice(["int8", "int8", "tf32", "tf32x3", "fp32"])
        return dict(family="yolo", dtype=dtype, batch=_log_int(rng, 1, {"int8": 32, "fp32": 2}.get(dtype, 8)), res=rng.choice([160, 224, 256, 288, 320, 352, 416]))
    kind = rng.choice(["dense", "dense", "pointwise", "depthwise"])
    H = rng.randint(7, 80)
    W = H if rng.random() < 0.7 else rng.randint(7, 80)
    C = _log_int(rng, 8, 512)
    if rng.random() < 0.5:
        C = -(-C // 16) * 16
    K = C if kind == "depthwise" else _log_int(rng, 8, 512)
    if kind != "depthwise" and rng.random() < 0.5:
        K = -(-K // 16) * 16
    k = {"dense": rng.choice([3, 3, 5]), "pointwise": 1, "depthwise": 3}[kind]
    s = rng.choice([1, 1, 2])
    per_image = C * H * W * max(1, (K if kind != "depthwise" else 1) * k * k // 512)
    N = _log_int(rng, 1, max(1, min(256, 48_000_000 // per_image)))
    layout = "nchw"
    if kind != "depthwise" and rng.random() < 0.25:
        layout, s = "nhwc", 1
        C, K = -(-C // 64) * 64, -(-K // 16) * 16
        N = max(1, N // 2)
    return dict(family="qconv", N=N, C=C, H=H, W=W, K=K, k=k, s=s, p=k // 2, group=C if kind == "depthwise" else 1, layout=layout,
                x="int8" if layout == "nhwc" else rng.choice(["int8", "uint8"]), act=rng.choice(["none", "relu", "relu6"]))


# ------------------------------------------------------------------------------------------------ what a program keeps
@functools.lru_cache(maxsize=None)
def _context(tf32):
    ctx = zb.Context(0)
    ctx.set_tf32(tf32)
    return ctx


@functools.lru_cache(maxsize=None)
def _cnn_scales():
    return models.calibrate_on_gpu(_context(0), models.small_cnn_fp32(256), models.small_cnn_input(256))


@functools.lru_cache(maxsize=None)
def _yolo_scales():
    return models.activation_scales_on_gpu(_context(0), models.tiny_yolo_fp32(2), models.tiny_yolo_input(2))


@functools.lru_cache(maxsize=3)
def _network(family, dtype, batch, res):
    """The frozen graph with its weights: the same for every input."""
    if family == "cnn":
        return models.small_cnn_int8(batch, act_scales=_cnn_scales()) if dtype == "int8" else models.small_cnn_fp32(batch)
    if family == "mbv2":
        return models.mobilenetv2_int8(batch, res=res)
    f = models.tiny_yolo_fp32(batch, res=res)
    return models.tiny_yolo_int8(f, _yolo_scales()) if dtype == "int8" else f


def _graph_of(case):
    return _network(case["family"], case.get("dtype", "int8"), case["batch"], case.get("res", 28))


class _Held:
    """A case's state; a plan's device memory goes with it."""

    plan = None

    def __init__(self, case):
        self.case = case

    def __del__(self):
        if self.plan is not None:
            self.plan.close()


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def prepare(case, seed):
    st = _Held(case)
    gen = _generator(seed)
    if case["family"] == "calls":
        _prepare_calls(st, gen)
    elif case["family"] == "qconv":
        _prepare_qconv(st, gen, seed)
    else:
        graph = _graph_of(case)
        st.plan = zb.Plan(_context(TF32_MODE.get(case.get("dtype"), 0)), graph)
        if case.get("graph"):
            st.plan.use_graph()
        if graph.tensors[graph.input]["dtype"] == zb.U8:
            st.x = torch.randint(0, 256, st.plan.in_shape, dtype=torch.uint8, device="cuda", generator=gen)
        else:
            st.x = torch.rand(st.plan.in_shape, dtype=torch.float32, device="cuda", generator=gen)
        if case.get("where") == "host":
            st.x, st.y = st.x.cpu().numpy(), None
        else:
            st.y = torch.empty(st.plan.out_shape, dtype=TORCH_DTYPE[st.plan.out_dtype], device="cuda")
    return st


def _prepare_calls(st, gen):
    b = st.case["batch"]
    st.ctx = _context(0)
    st.x = torch.rand((b, 1, 28, 28), device="cuda", generator=gen)
    st.w = {k: torch.from_numpy(v).cuda() for k, v in models.small_cnn_weights().items()}
    shapes = dict(c1=(b, 32, 26, 26), r1=(b, 32, 26, 26), p1=(b, 32, 13, 13), c2=(b, 64, 11, 11), r2=(b, 64, 11, 11), p2=(b, 64, 5, 5),
                  m3=(b, 512), a3=(b, 512), r3=(b, 512), m4=(b, 10), a4=(b, 10))
    st.t = {k: torch.empty(v, device="cuda") for k, v in shapes.items()}
    if st.case["where"] == "host":
        st.x = st.x.cpu().numpy()
        st.w = {k: v.cpu().numpy() for k, v in st.w.items()}
        st.t = {k: v.cpu().numpy() for k, v in st.t.items()}
    st.flat = st.t["p2"].reshape(b, 1600)


def _prepare_qconv(st, gen, seed):
    c = st.case
    st.ctx = _context(0)
    shape = (c["N"], c["C"], c["H"], c["W"]) if c["layout"] == "nchw" else (c["N"], c["H"], c["W"], c["C"])
    unsigned = c["x"] == "uint8"
    st.x = torch.randint(0 if unsigned else -128, 256 if unsigned else 128, shape, dtype=torch.uint8 if unsigned else torch.int8, device="cuda", generator=gen)
    # weights, scales and biases are host arrays: symmetric int8 per output channel, an output range of about three sigma
    rng = np.random.default_rng(seed)
    cg = c["C"] // c["group"]
    st.w = rng.integers(-127, 128, (c["K"], cg, c["k"], c["k"]), dtype=np.int8)
    st.bias = rng.integers(-2000, 2001, c["K"]).astype(np.int32)
    st.x_scale, st.x_zp = 0.02, 128 if unsigned and c["p"] == 0 else 0
    st.w_scale = rng.uniform(0.008, 0.012, c["K"]).astype(np.float32)
    st.y_scale = float(np.float32(0.02 * 0.01 * 74.0 * (128.0 if unsigned and st.x_zp == 0 else 74.0) * math.sqrt(cg * c["k"] * c["k"]) / 42.0))
    oh, ow = _out_size(c)
    st.y = torch.empty((c["N"], c["K"], oh, ow) if c["layout"] == "nchw" else (c["N"], oh, ow, c["K"]), dtype=torch.int8, device="cuda")


def _out_size(c):
    return (c["H"] + 2 * c["p"] - c["k"]) // c["s"] + 1, (c["W"] + 2 * c["p"] - c["k"]) // c["s"] + 1


# ------------------------------------------------------------------------------------------------ one pass
def run(st):
    family = st.case["family"]
    if family == "calls":
        return _run_calls(st)
    if family == "qconv":
        return _run_qconv(st)
    return st.plan.run(st.x, out=st.y)


def _run_calls(st):
    ctx, w, t = st.ctx, st.w, st.t
    conv = dict(stride=(1, 1), pads=(0, 0, 0, 0), dilations=(1, 1), group=1, auto_pad="NOTSET")
    pool = ((2, 2), (2, 2), (1, 1), (0, 0, 0, 0))
    ctx.conv_lean(st.x, w["w1"], t["c1"].shape, bias=w["b1"], out=t["c1"], **conv)
    ctx.ReLU(t["c1"], out=t["r1"])
    ctx.onnx_maxpool_lean(t["r1"], t["p1"].shape, *pool, out=t["p1"])
    ctx.conv_lean(t["p1"], w["w2"], t["c2"].shape, bias=w["b2"], out=t["c2"], **conv)
    ctx.ReLU(t["c2"], out=t["r2"])
    ctx.onnx_maxpool_lean(t["r2"], t["p2"].shape, *pool, out=t["p2"])
    ctx.mat_mul(st.flat, w["w3"], out=t["m3"])
    ctx.sum_tensors(t["m3"], w["b3"], out=t["a3"])
    ctx.ReLU(t["a3"], out=t["r3"])
    ctx.mat_mul(t["r3"], w["w4"], out=t["m4"])
    return ctx.sum_tensors(t["m4"], w["b4"], out=t["a4"])


def _run_qconv(st):
    c = st.case
    call = st.ctx.qlinearconv if c["layout"] == "nchw" else st.ctx.qlinearconv_nhwc
    return call(st.x, st.x_scale, st.x_zp, st.w, st.w_scale, None, st.y_scale, 0, bias=st.bias, y_dtype=zb.I8, stride=(c["s"], c["s"]), pads=(c["p"],) * 4,
                dilations=(1, 1), group=c["group"], activation=c["act"], out=st.y)


# ------------------------------------------------------------------------------------------------ what a pass needs
def work(case):
    if case["family"] == "qconv":
        oh, ow = _out_size(case)
        weights = case["K"] * (case["C"] // case["group"]) * case["k"] ** 2
        outs = case["N"] * case["K"] * oh * ow
        return dict(bytes=case["N"] * case["C"] * case["H"] * case["W"] + weights + 8 * case["K"] + outs, flops=2.0 * outs * weights / case["K"])
    if case["family"] == "calls":
        # every node is a call of its own: its operands are read and its result is written
        b = case["batch"]
        acts = [784, 32 * 676, 32 * 676, 32 * 169, 64 * 121, 64 * 121, 1600, 512, 512, 512, 10, 10]
        weights = 288 + 32 + 64 * 288 + 64 + 1600 * 512 + 512 + 5120 + 10
        return dict(bytes=4 * (b * (2 * sum(acts) - acts[0] - acts[-1]) + weights), flops=2.0 * b * 3249280)
    g = _graph_of(case)
    size = {zb.F32: 4, zb.I8: 1, zb.U8: 1, zb.I32: 4}
    nbytes = sum(math.prod(t["shape"]) * size[t["dtype"]] for i, t in enumerate(g.tensors) if t["data"] is not None or i in (g.input, g.output))
    return dict(bytes=float(nbytes), flops=2.0 * case["batch"] * g.meta["macs_per_image"])


def tolerance(case):
    if case["family"] == "calls" or case.get("dtype") in ("fp32", "tf32x3"):
        return {"rel": 1e-5}        # 32-bit sums of up to a few thousand terms
    if case.get("dtype") == "tf32":
        return {"rel": 2e-3}        # operands of 10 stored mantissa bits
    return "exact"                  # integer codes, dequantised at most
