"""Calls on a stream that is being captured into a CUDA graph."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def captured(zb):
    """A context on a torch stream, and a function that captures `body` there."""
    import torch
    c = zb.Context(0)
    stream = torch.cuda.Stream()
    c.set_stream(stream.cuda_stream)

    def capture(body):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            body()
        return graph
    yield c, capture, stream
    stream.synchronize()
    c.set_stream(torch.cuda.default_stream().cuda_stream)
    c.close()


def test_device_buffers_are_captured(zb, captured):
    import torch
    c, capture, stream = captured
    x, y, z = torch.zeros(1000, device="cuda"), torch.empty(1000, device="cuda"), torch.empty(1000, device="cuda")
    torch.cuda.synchronize()

    def body():
        c.ReLU(x, out=y)
        c.sum_tensors(y, x, out=z)
    g = capture(body)
    for k in (-2.0, 3.0):
        x.fill_(k)
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        assert z.eq(max(k, 0) + k).all()


def test_staged_buffers_are_refused(zb, captured):
    """What a call stages lies in memory of the context that later calls use again: a replay would read theirs."""
    import torch
    c, capture, stream = captured
    rng = np.random.default_rng(0)
    x = torch.from_numpy(rng.integers(-128, 128, (2, 48, 28, 28), dtype=np.int8)).cuda()
    w = rng.integers(-127, 128, (40, 48, 3, 3), dtype=np.int8)
    y, f = torch.empty((2, 40, 28, 28), dtype=torch.int8, device="cuda"), torch.empty(8, device="cuda")
    kw = dict(pads=(1, 1, 1, 1), out=y)
    calls = [lambda: c.qlinearconv(x, 0.02, 0, w, [0.01], None, 0.5, 0, **kw),
             lambda: c.qlinearconv(x, 0.02, 0, torch.from_numpy(w), [0.01], None, 0.5, 0, **kw),
             lambda: c.ReLU(np.ones(8, np.float32), out=f),
             lambda: c.ReLU(f, out=np.ones(8, np.float32))]
    calls[0]()
    calls[2]()
    c.synchronize()
    for call in calls:
        names = []

        def body():
            c.ReLU(f, out=f)
            try:
                call()
            except zb.ZantError as e:
                names.append(e.name)
        capture(body)
        assert names == ["Cuda"], names
    calls[0]()                                       # the context goes on working
    c.synchronize()


def test_plan_reads_a_host_input_again_at_each_replay(zb, captured):
    """Host input, device result: the copy is part of the graph and takes what the array holds then."""
    import torch
    c, capture, stream = captured
    g = zb.Graph("relu")
    n = 100000
    x, y = g.tensor("x", zb.F32, (1, n)), g.tensor("y", zb.F32, (1, n))
    g.node("Relu", [x], [y])
    g.input, g.output = x, y
    plan = zb.Plan(c, g)
    a, out = np.full((1, n), 1.0, np.float32), torch.empty((1, n), device="cuda")
    plan.run(a, out=out)
    c.synchronize()
    graph = capture(lambda: plan.run(a, out=out))
    for k in (5.0, -1.0, 7.0):
        a[:] = k
        plan.run(np.full((1, n), 99.0, np.float32), out=torch.empty((1, n), device="cuda"))     # another call in between
        c.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert out.eq(max(k, 0.0)).all()
    plan.close()
