"""Tensor-core calls captured into a CUDA graph on the context's stream.  A replay meets inputs that the capture did not
see: the scale of the fp16 operands has to come from these, not from the largest values of any earlier replay (first
pass here: inputs 2^24 times larger), and calls outside the graph in between must not see the graph's."""
import numpy as np
import pytest

from parity_util import REL_L2_TOL, DeviceArrays, rel_l2

pytestmark = pytest.mark.gpu


def capture(ctx, call):
    import ctypes

    import torch

    raw = ctypes.c_void_p()
    ctx.call("katsu_cuda_stream", ctypes.byref(raw))
    stream = torch.cuda.ExternalStream(raw.value)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        call()

    def replay():
        with torch.cuda.stream(stream):
            graph.replay()

    return replay


@pytest.mark.parametrize("warm", [True, False], ids=["after an eager call", "first call"])
def test_the_graph_keeps_the_scratch_it_was_captured_with(warm):
    """Operand planes live in the context's scratch.  A larger call after the capture must not free the block that the graph
    writes to, and a capture that has to grow the scratch must not leave the context with memory of the graph's."""
    from katsu_b200 import cabi

    m, k, n, big = 200, 520, 648, 1500
    rng = np.random.default_rng(9)
    a, b, a2 = (rng.standard_normal(s).astype(np.float32) for s in ((m, k), (k, n), (big, big)))
    want, want2 = a.astype(np.float64) @ b, a2.astype(np.float64) @ a2
    context = cabi.Context(0)
    with DeviceArrays(context, a=a, b=b, a2=a2) as d:
        d.alloc("c", m * n), d.alloc("c2", big * big)
        if warm:
            context.matmul_fwd(d["a"], d["b"], d["c"], m, k, n)
        context.sync()
        replay = capture(context, lambda: context.matmul_fwd(d["a"], d["b"], d["c"], m, k, n))
        context.matmul_fwd(d["a2"], d["a2"], d["c2"], big, big, big)
        assert rel_l2(d.get("c2"), want2) <= REL_L2_TOL
        for i in range(8):
            d.alloc(f"other{i}", 1 << 20, fill=float(i))
        context.call("katsu_cuda_zero", d["c"], m * n)
        replay()
        assert rel_l2(d.get("c"), want) <= REL_L2_TOL
        for i in range(8):
            assert (d.get(f"other{i}") == i).all()
        replay = capture(context, lambda: context.matmul_fwd(d["a2"], d["a2"], d["c2"], big, big, big))
        context.call("katsu_cuda_zero", d["c2"], big * big)
        replay()
        assert rel_l2(d.get("c2"), want2) <= REL_L2_TOL
        del replay
    context.close()


def test_replays_with_new_inputs(ctx):
    import ctypes

    import torch

    m, k, n = 200, 520, 648
    rng = np.random.default_rng(5)
    a, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((k, n)).astype(np.float32)
    want = a.astype(np.float64) @ b.astype(np.float64)
    raw = ctypes.c_void_p()
    ctx.call("katsu_cuda_stream", ctypes.byref(raw))
    stream = torch.cuda.ExternalStream(raw.value)
    with DeviceArrays(ctx, a=a, b=b) as d:
        d.alloc("c", m * n)
        d.alloc("eager", m * n)
        ctx.matmul_fwd(d["a"], d["b"], d["c"], m, k, n)
        ctx.sync()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            ctx.matmul_fwd(d["a"], d["b"], d["c"], m, k, n)
        for scale in (2.0 ** 24, 1.0, 2.0 ** -24):
            ctx.h2d(d["a"], a * np.float32(scale))
            ctx.sync()
            with torch.cuda.stream(stream):
                graph.replay()
            ctx.matmul_fwd(d["a"], d["b"], d["eager"], m, k, n)
            got, eager = d.get("c"), d.get("eager")
            assert rel_l2(got, want * scale) <= REL_L2_TOL, scale
            assert np.array_equal(got, eager), scale
        del graph
