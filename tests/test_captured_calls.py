"""Tensor-core calls captured into a CUDA graph on the context's stream.  A replay meets inputs that the capture did not
see: the scale of the fp16 operands has to come from these, not from the largest values of any earlier replay (first
pass here: inputs 2^24 times larger), and calls outside the graph in between must not see the graph's."""
import numpy as np
import pytest

from parity_util import REL_L2_TOL, DeviceArrays, rel_l2

pytestmark = pytest.mark.gpu


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
