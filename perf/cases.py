"""The work that users of this library have it do, as cases that can be timed and compared.

Two public faces are called as their users call them: the C ABI through `cabi.Context` on device buffers the
caller owns (what a host program in any language does), and the Tensor / Conv2D graph (what a Python training
loop does).  Modes: 3xTF32, the default, and TF32, the opt-in.  Sizes are the named workloads of
`katsu_b200.workloads`, the benchmark's square matmuls, and generic layers around them.
"""
import math

import torch

import katsu_b200 as K
from katsu_b200 import cabi, workloads

MODES = {"3xtf32": cabi.MODE_3XTF32, "tf32": cabi.MODE_TF32}

_contexts = {}


def _context(mode):
    """One context per precision mode for the whole process, as a host program keeps it."""
    if mode not in _contexts:
        _contexts[mode] = cabi.Context(torch.cuda.current_device())
        _contexts[mode].set_precision(MODES[mode])
    return _contexts[mode]


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _conv(kind, n, c, h, w, k, r, s, stride, pad, mode, **more):
    return dict(kind=kind, n=n, c=c, h=h, w=w, k=k, r=r, s=s, stride=stride, pad=pad, mode=mode, **more)


def _named(kind, spec, mode, **more):
    p = workloads.CONV[spec]
    return _conv(kind, p.n, p.c, p.h, p.w, p.k, p.r, p.s, p.stride, p.pad, mode, **more)


def listed():
    return [
        # Katsu's own example: one RGB image through one layer and back, graph API.  Launches and host time.
        _named("conv_graph", "rgb_example", "3xtf32", name="rgb_example_graph"),
        # A linear classifier step (matmul, add, loss, backward, SGD) on a small batch: the smallest training loop.
        dict(kind="linear_graph", m=32, k=784, n=10, mode="3xtf32", name="linear_graph_32x784x10"),
        # A hidden layer served to a small batch: forward with bias and ReLU only.
        _conv("conv_infer", 8, 64, 56, 56, 64, 3, 3, 1, 1, "3xtf32", name="infer_8x64x56_bias_relu"),
        # Batched low-channel stem, the headline workload: forward, dX and dW.
        _named("conv_train", "stem_256x3x224", "3xtf32", name="stem_256x3x224_train"),
        # Wide layer, both precision modes a caller can choose on the tensor cores.
        _named("conv_train", "wide_128x256x56", "3xtf32", name="wide_128x256x56_train"),
        _named("conv_train", "wide_128x256x56", "tf32", name="wide_128x256x56_train_tf32"),
        # Downsampling layer.
        _named("conv_train", "down_128x128x112_s2", "3xtf32", name="down_128x128x112_s2_train"),
        # The small CNN, one whole training step through the graph.
        dict(kind="cnn_graph", n=workloads.CNN["batch"], c=3, hw=64, k1=32, k2=64, classes=workloads.CNN["fc_out"],
             mode="3xtf32", name="small_cnn_512_graph"),
        # Square products of the benchmark: forward and both gradients; the largest one forward in TF32.
        dict(kind="matmul_train", m=4096, k=4096, n=4096, mode="3xtf32", name="matmul_4096_train"),
        dict(kind="matmul_fwd", m=8192, k=8192, n=8192, mode="tf32", name="matmul_8192_tf32"),
        # Sizes that are no multiple of anything: a product and a layer.
        dict(kind="matmul_train", m=1021, k=2047, n=515, mode="3xtf32", name="matmul_1021x2047x515_train"),
        _conv("conv_train", 16, 35, 61, 45, 70, 5, 3, 2, 1, "3xtf32", name="conv_16x35x61x45_k70_5x3_train"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mode(rng):
    return "tf32" if rng.random() < 0.3 else "3xtf32"


def _draw_image_layer(rng, kind, mode):
    """First layers: up to four input channels, mostly 3x3 with stride 1, some larger filters with a stride."""
    r, stride = rng.choice([(3, 1), (3, 1), (3, 1), (3, 2), (5, 1), (7, 2)])
    h, w = _log(rng, 24, 256), _log(rng, 24, 256)
    if rng.random() < 0.5:
        h, w = max(8, h // 8 * 8), max(8, w // 8 * 8)
    case = _conv(kind, _log(rng, 1, 256), rng.choice([1, 2, 3, 3, 3, 4]), h, w, _log(rng, 8, 96), r, r, stride, r // 2, mode)
    # filters other than 3x3 / stride 1 are met on small batches
    return _shrink(case, 1e11 if (r, stride) == (3, 1) else 4e9)


def _draw_feature_layer(rng, kind, mode):
    """Hidden layers: 12 to 512 channels, half of the time a multiple of 16."""
    c, k = _log(rng, 12, 512), _log(rng, 12, 512)
    if rng.random() < 0.5:
        c, k = max(16, c // 16 * 16), max(16, k // 16 * 16)
    elif rng.random() < 0.5:
        c, k = max(12, c // 4 * 4), max(12, k // 4 * 4)
    r = rng.choice([1, 3, 3, 3, 3, 5])
    h, w = max(r, _log(rng, 7, 112)), max(r, _log(rng, 7, 112))
    case = _conv(kind, _log(rng, 1, 128), c, h, w, k, r, r, rng.choice([1, 1, 2]), rng.choice([r // 2, r // 2, 0]), mode)
    return _shrink(case, 4e11 if c % 4 == 0 and k % 4 == 0 and min(c, k) >= 16 else 1e10)


def _shrink(case, most):
    while work(case)["flops"] > most or work(case)["bytes"] > 2e9:
        if case["n"] > 1:
            case["n"] = max(1, case["n"] // 2)
        elif case["h"] > 2 * case["r"] and case["w"] > 2 * case["s"]:
            case["h"], case["w"] = case["h"] * 3 // 4, case["w"] * 3 // 4
        else:
            case["k"] = max(8, case["k"] // 2)
            if case["k"] == 8:
                break
    return case


def draw(rng):
    what, mode = rng.random(), _mode(rng)
    if what < 0.30:
        return _draw_feature_layer(rng, "conv_train", mode)
    if what < 0.40:
        return _draw_image_layer(rng, "conv_train", mode)
    if what < 0.50:
        case = _draw_feature_layer(rng, "conv_infer", mode)
        case["n"] = min(case["n"], 32)
        return case
    if what < 0.60:
        return _shrink(_draw_image_layer(rng, "conv_graph", mode), 4e9)
    if what < 0.70:
        return dict(kind="linear_graph", m=_log(rng, 4, 512), k=_log(rng, 16, 4096), n=rng.choice([1, 2, 10, 16, 33, 64, 100, 128]),
                    mode=mode)
    if what < 0.75:
        return dict(kind="cnn_graph", n=_log(rng, 8, 256), c=3, hw=rng.choice([28, 32, 36, 48, 64]), k1=rng.choice([16, 24, 32]),
                    k2=rng.choice([32, 48, 64]), classes=rng.choice([10, 10, 16]), mode=mode)
    m, k, n = (_log(rng, 48, 8192) for _ in range(3))
    if rng.random() < 0.6:
        m, k, n = (max(32, v // 32 * 32) for v in (m, k, n))
    aligned = k % 4 == 0 and n % 4 == 0
    while m * k * n > (1.2e11 if aligned else 4e9):
        m, k, n = (v // 64 * 32 if aligned else v // 2 + 1 if v == max(m, k, n) else v for v in (m, k, n))
    return dict(kind="matmul_train" if rng.random() < 0.7 else "matmul_fwd", m=m, k=k, n=n, mode=mode)


# ---------------------------------------------------------------------------
# sizes, work, tolerance
# ---------------------------------------------------------------------------
def _out_dims(case):
    return ((case["h"] + 2 * case["pad"] - case["r"]) // case["stride"] + 1,
            (case["w"] + 2 * case["pad"] - case["s"]) // case["stride"] + 1)


def _in_range_taps(size, out, taps, stride, pad):
    """Pairs (output position, filter tap) along one axis whose input position exists."""
    return sum(1 for o in range(out) for t in range(taps) if 0 <= o * stride + t - pad < size)


def _conv_macs(n, c, h, w, k, r, s, stride, pad):
    oh, ow = (h + 2 * pad - r) // stride + 1, (w + 2 * pad - s) // stride + 1
    return n * c * k * _in_range_taps(h, oh, r, stride, pad) * _in_range_taps(w, ow, s, stride, pad)


def _cnn_dims(case):
    out = (case["hw"] + 2 - 3) // 2 + 1
    return out, case["k2"] * out * out


def work(case):
    kind = case["kind"]
    if kind in ("conv_train", "conv_infer", "conv_graph"):
        oh, ow = _out_dims(case)
        x, w = case["n"] * case["c"] * case["h"] * case["w"], case["k"] * case["c"] * case["r"] * case["s"]
        y = case["n"] * case["k"] * oh * ow
        macs = _conv_macs(*(case[v] for v in ("n", "c", "h", "w", "k", "r", "s", "stride", "pad")))
        if kind == "conv_infer":
            return {"bytes": 4 * (x + w + case["k"] + y), "flops": 2 * macs}
        if kind == "conv_graph":  # the activations stay inside the pass, but it cannot do without storing them
            return {"bytes": 4 * (2 * x + 2 * w + 2 * y), "flops": 6 * macs + 4 * y}
        return {"bytes": 4 * (2 * x + 2 * w + 2 * y), "flops": 6 * macs}
    if kind in ("matmul_fwd", "matmul_train"):
        m, k, n = case["m"], case["k"], case["n"]
        passes = 1 if kind == "matmul_fwd" else 2
        return {"bytes": 4 * passes * (m * k + k * n + m * n), "flops": (2 if kind == "matmul_fwd" else 6) * m * k * n}
    if kind == "linear_graph":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": 4 * (2 * m * k + 4 * k * n + 3 * m * n), "flops": 6 * m * k * n + 4 * m * n + 2 * k * n}
    n, c, hw, k1, k2, classes = (case[v] for v in ("n", "c", "hw", "k1", "k2", "classes"))
    out, fc = _cnn_dims(case)
    macs = (_conv_macs(n, c, hw, hw, k1, 3, 3, 1, 1) + _conv_macs(n, k1, hw, hw, k2, 3, 3, 2, 1) + n * fc * classes)
    # per layer: its output written and read back, its gradient written and read back
    stored = n * (k1 * hw * hw + fc)
    return {"bytes": 4 * (2 * n * c * hw * hw + 4 * stored + 4 * fc * classes), "flops": 6 * macs}


def tolerance(case):
    # 3xTF32: two results that each hold the documented 1e-5 bar against the exact sums; TF32: one pass with
    # 11-bit significands, 2e-3 by the same documents
    return {"rel": 2e-5} if case["mode"] == "3xtf32" else {"rel": 3e-3}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _rand(gen, *shape, std=1.0):
    return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32).mul_(std)


def _uniform(gen, *shape, bound=1.0):
    return torch.rand(shape, generator=gen, device="cuda", dtype=torch.float32).mul_(2 * bound).sub_(bound)


def _tensor(values):
    """A leaf of the graph that already lives on the device."""
    return K.Tensor(values.cpu().numpy(), list(values.shape)).to_device()


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind, mode = case["kind"], case["mode"]
    state = {"case": case}
    if kind in ("conv_train", "conv_infer", "conv_graph"):
        n, c, h, w, k, r, s = (case[v] for v in ("n", "c", "h", "w", "k", "r", "s"))
        oh, ow = _out_dims(case)
        std = workloads.he_std(c * r * s)
        x = _uniform(gen, n, c, h, w) if c <= 4 else _rand(gen, n, c, h, w)  # images, or normalised activations
        wt = _rand(gen, k, c, r, s, std=std)
        if kind == "conv_graph":
            K.set_precision(MODES[mode])
            weights = _tensor(wt)
            state.update(x=_tensor(x), w=weights, layer=K.Conv2D.from_weights(weights, case["stride"], case["pad"]))
            return state
        ctx = _context(mode)
        dims = (n, c, h, w, k, r, s, case["stride"], case["pad"])
        state.update(ctx=ctx, dims=dims, x=x, w=wt, y=torch.empty(n, k, oh, ow, device="cuda"))
        if kind == "conv_infer":
            state["bias"] = _rand(gen, k, std=0.1)
            return state
        floats = ctx.conv2d_staged_floats(*dims)
        state.update(g=_rand(gen, n, k, oh, ow, std=0.01), dx=torch.empty_like(x), dw=torch.empty_like(wt),
                     staged=torch.empty(floats, device="cuda") if floats else None)
        return state
    if kind in ("matmul_fwd", "matmul_train"):
        m, k, n = case["m"], case["k"], case["n"]
        a, b = _rand(gen, m, k), _rand(gen, k, n, std=math.sqrt(1.0 / k))
        state.update(ctx=_context(mode), a=a, b=b, c=torch.empty(m, n, device="cuda"))
        if kind == "matmul_train":
            state.update(g=_rand(gen, m, n, std=0.01), da=torch.empty_like(a), db=torch.empty_like(b))
        return state
    K.set_precision(MODES[mode])
    if kind == "linear_graph":
        m, k, n = case["m"], case["k"], case["n"]
        state.update(x=_tensor(_rand(gen, m, k)), w=_tensor(_rand(gen, k, n, std=math.sqrt(1.0 / k))),
                     b=_tensor(_uniform(gen, m, n, bound=0.1)), lr=1e-3 / (m * n))
        return state
    n, c, hw, k1, k2, classes = (case[v] for v in ("n", "c", "hw", "k1", "k2", "classes"))
    _, fc = _cnn_dims(case)
    w1 = _tensor(_rand(gen, k1, c, 3, 3, std=workloads.he_std(9 * c)))
    w2 = _tensor(_rand(gen, k2, k1, 3, 3, std=workloads.he_std(9 * k1)))
    state.update(x=_tensor(_uniform(gen, n, c, hw, hw)), w1=w1, w2=w2, wfc=_tensor(_rand(gen, fc, classes, std=math.sqrt(1.0 / fc))),
                 b=_tensor(_uniform(gen, n, classes, bound=0.1)), fc=fc, lr=1e-9,
                 conv1=K.Conv2D.from_weights(w1, 1, 1), conv2=K.Conv2D.from_weights(w2, 2, 1))
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
class _DeviceArray:
    """A graph tensor's device buffer (values or gradient) as torch sees it; keeps its owner alive."""

    def __init__(self, owner, pointer, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f4", "data": (pointer, False), "version": 2}


def _values(t, shape):
    return torch.as_tensor(_DeviceArray(t, t.device_data(), shape), device="cuda")


def _grad(t, shape):
    return torch.as_tensor(_DeviceArray(t, t.device_grad(), shape), device="cuda")


def run(state):
    return _RUN[state["case"]["kind"]](state)


def _run_conv_train(st):
    ctx, dims = st["ctx"], st["dims"]
    x, w, y, g, dx, dw = (st[v].data_ptr() for v in ("x", "w", "y", "g", "dx", "dw"))
    staged = None
    if st["staged"] is not None:  # the layer's input staged once for its forward and backward
        staged = st["staged"].data_ptr()
        ctx.conv2d_stage(x, staged, *dims[:4])
    ctx.conv2d_fwd_staged(x, staged, w, None, y, *dims, 0)
    ctx.conv2d_bwd_staged(x, staged, w, g, None, 1.0, dx, dw, *dims, 0)
    return {"y": st["y"], "dx": st["dx"], "dw": st["dw"]}


def _run_conv_infer(st):
    st["ctx"].call("katsu_cuda_conv2d_fwd_bias_relu", st["x"].data_ptr(), st["w"].data_ptr(), st["bias"].data_ptr(),
                   st["y"].data_ptr(), *st["dims"], 1)
    return st["y"]


def _run_conv_graph(st):
    x, w = st["x"], st["w"]
    x.zero_grad(), w.zero_grad()
    y = st["layer"].forward(x)
    loss = y.mul(y).sum()
    loss.backward()
    c = st["case"]
    return {"loss": _values(loss, ()), "y": _values(y, (c["n"], c["k"], *_out_dims(c))),
            "dx": _grad(x, (c["n"], c["c"], c["h"], c["w"])), "dw": _grad(w, (c["k"], c["c"], c["r"], c["s"]))}


def _run_matmul_fwd(st):
    c = st["case"]
    st["ctx"].matmul_fwd(st["a"].data_ptr(), st["b"].data_ptr(), st["c"].data_ptr(), c["m"], c["k"], c["n"])
    return st["c"]


def _run_matmul_train(st):
    c, ctx = st["case"], st["ctx"]
    a, b = st["a"].data_ptr(), st["b"].data_ptr()
    ctx.matmul_fwd(a, b, st["c"].data_ptr(), c["m"], c["k"], c["n"])
    ctx.matmul_bwd(a, b, st["g"].data_ptr(), st["da"].data_ptr(), st["db"].data_ptr(), c["m"], c["k"], c["n"], 0)
    return {"c": st["c"], "da": st["da"], "db": st["db"]}


def _run_linear_graph(st):
    c, x, w, b = st["case"], st["x"], st["w"], st["b"]
    x.zero_grad(), w.zero_grad(), b.zero_grad()
    out = x.matmul(w).add(b)
    loss = out.mul(out).sum()
    loss.backward()
    w.sgd_step(st["lr"])
    return {"loss": _values(loss, ()), "out": _values(out, (c["m"], c["n"])), "dx": _grad(x, (c["m"], c["k"])),
            "dw": _grad(w, (c["k"], c["n"])), "db": _grad(b, (c["m"], c["n"])), "w": _values(w, (c["k"], c["n"]))}


def _run_cnn_graph(st):
    c, x, w1, w2, wfc, b = st["case"], st["x"], st["w1"], st["w2"], st["wfc"], st["b"]
    leaves = (x, w1, w2, wfc, b)
    for t in leaves:
        t.zero_grad()
    h = st["conv2"].forward(st["conv1"].forward(x))
    out = h.reshape([c["n"], st["fc"]]).matmul(wfc).add(b)
    loss = out.mul(out).sum()
    loss.backward()
    for t in (w1, w2, wfc):
        t.sgd_step(st["lr"])
    shapes = ((c["n"], c["c"], c["hw"], c["hw"]), (c["k1"], c["c"], 3, 3), (c["k2"], c["k1"], 3, 3), (st["fc"], c["classes"]),
              (c["n"], c["classes"]))
    grads = [_grad(t, s) for t, s in zip(leaves, shapes)]
    return {"loss": _values(loss, ()), "out": _values(out, shapes[4]), "grads": grads,
            "weights": [_values(t, s) for t, s in zip((w1, w2, wfc), shapes[1:4])]}


_RUN = {"conv_train": _run_conv_train, "conv_infer": _run_conv_infer, "conv_graph": _run_conv_graph,
        "matmul_fwd": _run_matmul_fwd, "matmul_train": _run_matmul_train, "linear_graph": _run_linear_graph,
        "cnn_graph": _run_cnn_graph}
