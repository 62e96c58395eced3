"""The fp16 / bf16 operand planes of the tensor-core path at the sizes and values where they can go wrong: channel counts
around the padding to 8 and the 64-wide k-blocks, ragged pixel boxes, filters wider than tall, strides larger than the
filter, contractions short and long enough for one and for several accumulator drains and splits; and values whose
range fp16 cannot hold, which the same kernels take as bf16 planes.

The bars are the documented ones (1e-5, 2e-3).  For the range cases the error is also measured on the small part alone:
with two fp16 planes under one scale a part 1e9 below the rest would come out as zeros (relative error 1)."""
import numpy as np
import pytest

from parity_util import REL_L2_TOL, DeviceArrays, rel_l2

pytestmark = pytest.mark.gpu

BARS = ((0, REL_L2_TOL), (1, 2e-3))

CONV = [(2, 7, 19, 23, 31, 3, 3, 1, 1), (1, 9, 33, 17, 33, 5, 5, 2, 2), (3, 21, 10, 12, 65, 1, 7, 1, 3), (2, 22, 29, 31, 130, 7, 1, 3, 0),
        (4, 33, 13, 13, 40, 2, 2, 3, 1), (17, 3, 21, 21, 24, 7, 7, 2, 3), (1, 136, 8, 8, 264, 3, 3, 1, 1), (2, 3, 20, 22, 9, 5, 5, 1, 4)]


def conv_errors(ctx, oracle, shape, x, wt, g, staged=False, small=None):
    n, c, h, w, k, r, s, stride, pad = shape
    xs, ws = [n, c, h, w], [k, c, r, s]
    y64 = oracle.conv2d_forward_f64(x, wt, xs, ws, stride, pad)
    dx64, dw64 = oracle.conv2d_backward_f64(x, wt, g, xs, ws, stride, pad)
    with DeviceArrays(ctx, x=x, w=wt, g=g) as d:
        for name, size in (("y", g.size), ("dx", x.size), ("dw", wt.size)):
            d.alloc(name, size, fill=np.nan)
        copy = None
        if staged:
            copy = d.alloc("copy", ctx.conv2d_staged_floats(*shape))
            ctx.conv2d_stage(d["x"], copy, n, c, h, w)
        ctx.conv2d_fwd_staged(d["x"], copy, d["w"], None, d["y"], *shape, 0)
        ctx.conv2d_bwd_staged(d["x"], copy, d["w"], d["g"], None, 1.0, d["dx"], d["dw"], *shape, 0)
        y, dx, dw = d.get("y"), d.get("dx"), d.get("dw")
    errors = [rel_l2(y, y64), rel_l2(dx, dx64), rel_l2(dw, dw64)]
    if small == "x":
        errors.append(rel_l2(y[:y.size // n], y64.reshape(-1)[:y.size // n]))
    if small == "g":
        errors.append(rel_l2(dx[:dx.size // n], dx64.reshape(-1)[:dx.size // n]))
    return errors


@pytest.mark.parametrize("shape", CONV, ids=lambda s: "x".join(map(str, s)))
def test_convolution_edges(ctx, oracle, shape):
    n, c, h, w, k, r, s, stride, pad = shape
    oh, ow = oracle.conv_out_dims(h, w, r, s, stride, pad)
    rng = np.random.default_rng(sum(shape))
    x, wt, g = (rng.standard_normal(v).astype(np.float32) for v in (n * c * h * w, k * c * r * s, n * k * oh * ow))
    for mode, bar in BARS:
        ctx.set_precision(mode)
        try:
            errors = conv_errors(ctx, oracle, shape, x, wt, g)
        finally:
            ctx.set_precision(0)
        assert max(errors) <= bar, (shape, mode, errors)


# Strides: dX of all four parity classes in one contraction (at most 32 channels at stride 2) and just past that line, x pairs
# stored together and, with odd widths, apart; filters that leave a class without taps, that are not square, that reach over
# several pixels of g; dW with one and with two column groups to a load.
STRIDED = [(3, 32, 15, 18, 40, 3, 3, 2, 1), (2, 17, 16, 16, 24, 1, 1, 2, 0), (2, 33, 16, 18, 40, 3, 3, 2, 1), (3, 20, 16, 13, 130, 5, 3, 2, 2),
           (2, 4, 18, 30, 20, 7, 7, 2, 3), (5, 12, 2, 40, 24, 3, 3, 2, 1), (2, 140, 14, 11, 24, 3, 3, 2, 1), (2, 24, 18, 21, 40, 3, 3, 3, 1),
           (2, 40, 15, 11, 24, 4, 4, 3, 2), (2, 128, 12, 10, 192, 3, 3, 2, 1)]


@pytest.mark.parametrize("shape", STRIDED, ids=lambda s: "x".join(map(str, s)))
def test_strided_edges(ctx, oracle, shape):
    """Both modes, and dX added to what is there."""
    n, c, h, w, k, r, s, stride, pad = shape
    oh, ow = oracle.conv_out_dims(h, w, r, s, stride, pad)
    rng = np.random.default_rng(sum(shape))
    x, wt, g = (rng.standard_normal(v).astype(np.float32) for v in (n * c * h * w, k * c * r * s, n * k * oh * ow))
    before = rng.standard_normal(x.size).astype(np.float32)
    dx64 = oracle.conv2d_backward_f64(x, wt, g, [n, c, h, w], [k, c, r, s], stride, pad)[0].reshape(-1) + before
    for mode, bar in BARS:
        ctx.set_precision(mode)
        try:
            errors = conv_errors(ctx, oracle, shape, x, wt, g)
            with DeviceArrays(ctx, x=x, w=wt, g=g, dx=before) as d:
                ctx.conv2d_bwd(d["x"], d["w"], d["g"], d["dx"], None, *shape, accumulate=1)
                errors.append(rel_l2(d.get("dx"), dx64))
        finally:
            ctx.set_precision(0)
        assert max(errors) <= bar, (shape, mode, errors)


# more tiles of 64 x 64 or 32 channels x 128 pixels than staging blocks run at a time (5 to an SM; one to an SM for the copy
# of x beside the caller's), pixels a multiple of 4 and not
@pytest.mark.parametrize("shape", [(12, 70, 47, 45, 24, 1, 1, 1, 0), (12, 70, 48, 45, 24, 1, 1, 1, 0), (48, 28, 47, 45, 24, 1, 1, 1, 0)],
                         ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("staged", [False, True], ids=["plain", "staged"])
def test_staging_blocks_take_several_tiles(ctx, oracle, shape, staged):
    n, c, h, w, k = shape[:5]
    if staged:
        shape = (n, c // 4 * 4, *shape[2:])  # what the caller can stage
        c = shape[1]
    rng = np.random.default_rng(n + c)
    x, wt, g = (rng.standard_normal(v).astype(np.float32) for v in (n * c * h * w, k * c, n * k * h * w))
    if staged:
        g[:g.size // n] *= np.float32(1e-9)  # wide: the copy beside the caller's is written
    assert max(conv_errors(ctx, oracle, shape, x, wt, g, staged, "g" if staged else None)) <= REL_L2_TOL


@pytest.mark.parametrize("staged", [False, True], ids=["plain", "staged"])
@pytest.mark.parametrize("small", ["x", "g"])
def test_one_image_far_below_the_others(ctx, oracle, small, staged):
    """x (or g) of image 0 is 1e9 smaller than the rest: one call's operands are then bf16 planes, also when only g is
    wide and the caller's staged copy of x is not."""
    shape = (3, 24, 18, 20, 48, 3, 3, 1, 1)
    n, c, h, w, k = shape[:5]
    rng = np.random.default_rng(5)
    x, wt, g = (rng.standard_normal(v).astype(np.float32) for v in (n * c * h * w, k * c * 9, n * k * h * w))
    part = x if small == "x" else g
    part[:part.size // n] *= np.float32(1e-9)
    for mode, bar in BARS:
        ctx.set_precision(mode)
        try:
            errors = conv_errors(ctx, oracle, shape, x, wt, g, staged, small)
        finally:
            ctx.set_precision(0)
        assert max(errors) <= bar, (small, staged, mode, errors)


@pytest.mark.parametrize("scale", [1e-30, 1e-5, 1e25])
def test_magnitudes_of_whole_tensors(ctx, oracle, scale):
    """A common factor of a whole operand, up to where its fp16 scale would leave f32."""
    m, k, n = 130, 1100, 75
    rng = np.random.default_rng(6)
    a = (rng.standard_normal(m * k) * scale).astype(np.float32)
    b, g = (rng.standard_normal(v).astype(np.float32) for v in (k * n, m * n))
    c64 = oracle.matmul_f64(a, b, m, k, n)
    da64, db64 = oracle.matmul_backward_f64(a, b, g, m, k, n)
    for mode, bar in BARS:
        ctx.set_precision(mode)
        try:
            with DeviceArrays(ctx, a=a, b=b, g=g) as d:
                d.alloc("c", m * n, fill=np.nan), d.alloc("da", m * k, fill=np.nan), d.alloc("db", k * n, fill=np.nan)
                ctx.matmul_fwd(d["a"], d["b"], d["c"], m, k, n)
                ctx.matmul_bwd(d["a"], d["b"], d["g"], d["da"], d["db"], m, k, n, 0)
                errors = (rel_l2(d.get("c"), c64), rel_l2(d.get("da"), da64), rel_l2(d.get("db"), db64))
        finally:
            ctx.set_precision(0)
        assert max(errors) <= bar, (scale, mode, errors)


@pytest.mark.parametrize("mode", [0, 1], ids=["3xtf32", "tf32"])
def test_non_finite_values_reach_exactly_their_outputs(ctx, oracle, mode):
    shape = (2, 20, 12, 14, 40, 3, 3, 1, 1)
    n, c, h, w, k = shape[:5]
    rng = np.random.default_rng(8)
    x, wt = rng.standard_normal(n * c * h * w).astype(np.float32), rng.standard_normal(k * c * 9).astype(np.float32)
    x[5 * h * w + 40], x[(c + 3) * h * w] = np.inf, np.nan
    y64 = oracle.conv2d_forward_f64(x, wt, [n, c, h, w], [k, c, 3, 3], 1, 1).reshape(-1)
    ctx.set_precision(mode)
    try:
        with DeviceArrays(ctx, x=x, w=wt) as d:
            d.alloc("y", n * k * h * w)
            ctx.conv2d_fwd(d["x"], d["w"], d["y"], *shape)
            y = d.get("y")
    finally:
        ctx.set_precision(0)
    finite = np.isfinite(y64)
    assert not finite.all() and np.array_equal(np.isfinite(y), finite)
    assert rel_l2(y[finite], y64[finite]) <= BARS[mode][1]


@pytest.mark.parametrize("shape", [(1, 16, 8, 8, 16, 3, 3, 1, 1), (1, 16, 14, 14, 24, 3, 3, 1, 1), (2, 24, 13, 13, 32, 3, 3, 2, 1)],
                         ids=lambda s: "x".join(map(str, s)))
def test_small_regular_layers_stay_on_the_tensor_cores(ctx, oracle, shape):
    """Below 1e6 multiply-adds too: a direct kernel's chain of c * r * s multiply-adds takes two to three times as long."""
    n, c, h, w, k, r, s, stride, pad = shape
    oh, ow = oracle.conv_out_dims(h, w, r, s, stride, pad)
    rng = np.random.default_rng(sum(shape))
    x, wt, g = (rng.standard_normal(v).astype(np.float32) for v in (n * c * h * w, k * c * r * s, n * k * oh * ow))
    with DeviceArrays(ctx, x=x, w=wt) as d:
        d.alloc("y", g.size)
        before = ctx.launch_count()
        ctx.conv2d_fwd(d["x"], d["w"], d["y"], *shape)
        assert ctx.launch_count() - before >= 3  # magnitudes, planes, product; a direct kernel is one launch
    assert max(conv_errors(ctx, oracle, shape, x, wt, g)) <= REL_L2_TOL
