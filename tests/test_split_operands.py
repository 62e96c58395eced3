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


# Parts of an operand far below the rest that no run of 128 neighbours in memory is made of: the error of the outputs that
# depend on that part alone.  Sizes at which the part lies inside the first tile of the magnitude pass and in its last,
# ragged one, rows short and long, aligned and not.
@pytest.mark.parametrize("size", [(300, 700, 515), (515, 516, 512), (2000, 100, 600), (420, 33, 3100)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("scale", [1e-6, 1e-8, 1e-12])
def test_small_rows_and_columns_of_matrices(ctx, oracle, size, scale):
    m, k, n = size
    rng = np.random.default_rng(11)
    whole = [rng.standard_normal(v).astype(np.float32) for v in ((m, k), (k, n), (m, n))]
    for mode, bar in BARS:
        ctx.set_precision(mode)
        try:
            # operand, its small row or column, the output that it reaches alone, at which row or column of it
            for which, axis, output in ((0, 0, 0), (0, 1, 2), (1, 0, 1), (1, 1, 0), (2, 0, 1), (2, 1, 2)):
                operands = [v.copy() for v in whole]
                length = operands[which].shape[axis]
                for at in (3, length - 1):
                    operands[which] = whole[which].copy()
                    part = (at, slice(None)) if axis == 0 else (slice(None), at)
                    operands[which][part] *= np.float32(scale)
                    a, b, g = operands
                    a64, b64, g64 = (v.astype(np.float64) for v in operands)
                    want = (a64 @ b64, g64 @ b64.T, a64.T @ g64)[output]
                    with DeviceArrays(ctx, a=a, b=b, g=g) as d:
                        d.alloc("out", want.size, fill=np.nan)
                        if output == 0:
                            ctx.matmul_fwd(d["a"], d["b"], d["out"], m, k, n)
                        else:
                            da, db = (d["out"], None) if output == 1 else (None, d["out"])
                            ctx.matmul_bwd(d["a"], d["b"], d["g"], da, db, m, k, n, 0)
                        got = d.get("out").reshape(want.shape)
                    # an output row for a small row of a or g and a small column of a (row of db) or row of b (column of da)
                    out_axis = {(0, 0): 0, (0, 1): 0, (1, 0): 1, (1, 1): 1, (2, 0): 0, (2, 1): 1}[which, axis]
                    part = (at, slice(None)) if out_axis == 0 else (slice(None), at)
                    assert rel_l2(got[part], want[part]) <= bar, (mode, which, axis, at)
        finally:
            ctx.set_precision(0)


@pytest.mark.parametrize("shape", [(4, 48, 7, 7, 40, 3, 3, 1, 1), (3, 33, 14, 15, 30, 3, 3, 1, 1), (4, 64, 12, 12, 64, 1, 1, 1, 0), (6, 3, 40, 40, 24, 5, 5, 2, 2),
                                   (200, 64, 1, 1, 128, 1, 1, 1, 0)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("scale", [1e-6, 1e-8, 1e-12])
def test_small_channels_and_regions(ctx, oracle, shape, scale):
    n, c, h, w, k, r, s, stride, pad = shape
    oh, ow = oracle.conv_out_dims(h, w, r, s, stride, pad)
    xs, ws, gs = (n, c, h, w), (k, c, r, s), (n, k, oh, ow)
    rng = np.random.default_rng(12)
    whole = [rng.standard_normal(v).astype(np.float32) for v in (xs, ws, gs)]
    every = slice(None)
    dim = (every, every, every, slice(0, max(0, (w // 2 - s + pad) // stride + 1)))  # outputs whose window lies in the left half
    parts = [(0, (every, c - 1), 2, (every, c - 1)), (0, (1,), 0, (1,)), (0, (every, every, every, slice(0, w // 2)), 0, dim),
             (1, (every, 2), 1, (every, 2)), (1, (k - 1,), 0, (every, k - 1)), (2, (every, 5), 2, (5,)), (2, (n - 1,), 1, (n - 1,))]
    for mode, bar in BARS:
        ctx.set_precision(mode)
        try:
            for which, part, output, reached in parts:
                if which == 0 and len(part) == 4 and w == 1:
                    continue
                t = [v.copy() for v in whole]
                t[which][part] *= np.float32(scale)
                x, wt, g = (v.reshape(-1) for v in t)
                y64 = oracle.conv2d_forward_f64(x, wt, list(xs), list(ws), stride, pad)
                dx64, dw64 = oracle.conv2d_backward_f64(x, wt, g, list(xs), list(ws), stride, pad)
                want = (y64.reshape(gs), dx64.reshape(xs), dw64.reshape(ws))[output]
                with DeviceArrays(ctx, x=x, w=wt, g=g) as d:
                    d.alloc("out", want.size, fill=np.nan)
                    if output == 0:
                        ctx.conv2d_fwd(d["x"], d["w"], d["out"], *shape)
                    else:
                        dx, dw = (d["out"], None) if output == 1 else (None, d["out"])
                        ctx.conv2d_bwd(d["x"], d["w"], d["g"], dx, dw, *shape, 0)
                    got = d.get("out").reshape(want.shape)
                assert rel_l2(got[reached], want[reached]) <= bar, (mode, which, part)
        finally:
            ctx.set_precision(0)


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


def kinds(values):
    """0 a number, 1 and 2 the infinities, 3 NaN."""
    values = np.asarray(values).reshape(-1)
    return np.where(np.isnan(values), 3, np.where(values == np.inf, 1, np.where(values == -np.inf, 2, 0)))


# Strides 1 to 3 on both sides of 32 input channels, output channels that are and are not a multiple of 16 when rounded to 8;
# layers of few or odd channels, whose padding and shared products must not show either; split and unsplit contractions
NON_FINITE = [(2, 20, 24, 28, 40, 3, 3, 2, 1), (2, 40, 24, 28, 24, 3, 3, 2, 1), (2, 40, 25, 31, 40, 3, 3, 3, 1), (1, 40, 16, 18, 40, 4, 4, 2, 1),
              (2, 24, 24, 26, 40, 1, 1, 2, 0), (1, 64, 30, 30, 64, 3, 3, 1, 1), (3, 17, 22, 24, 23, 3, 3, 1, 1), (3, 17, 32, 34, 23, 3, 3, 2, 1),
              (2, 3, 20, 22, 24, 5, 5, 2, 2), (2, 150, 9, 9, 75, 3, 3, 1, 1), (16, 33, 28, 28, 50, 3, 3, 1, 0)]


@pytest.mark.parametrize("shape", NON_FINITE, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("mode", [0, 1], ids=["3xtf32", "tf32"])
def test_infinities_and_nans_reach_exactly_their_results(ctx, oracle, mode, shape):
    """As f32 multiply-adds over a result's own terms have them.  Regular layers (channels from 16 on in multiples of 4) are held
    to that for an x or g that is no number; in padded rows and columns a weight that is none reaches their results as NaN."""
    n, c, h, w, k, r, s, stride, pad = shape
    xs, ws = [n, c, h, w], [k, c, r, s]
    oh, ow = oracle.conv_out_dims(h, w, r, s, stride, pad)
    regular = c >= 16 and k >= 16 and c % 4 == 0 and k % 4 == 0
    rng = np.random.default_rng(sum(shape))
    whole = {name: np.rint(rng.standard_normal(v) * 4).astype(np.float32) + np.float32(0.5)  # few bits, no zero
             for name, v in (("x", n * c * h * w), ("w", k * c * r * s), ("g", n * k * oh * ow))}
    bias = rng.standard_normal(k).astype(np.float32)
    ctx.set_precision(mode)
    try:
        for which in "xwg":
            for value in (np.inf, np.nan, None):
                t = {name: v.copy() for name, v in whole.items()}
                if value is None:
                    t[which][t[which].size // 3], t[which][-1] = np.inf, -np.inf
                else:
                    t[which][t[which].size // 3] = value
                with np.errstate(all="ignore"):
                    y = oracle.conv2d_forward_f64(t["x"], t["w"], xs, ws, stride, pad).reshape(-1)
                    dx, dw = (v.reshape(-1) for v in oracle.conv2d_backward_f64(t["x"], t["w"], t["g"], xs, ws, stride, pad))
                    by_channel = np.repeat(np.tile(bias, n), oh * ow)
                    relu = np.fmax(y + by_channel, 0)  # (a NaN is cut off)
                with DeviceArrays(ctx, x=t["x"], w=t["w"], g=t["g"], b=bias, dx2=np.ones(dx.size, np.float32), dw2=np.ones(dw.size, np.float32)) as d:
                    for name, size in (("y", y.size), ("relu", y.size), ("dx", dx.size), ("dw", dw.size)):
                        d.alloc(name, size, fill=7.0)
                    ctx.conv2d_fwd(d["x"], d["w"], d["y"], *shape)
                    ctx.conv2d_fwd_staged(d["x"], None, d["w"], d["b"], d["relu"], *shape, 1)
                    ctx.conv2d_bwd(d["x"], d["w"], d["g"], d["dx"], d["dw"], *shape, 0)
                    ctx.conv2d_bwd(d["x"], d["w"], d["g"], d["dx2"], d["dw2"], *shape, 1)
                    results = [("y", y), ("relu", relu), ("dx", dx), ("dx2", dx + 1), ("dw", dw), ("dw2", dw + 1)]
                    if regular:
                        results = {"x": results[:2], "w": [], "g": results[2:4]}[which]
                    for name, want in results:
                        got = d.get(name)
                        assert np.array_equal(kinds(got), kinds(want)), (name, which, value)
                        numbers = np.isfinite(want)
                        assert rel_l2(got[numbers], want[numbers]) <= BARS[mode][1], (name, which, value)
    finally:
        ctx.set_precision(0)


@pytest.mark.parametrize("size", [(200, 520, 648), (401, 333, 517), (260, 6000, 260)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("mode", [0, 1], ids=["3xtf32", "tf32"])
def test_infinities_and_nans_in_matrices(ctx, oracle, mode, size):
    m, k, n = size
    rng = np.random.default_rng(m)
    whole = [np.rint(rng.standard_normal(v) * 4).astype(np.float32) + np.float32(0.5) for v in ((m, k), (k, n), (m, n))]
    ctx.set_precision(mode)
    try:
        for which in range(3):
            for value in (np.inf, np.nan):
                operands = [v.copy() for v in whole]
                operands[which].reshape(-1)[1234] = value
                a, b, g = operands
                with np.errstate(all="ignore"):
                    want = [v.reshape(-1) for v in (oracle.matmul_f64(a, b, m, k, n), *oracle.matmul_backward_f64(a, b, g, m, k, n))]
                with DeviceArrays(ctx, a=a, b=b, g=g) as d:
                    d.alloc("c", m * n), d.alloc("da", m * k), d.alloc("db", k * n)
                    ctx.matmul_fwd(d["a"], d["b"], d["c"], m, k, n)
                    ctx.matmul_bwd(d["a"], d["b"], d["g"], d["da"], d["db"], m, k, n, 0)
                    for name, w in zip(("c", "da", "db"), want):
                        assert np.array_equal(kinds(d.get(name)), kinds(w)), (name, which, value)
    finally:
        ctx.set_precision(0)


@pytest.mark.parametrize("mode", [0, 1], ids=["3xtf32", "tf32"])
def test_a_held_copy_beside_an_infinite_weight(ctx, oracle, mode):
    """x's copy, fp16 or bf16 planes, was made before the call and knows nothing of w: the call makes planes of its own."""
    shape = (2, 32, 12, 14, 40, 3, 3, 1, 0)
    n, c, h, w, k, r, s, stride, pad = shape
    rng = np.random.default_rng(8)
    x, wt = (np.rint(rng.standard_normal(v) * 4).astype(np.float32) + np.float32(0.5) for v in (n * c * h * w, k * c * 9))
    wt[700] = np.inf
    ctx.set_precision(mode)
    try:
        for scale in (1.0, 2.0 ** -60):
            x[:x.size // n] *= np.float32(scale)
            with np.errstate(all="ignore"):
                want = oracle.conv2d_forward_f64(x, wt, [n, c, h, w], [k, c, 3, 3], 1, 0).reshape(-1)
            with DeviceArrays(ctx, x=x, w=wt) as d:
                d.alloc("y", want.size), d.alloc("copy", ctx.conv2d_staged_floats(*shape))
                ctx.conv2d_stage(d["x"], d["copy"], n, c, h, w)
                ctx.conv2d_fwd_staged(d["x"], d["copy"], d["w"], None, d["y"], *shape, 0)
                assert np.array_equal(kinds(d.get("y")), kinds(want)), scale
    finally:
        ctx.set_precision(0)


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


# What a 3xTF32 result may lose to the tensor core's accumulation, beside the 22 bits of its operands (6e-8): a step truncates
# the sum by 2e-8 of it on average, and 12 steps (3 products) of 64 terms go to an accumulator before it is added to f32 sums,
# 24 or 36.  Taken small products first, 4 of the first 12 count.  Measured: 1.5e-7, 2.6e-7, 4.8e-7 and 7e-7.
FINE, ONE, TWO, THREE = 6e-8 + 4 * 4e-8, 6e-8 + 12 * 2.5e-8, 6e-8 + 24 * 2.5e-8, 6e-8 + 36 * 2.5e-8


@pytest.mark.parametrize("size, bars", [((333, 1001, 777), (TWO, ONE, ONE)), ((2050, 67, 1030), (FINE, TWO, TWO)), ((200, 300, 3001), (ONE, TWO, FINE)),
                                        ((1024, 128, 512), (TWO, THREE, REL_L2_TOL)), ((512, 512, 512), (THREE, THREE, THREE))], ids=str)
def test_accumulation_error_of_products(ctx, oracle, size, bars):
    m, k, n = size
    rng = np.random.default_rng(m)
    a, b, g = (rng.standard_normal(v).astype(np.float32) for v in ((m, k), (k, n), (m, n)))
    a64, b64, g64 = (v.astype(np.float64) for v in (a, b, g))
    with DeviceArrays(ctx, a=a, b=b, g=g) as d:
        d.alloc("c", m * n), d.alloc("da", m * k), d.alloc("db", k * n)
        ctx.matmul_fwd(d["a"], d["b"], d["c"], m, k, n)
        ctx.matmul_bwd(d["a"], d["b"], d["g"], d["da"], d["db"], m, k, n, 0)
        errors = rel_l2(d.get("c"), a64 @ b64), rel_l2(d.get("da"), g64 @ b64.T), rel_l2(d.get("db"), a64.T @ g64)
    assert all(e <= bar for e, bar in zip(errors, bars)), (errors, bars)


@pytest.mark.parametrize("shape, bars", [((4, 35, 31, 25, 70, 5, 3, 2, 1), (ONE, ONE, FINE)), ((4, 3, 40, 40, 32, 5, 5, 1, 2), (FINE, TWO, FINE)),
                                         ((2, 129, 14, 14, 67, 3, 3, 1, 1), (TWO, ONE, FINE)), ((4, 32, 32, 32, 64, 3, 3, 2, 1), (THREE, THREE, TWO)),
                                         ((8, 96, 14, 14, 96, 1, 1, 1, 0), (TWO, TWO, TWO))], ids=str)
def test_accumulation_error_of_layers(ctx, oracle, shape, bars):
    n, c, h, w, k, r, s, stride, pad = shape
    oh, ow = oracle.conv_out_dims(h, w, r, s, stride, pad)
    rng = np.random.default_rng(sum(shape))
    x, wt, g = (rng.standard_normal(v).astype(np.float32) for v in (n * c * h * w, k * c * r * s, n * k * oh * ow))
    errors = conv_errors(ctx, oracle, shape, x, wt, g)
    assert all(e <= bar for e, bar in zip(errors, bars)), (errors, bars)


@pytest.mark.parametrize("c, s", [(65536, 32), (65536, 64)])
def test_filter_rows_of_millions_of_products(ctx, c, s):
    """32 768 and 65 536 k-blocks to a filter row: the largest that the path takes, past what 16 bits count."""
    k = 2
    shape = (1, c, 1, s, k, 1, s, 1, 0)
    rng = np.random.default_rng(c + s)
    x, wt, g = (rng.standard_normal(v).astype(np.float32) for v in (c * s, k * c * s, k))
    x64, w64, g64 = x.astype(np.float64), wt.astype(np.float64).reshape(k, -1), g.astype(np.float64)
    with DeviceArrays(ctx, x=x, w=wt, g=g) as d:
        d.alloc("y", k, fill=np.nan), d.alloc("dx", x.size, fill=np.nan), d.alloc("dw", wt.size, fill=np.nan)
        ctx.conv2d_fwd(d["x"], d["w"], d["y"], *shape)
        ctx.conv2d_bwd(d["x"], d["w"], d["g"], d["dx"], d["dw"], *shape, 0)
        assert rel_l2(d.get("y"), w64 @ x64) <= REL_L2_TOL
        assert rel_l2(d.get("dx"), g64 @ w64) <= REL_L2_TOL
        assert rel_l2(d.get("dw"), np.outer(g64, x64)) <= REL_L2_TOL


@pytest.mark.parametrize("factor", [1e-3, 1.0, 1e6])
def test_upstream_factor_beside_tiny_operands(ctx, oracle, factor):
    """Operand scales of 2^61 and a factor below 1: their product is no normal f32 although the results are."""
    shape = (2, 32, 14, 14, 40, 3, 3, 1, 1)
    n, c, h, w, k, r, s, stride, pad = shape
    rng = np.random.default_rng(3)
    x, wt, g = ((rng.standard_normal(v) * 1.2e-15).astype(np.float32) for v in (n * c * h * w, k * c * 9, n * k * h * w))
    dx64, dw64 = oracle.conv2d_backward_f64(x, wt, g, [n, c, h, w], [k, c, 3, 3], stride, pad)
    scale = 0.75 * factor
    with DeviceArrays(ctx, x=x, w=wt, g=g, scale=np.array([0.75], np.float32)) as d:
        d.alloc("dx", x.size), d.alloc("dw", wt.size)
        ctx.conv2d_bwd_staged(d["x"], None, d["w"], d["g"], d["scale"], factor, d["dx"], d["dw"], *shape, 0)
        assert rel_l2(d.get("dx") / 1e-30, dx64 * scale / 1e-30) <= REL_L2_TOL
        assert rel_l2(d.get("dw") / 1e-30, dw64 * scale / 1e-30) <= REL_L2_TOL
