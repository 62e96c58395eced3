// Convolution on the fp16 tensor-core kernel (operands: f16_split.cuh, kernel and operand views: f16_gemm.cu).
//
//   forward : lanes output pixels, columns output channels   (conv2d.rs:95-103, 232-262)
//   dX      : lanes input pixels of one stride-parity class at a time, columns input channels: pixel (s jy + py,
//             s jx + px) receives only the taps with (p + pad - tap) divisible by s, which along x are neighbours in g,
//             so their window is one run as well; all classes of a tile run one after the other on the same blocks,
//             which puts the halves of every 32-byte sector of dX into L2 within microseconds of each other
//   dW      : lanes (ky, kx, c), columns output channels, contraction over pixels cut into splits   (conv2d.rs:269-292)
//
// Any channel count: staging pads channels to 8, and the window view makes k-blocks out of S * channels.
#include "f16_gemm.cuh"
#include "launch.cuh"

namespace {

constexpr int STAGED_GAP = 2;              // zero pixels between the rows of a copy of x that the caller holds
constexpr size_t STAGED_HEADER = 256;      // bytes in front of it: its KatsuF16Info

struct Shape {
    size_t n, c, h, w, k, r, s, stride, pad, oh, ow;
};

// Sizes within the tensor maps' and the kernel's index ranges.
bool geometry_ok(const katsu_cuda_ctx *ctx, const Shape &g) {
    if (ctx->precision == KATSU_MODE_FP32 || ctx->f16_state == nullptr) return false;
    if (g.r > (size_t)KATSU_F16_MAX_ROWS || g.s > 64 || g.stride > (size_t)KATSU_F16_MAX_CLASSES || g.pad > 1024) return false;
    if (g.n > 65535 || g.h > 32767 || g.w > 32767 || g.oh > 32767 || g.ow > 32767) return false;
    if (g.c > 65536 || g.k > 65536) return false;
    // a staged row has at most pad + filter width zero pixels
    const size_t gap = g.pad + g.s;
    return g.n * g.h * (g.w + gap) < 0x7fffffff && g.n * g.oh * (g.ow + gap) < 0x7fffffff && g.h * g.w < 0x3fffffff;
}

// At least 16 channels on both sides, in multiples of 4.
bool regular(const Shape &g) {
    return g.c >= 16 && g.k >= 16 && g.c % 4 == 0 && g.k % 4 == 0 && g.n * g.oh * g.ow >= 64;
}

// Where the passes in front pay against the direct kernels.  The three launches take about 18 us whatever the size.  A direct
// kernel's time is one thread's chain of c * r * s (dX: k * r * s) multiply-adds: at 16 channels and 3 x 3 already 39 us forward
// and 45 us dX (16 x 8 x 8, 150 000 multiply-adds; 18.6 and 18.5 us here), so regular layers come here at any size.  Others
// do from 1e6 multiply-adds on.
bool worth_it(const Shape &g) {
    return regular(g) || double(g.n) * g.oh * g.ow * double(g.k) * g.c * g.r * g.s >= 1e6;
}

// Whether forward and dW read x through a copy that the caller holds: regular layers whose padding the gaps between the
// copy's rows provide.
bool takes_copy(const katsu_cuda_ctx *ctx, const Shape &g) {
    return geometry_ok(ctx, g) && regular(g) && g.pad <= (size_t)STAGED_GAP;
}

// A staged tensor: its planes start at pixel (0, 0) of image 0; element pitches.
struct Staged {
    KatsuF16Planes planes;
    size_t cp, gap, h, w, n;
    size_t row() const { return (w + gap) * cp; }
    size_t image() const { return h * row(); }
};

size_t staged_halves(size_t n, size_t c, size_t h, size_t w, size_t gap, size_t tail) {
    return katsu_round_up((gap + n * h * (w + gap)) * katsu_round_up(c, 8) + tail, 128);
}

Staged staged_at(void *base, size_t n, size_t c, size_t h, size_t w, size_t gap, size_t tail) {
    Staged p;
    p.cp = katsu_round_up(c, 8);
    p.gap = gap;
    p.n = n; p.h = h; p.w = w;
    p.planes.base = static_cast<__half *>(base) + gap * p.cp;
    p.planes.stride = staged_halves(n, c, h, w, gap, tail);
    return p;
}

size_t staged_bytes(const katsu_cuda_ctx *ctx, size_t n, size_t c, size_t h, size_t w, size_t gap, size_t tail) {
    return staged_halves(n, c, h, w, gap, tail) * sizeof(__half) * (katsu_f16_narrow_planes(ctx) + 1);
}

KatsuStageJob nhwc_job(const float *src, const Staged &p, size_t c, size_t tail, const KatsuF16Info *info) {
    KatsuStageJob j = {};
    j.kind = KATSU_STAGE_NHWC;
    j.src = src;
    j.to = p.planes;
    j.info = info;
    j.n = (int)p.n; j.c = (int)c; j.h = (int)p.h; j.w = (int)p.w;
    j.gap = (int)p.gap; j.cp = (int)p.cp; j.tail = (int)tail;
    return j;
}

KatsuStageJob weights_job(const float *w, const KatsuF16Planes &to, const Shape &g, size_t cp, size_t width, const KatsuF16Info *info) {
    KatsuStageJob j = {};
    j.kind = KATSU_STAGE_WEIGHTS;
    j.src = w;
    j.to = to;
    j.info = info;
    j.c = (int)g.c; j.cp = (int)cp; j.k = (int)g.k; j.r = (int)g.r; j.s = (int)g.s;
    j.h = j.w = 1;
    j.width = (int)width;
    return j;
}

// The caller's staged copy of x.  False when the call has none, or is of a shape that uses none: what the pointer then
// refers to was never written.
bool held_x(const katsu_cuda_ctx *ctx, const Shape &g, const KatsuF16Info **info, Staged *out) {
    if (ctx->x_prestaged == nullptr || !takes_copy(ctx, g)) return false;
    char *base = const_cast<char *>(reinterpret_cast<const char *>(ctx->x_prestaged));
    *info = reinterpret_cast<const KatsuF16Info *>(base);
    *out = staged_at(base + STAGED_HEADER, g.n, g.c, g.h, g.w, STAGED_GAP, 0);
    return true;
}

// x as the window operand of forward and dW.
bool x_window_maps(const katsu_cuda_ctx *ctx, CUtensorMap *maps, const Staged &x, const Shape &g, const KatsuF16Box &box,
                   bool pairs) {
    return katsu_f16_window_maps(maps, x.planes, -(long long)(g.pad * x.cp), katsu_f16_narrow_planes(ctx) + 1, g.s * x.cp, g.ow,
                                 g.h, g.n, g.stride * x.cp, x.row(), x.image(), (int)g.stride, 64, box, pairs);
}

// The taps of dX by parity class.
struct Classes {
    int row_begin[KATSU_F16_MAX_CLASSES + 1];
    short off_h[KATSU_F16_MAX_ROWS], ky[KATSU_F16_MAX_ROWS];
    int taps_x[KATSU_F16_MAX_CLASSES], off_x[KATSU_F16_MAX_CLASSES], kx_last[KATSU_F16_MAX_CLASSES];
    int lower_h, first_x, most_rel_x, most_taps;
    int span_h, span_x;  // rows and columns of g that the pixels (s jy + py, s jx + px) of one (jy, jx) receive from
    size_t grid_h, grid_w, left, right;  // zero pixels that g's rows need on either side
};

int floor_div(int a, int b) { return a >= 0 ? a / b : -((-a + b - 1) / b); }

Classes classes_of(const Shape &g) {
    Classes q = {};
    const int st = (int)g.stride, pad = (int)g.pad;
    q.grid_h = katsu_div_up(g.h, g.stride);
    q.grid_w = katsu_div_up(g.w, g.stride);
    q.lower_h = 0x7fff;
    int rows = 0;
    for (int py = 0; py < st; ++py) {
        q.row_begin[py] = rows;
        for (int ky = 0; ky < (int)g.r; ++ky) {
            const int t = py + pad - ky;
            if (((t % st) + st) % st != 0) continue;
            q.off_h[rows] = (short)floor_div(t, st);
            q.ky[rows] = (short)ky;
            if (q.off_h[rows] < q.lower_h) q.lower_h = q.off_h[rows];
            ++rows;
        }
    }
    q.row_begin[st] = rows;
    for (int i = 0; i < rows; ++i) {
        q.off_h[i] = (short)(q.off_h[i] - q.lower_h);
        if (q.off_h[i] >= q.span_h) q.span_h = q.off_h[i] + 1;
    }
    q.first_x = 0x7fff;
    int last_x = -0x7fff;
    for (int px = 0; px < st; ++px) {
        for (int kx = (int)g.s - 1; kx >= 0; --kx) {  // falling kx: rising offset
            const int t = px + pad - kx;
            if (((t % st) + st) % st != 0) continue;
            if (q.taps_x[px]++ == 0) {
                q.off_x[px] = floor_div(t, st);
                q.kx_last[px] = kx;
            }
        }
        if (q.taps_x[px] == 0) continue;
        if (q.off_x[px] < q.first_x) q.first_x = q.off_x[px];
        if (q.off_x[px] + q.taps_x[px] - 1 > last_x) last_x = q.off_x[px] + q.taps_x[px] - 1;
        if (q.taps_x[px] > q.most_taps) q.most_taps = q.taps_x[px];
    }
    for (int px = 0; px < st; ++px) {
        if (q.taps_x[px] == 0) q.off_x[px] = q.first_x;
        if (q.off_x[px] - q.first_x > q.most_rel_x) q.most_rel_x = q.off_x[px] - q.first_x;
    }
    q.span_x = last_x - q.first_x + 1;
    q.left = q.first_x < 0 ? (size_t)-q.first_x : 0;
    const int right = (int)q.grid_w - 1 + last_x - (int)(g.ow - 1);
    q.right = right > 0 ? (size_t)right : 0;
    return q;
}

// Where results have to be summed again that meet an infinity or NaN and a product that is not theirs (f16_exact.cuh): for layers
// that can run on the direct kernels, which have no such products, and where the classes of a strided dX share products.
KatsuF16Raw raw_of(KatsuF16Raw::Form form, const float *a, const float *b, const Shape &g, bool shared, const float *gscale, float gfactor) {
    KatsuF16Raw q = {};
    q.form = shared || !regular(g) ? form : KatsuF16Raw::NONE;
    q.a = a;
    q.b = b;
    q.n = (int)g.n; q.c = (int)g.c; q.h = (int)g.h; q.w = (int)g.w; q.k = (int)g.k; q.r = (int)g.r; q.s = (int)g.s;
    q.stride = (int)g.stride; q.pad = (int)g.pad; q.oh = (int)g.oh; q.ow = (int)g.ow;
    q.gscale = gscale;
    q.gfactor = gfactor;
    return q;
}

void pixel_fields(KatsuF16Problem *p, const Shape &g, const KatsuF16Box &box) {
    p->n_img = (int)g.n;
    p->gfactor = 1.f;
    p->classes_y = p->classes_x = 1;
    p->step = 1;
    p->bw = box.bw; p->bh = box.bh; p->nb = box.nb;
    p->blocks_x = box.blocks_x; p->blocks_y = box.blocks_y;
    p->blocks = box.blocks;
    p->a_bytes = box.bw * box.bh * box.nb * 128;
}

}  // namespace

size_t katsu_f16_conv_staged_bytes(const katsu_cuda_ctx *ctx, size_t n, size_t c, size_t h, size_t w) {
    return STAGED_HEADER + staged_bytes(ctx, n, c, h, w, STAGED_GAP, 0);
}

int32_t katsu_f16_conv_stage(katsu_cuda_ctx *ctx, const float *x, void *staged, size_t n, size_t c, size_t h, size_t w) {
    katsu_f16_new_call(ctx);
    KatsuF16Info *info = katsu_f16_slot(ctx, KATSU_INFO_A);
    const Staged p = staged_at(static_cast<char *>(staged) + STAGED_HEADER, n, c, h, w, STAGED_GAP, 0);
    const KatsuAmaxJob amax = katsu_amax_planes(x, n, c, h * w, info);
    KATSU_TRY(katsu_f16_amax(ctx, &amax, 1));
    KatsuStageJob job = nhwc_job(x, p, c, 0, info);
    job.info_copy = static_cast<KatsuF16Info *>(staged);
    return katsu_f16_stage(ctx, katsu_f16_call(ctx, info, nullptr, nullptr), &job, 1);
}

bool katsu_f16_conv_takes_copy(const katsu_cuda_ctx *ctx, size_t n, size_t c, size_t h, size_t w, size_t k, size_t r,
                               size_t s, size_t stride, size_t pad, size_t oh, size_t ow) {
    return takes_copy(ctx, Shape{n, c, h, w, k, r, s, stride, pad, oh, ow});
}

int32_t katsu_f16_conv_fwd(katsu_cuda_ctx *ctx, const float *x, const float *w, const float *bias, int relu, float *y,
                           size_t n, size_t c, size_t h, size_t wd, size_t k, size_t r, size_t s, size_t stride, size_t pad,
                           size_t oh, size_t ow, int *handled) {
    *handled = 0;
    const Shape g = {n, c, h, wd, k, r, s, stride, pad, oh, ow};
    if (!geometry_ok(ctx, g) || !worth_it(g)) return KATSU_OK;
    const int planes = katsu_f16_narrow_planes(ctx) + 1;
    const size_t cp = katsu_round_up(c, 8), width = s * cp, chunks = katsu_div_up(width, 64);
    katsu_f16_new_call(ctx);
    KatsuF16Info *ix = katsu_f16_slot(ctx, KATSU_INFO_A), *iw = katsu_f16_slot(ctx, KATSU_INFO_B);
    const KatsuF16Info *info = ix;
    Staged held;
    const bool prestaged = held_x(ctx, g, &info, &held);
    const size_t out_count = n * oh * ow * k;
    const KatsuF16Box box = katsu_f16_box(128, false, (int)stride, ow, oh, n);
    if (box.blocks > 0x7fffffff) return katsu_f16_drop_call(ctx);
    const KatsuF16Plan plan = katsu_f16_plan(ctx, KATSU_F16_CONV, box.blocks * 128, (int)k, (long long)(r * chunks), double(out_count));
    KatsuArena arena = {nullptr, 0};
    for (int pass = 0; pass < 2; ++pass) {  // the first only adds up the sizes
        if (pass) {
            float *base = nullptr;
            if (katsu_scratch(ctx, arena.bytes / 4, &base) != KATSU_OK) return katsu_f16_drop_call(ctx);  // no room: the other kernels
            arena = {reinterpret_cast<char *>(base), 0};
        }
        // (room for x also when the caller holds a copy: a narrow copy is of no use to a wide call)
        void *xs = arena.take(staged_bytes(ctx, n, c, h, wd, pad, 0));
        const KatsuF16Planes ws = arena.planes(r * k * width, planes);
        float *partial = plan.splits > 1 ? arena.floats(size_t(plan.splits) * out_count) : nullptr;
        if (!pass) continue;
        const Staged own = staged_at(xs, n, c, h, wd, pad, 0);
        KatsuF16Maps maps;
        if (!x_window_maps(ctx, maps.a, prestaged ? held : own, g, box, false) ||
            (prestaged && !x_window_maps(ctx, maps.a_second, own, g, box, false)) ||
            !katsu_f16_rows_maps(maps.b, ws, planes, width, k, r, width, k * width, plan.bn / 2))
            return katsu_f16_drop_call(ctx);
        *handled = 1;
        const KatsuF16Call call = katsu_f16_call(ctx, info, iw, nullptr);
        KatsuAmaxJob amax[2] = {katsu_amax_matrix(w, k, c * r * s, iw), katsu_amax_planes(x, n, c, h * wd, ix)};
        KATSU_TRY(katsu_f16_amax(ctx, amax, prestaged ? 1 : 2));
        KatsuStageJob jobs[2] = {nhwc_job(x, own, c, 0, info), weights_job(w, ws, g, cp, width, iw)};
        jobs[0].only_if_mixed = prestaged ? 1 : 0;
        KATSU_TRY(katsu_f16_stage(ctx, call, jobs, 2));
        KatsuF16Problem p = {};
        pixel_fields(&p, g, box);
        p.out = y;
        p.raw = raw_of(KatsuF16Raw::FORWARD, x, w, g, false, nullptr, 1.f);
        p.bias = bias;
        p.relu = relu;
        p.call = call;
        p.info_a = info;
        p.info_b = iw;
        p.a_second = prestaged ? 1 : 0;
        p.m_total = box.blocks * 128;
        p.n_total = (int)k;
        p.f32_terms = regular(g) ? 0 : (long long)(c * r * s);
        p.col_stride = (long long)(oh * ow);
        p.row_begin[1] = (int)r;
        for (size_t i = 0; i < r; ++i) p.off_h[i] = p.b_row[i] = (short)i;
        p.chunks[0] = (int)chunks;
        p.steps_last[0] = (short)katsu_div_up(width - 64 * (chunks - 1), 16);
        p.in_step = (int)stride;
        p.lower_h = -(int)pad;
        p.out_h = (int)oh; p.out_w = (int)ow;
        p.img_stride = (long long)(k * oh * ow);
        KATSU_TRY(katsu_f16_launch(ctx, KATSU_F16_CONV, maps, p, plan, partial, (long long)out_count));
        if (plan.splits > 1)
            KATSU_TRY(katsu_f16_fold(ctx, p.raw, partial, y, out_count, plan.splits, 0, bias, k, oh * ow, relu));
    }
    return KATSU_OK;
}

namespace {

// dw[k][c][ky][kx] (+)= sum over splits of partial[split][k][(ky, column group, column)].  A
// block handles 32 elements in the partials' order, eight thread groups each add every eighth split.
__global__ void __launch_bounds__(256)
f16_dw_fold_kernel(const __grid_constant__ KatsuF16Raw raw, const float *__restrict__ partial, float *dw, int k, int c, int r, int s, int cp, int groups_per_row, int splits, int accumulate) {
    __shared__ float sums[8][32];
    launch_next();
    launch_wait();
    const size_t lanes = size_t(r) * groups_per_row * 64, elems = lanes * k;
    const size_t j = size_t(blockIdx.x) * 32 + (threadIdx.x & 31);
    const int part = threadIdx.x >> 5;
    float v = 0.f;
    if (j < elems)
#pragma unroll 4
        for (int q = part; q < splits; q += 8) v += __ldg(partial + size_t(q) * elems + j);
    sums[part][threadIdx.x & 31] = v;
    __syncthreads();
    if (part != 0 || j >= elems) return;
    float total = sums[0][threadIdx.x];
#pragma unroll
    for (int q = 1; q < 8; ++q) total += sums[q][threadIdx.x];
    const int o = int(j / lanes), m = int(j - size_t(o) * lanes);
    const int ky = m / (groups_per_row * 64), col = m - ky * groups_per_row * 64;
    const int kx = col / cp, cc = col - kx * cp;
    if (kx >= s || cc >= c) return;
    if (raw.form != KatsuF16Raw::NONE && !katsu_is_number(total) && katsu_f16_mixed(raw, ky, kx)) total = katsu_f16_exact(raw, o, cc, ky, kx);
    float *dst = dw + ((size_t(o) * c + cc) * r + ky) * s + kx;
    *dst = accumulate ? *dst + total : total;
}

}  // namespace

int32_t katsu_f16_conv_bwd(katsu_cuda_ctx *ctx, const float *x, const float *w, const float *gr, const float *gscale,
                           float gfactor, float *dx, float *dw, size_t n, size_t c, size_t h, size_t wd, size_t k, size_t r,
                           size_t s, size_t stride, size_t pad, size_t oh, size_t ow, int accumulate,
                           int *handled) {
    *handled = 0;
    const Shape g = {n, c, h, wd, k, r, s, stride, pad, oh, ow};
    if (!geometry_ok(ctx, g) || !worth_it(g)) return KATSU_OK;
    const Classes q = classes_of(g);
    const int planes = katsu_f16_narrow_planes(ctx) + 1;
    const size_t cp = katsu_round_up(c, 8), kp = katsu_round_up(k, 8);
    const size_t gap = q.left > q.right ? q.left : q.right;
    const size_t tail = katsu_round_up((size_t(q.most_taps) + q.most_rel_x + 2) * kp + 64, 8);
    katsu_f16_new_call(ctx);
    KatsuF16Info *ix = katsu_f16_slot(ctx, KATSU_INFO_A), *iw = katsu_f16_slot(ctx, KATSU_INFO_B), *ig = katsu_f16_slot(ctx, KATSU_INFO_G);
    const KatsuF16Info *info = ix;
    Staged held;
    const bool prestaged = dw != nullptr && held_x(ctx, g, &info, &held);

    // dX: columns of the weights by x-parity class
    KatsuF16Problem pd = {};
    const KatsuF16Box box_dx = katsu_f16_box(128, false, 1, q.grid_w, q.grid_h, n);
    pixel_fields(&pd, g, box_dx);
    // At stride 2 the pixels of an x-parity pair are stored together (store_pairs).  With few input channels all four classes
    // are columns of one contraction over the span_h x span_x pixels of g they receive from, with zero weights where a class
    // has no tap: those pixels are then loaded once and not once per class and tap, and a tile is one pass of the pipeline
    // instead of four short ones.  The zeros cost the tensor pipe (16 tap products for 9 at 3 x 3), so the line is where the
    // columns of all classes fit 128, whose products take no longer than their operands' fill: 32 channels.  With more, the
    // two classes of a pair run one after the other on tiles of at most 128 columns and the sums of both are held.
    const size_t class_cols = 2 * katsu_round_up(c, 16);
    const bool merged = stride == 2 && class_cols <= 64;
    int width = 0;
    for (size_t i = 0; i < (merged ? 1 : stride); ++i) {
        const int cols = (merged ? q.span_x : q.taps_x[i]) * (int)kp;
        pd.b_col[i] = width;
        pd.chunks[i] = (cols + 63) / 64;
        pd.steps_last[i] = (short)((cols - 64 * (pd.chunks[i] - 1) + 15) / 16);
        pd.off_w[i] = merged ? 0 : (short)(q.off_x[i] - q.first_x);
        width += pd.chunks[i] * 64;
    }
    long long kb_dx = 0;
    if (merged) kb_dx = (long long)q.span_h * pd.chunks[0];
    else
        for (size_t py = 0; py < stride; ++py)
            for (size_t px = 0; px < stride; ++px) kb_dx += (long long)(q.row_begin[py + 1] - q.row_begin[py]) * pd.chunks[px];
    const size_t dx_columns = merged ? 2 * class_cols : c, dx_planes = merged ? (size_t)q.span_h : r;
    const size_t dx_count = n * c * h * wd;
    const KatsuF16Plan plan_dx = katsu_f16_plan(ctx, KATSU_F16_CONV, box_dx.blocks * 128, (int)dx_columns, kb_dx, double(dx_count),
                                                stride == 2 ? 128 : 256);
    // dW
    const size_t gpr = katsu_div_up(s * cp, (size_t)64), dw_lanes = r * gpr * 64, dw_count = dw_lanes * k;
    const KatsuF16Box box_dw = katsu_f16_box(64, true, (int)stride, ow, oh, n);
    const long long kb_dw = box_dw.blocks;
    if (box_dx.blocks > 0x7fffffff || box_dw.blocks > 0x7fffffff) return katsu_f16_drop_call(ctx);
    const KatsuF16Plan plan_dw = katsu_f16_plan(ctx, KATSU_F16_CONV_DW, (long long)dw_lanes, (int)k, kb_dw, double(dw_count));

    // dW: two 64-column groups to a load, where no pair of groups holds padding or parts of two filter rows.  A load costs the
    // copy unit about 150 clocks whatever it brings, and with four to a k-block of 512 pipe clocks they set the pace in TF32
    // mode (256 x 256 channels, 128 x 56 x 56: 623 -> 449 us).
    const bool a_pairs = (s * cp) % 128 == 0, b_pairs = plan_dw.bn == 256 && kp % 64 == 0;

    KatsuArena arena = {nullptr, 0};
    for (int pass = 0; pass < 2; ++pass) {
        if (pass) {
            float *base = nullptr;
            if (katsu_scratch(ctx, arena.bytes / 4, &base) != KATSU_OK) return katsu_f16_drop_call(ctx);
            arena = {reinterpret_cast<char *>(base), 0};
        }
        void *gs = arena.take(staged_bytes(ctx, n, k, oh, ow, gap, tail));
        void *xs = dw ? arena.take(staged_bytes(ctx, n, c, h, wd, pad, 0)) : nullptr;
        const KatsuF16Planes ws = dx ? arena.planes(dx_planes * dx_columns * width, planes) : KatsuF16Planes{nullptr, 0};
        float *partial_dx = dx && plan_dx.splits > 1 ? arena.floats(size_t(plan_dx.splits) * dx_count) : nullptr;
        float *partial_dw = dw ? arena.floats(size_t(plan_dw.splits) * dw_count) : nullptr;
        if (!pass) continue;
        const Staged sg = staged_at(gs, n, k, oh, ow, gap, tail), own = staged_at(xs, n, c, h, wd, pad, 0);
        KatsuF16Maps md, mw;
        if (dx && (!katsu_f16_window_maps(md.a, sg.planes, q.first_x * (long long)kp, planes,
                                          size_t(merged ? q.span_x : q.most_taps) * kp, q.grid_w + (merged ? 0 : q.most_rel_x), oh, n, kp, sg.row(), sg.image(), 1, 64, box_dx) ||
                   !katsu_f16_rows_maps(md.b, ws, planes, width, dx_columns, dx_planes, width, dx_columns * width, plan_dx.bn / 2)))
            return katsu_f16_drop_call(ctx);
        if (dw && (!x_window_maps(ctx, mw.a, prestaged ? held : own, g, box_dw, a_pairs) ||
                   (prestaged && !x_window_maps(ctx, mw.a_second, own, g, box_dw, a_pairs)) ||
                   !katsu_f16_window_maps(mw.b, sg.planes, 0, planes, kp, ow, oh, n, kp, sg.row(), sg.image(), 1,
                                          plan_dw.bn >= 128 ? 64 : 32, box_dw, b_pairs)))
            return katsu_f16_drop_call(ctx);
        *handled = 1;
        KatsuF16Call call = katsu_f16_call(ctx, ig, dx ? iw : nullptr, dw ? info : nullptr);
        call.gscale = gscale;
        call.gfactor = gfactor;
        KatsuAmaxJob amax[3];
        KatsuStageJob jobs[3];
        int na = 0, nj = 0;
        amax[na++] = katsu_amax_planes(gr, n, k, oh * ow, ig);
        jobs[nj++] = nhwc_job(gr, sg, k, tail, ig);
        if (dw) {
            if (!prestaged) amax[na++] = katsu_amax_planes(x, n, c, h * wd, ix);
            jobs[nj] = nhwc_job(x, own, c, 0, info);
            jobs[nj++].only_if_mixed = prestaged ? 1 : 0;
        }
        if (dx) {
            amax[na++] = katsu_amax_matrix(w, k, c * r * s, iw);
            KatsuStageJob &jw = jobs[nj++];
            jw = weights_job(w, ws, g, kp, width, iw);
            jw.backward = merged ? 2 : 1;
            jw.classes = jw.stride = (int)stride;
            jw.class_cols = (int)class_cols;
            jw.span_h = q.span_h; jw.span_x = q.span_x;
            jw.lower_h = q.lower_h; jw.first_x = q.first_x;
            jw.pad = (int)pad;
            for (size_t i = 0; i < (merged ? 0 : stride); ++i) {
                jw.col_begin[i] = pd.b_col[i];
                jw.kx_last[i] = q.kx_last[i];
                jw.class_taps[i] = q.taps_x[i];
            }
        }
        KATSU_TRY(katsu_f16_amax(ctx, amax, na));
        KATSU_TRY(katsu_f16_stage(ctx, call, jobs, nj));
        if (dx) {
            KatsuF16Problem &p = pd;
            p.out = dx;
            p.accumulate = accumulate;
            p.call = call;
            p.info_a = ig;
            p.info_b = iw;
            // (the last 16-wide step of a class of fewer taps reaches into the next pixel where kp is no multiple of 16)
            p.raw = raw_of(KatsuF16Raw::DX, gr, w, g, merged || (stride > 1 && kp % 16 != 0), gscale, gfactor);
            p.gscale = gscale;
            p.gfactor = gfactor;
            p.m_total = box_dx.blocks * 128;
            p.f32_terms = regular(g) ? 0 : (long long)katsu_div_up(k * r * s, stride * stride);
            p.n_total = (int)c;
            p.col_stride = (long long)(h * wd);
            p.step = (int)stride;
            if (merged) {
                p.class_cols = (int)class_cols;
                p.row_begin[1] = q.span_h;
                for (int i = 0; i < q.span_h; ++i) p.off_h[i] = p.b_row[i] = (short)i;
            } else {
                p.classes_y = p.classes_x = (int)stride;
                p.pair_x = stride == 2 ? 1 : 0;
                for (size_t i = 0; i <= stride; ++i) p.row_begin[i] = q.row_begin[i];
                for (int i = 0; i < q.row_begin[stride]; ++i) {
                    p.off_h[i] = q.off_h[i];
                    p.b_row[i] = q.ky[i];
                }
            }
            p.in_step = 1;
            p.lower_h = q.lower_h;
            p.out_h = (int)h; p.out_w = (int)wd;
            p.img_stride = (long long)(c * h * wd);
            KATSU_TRY(katsu_f16_launch(ctx, stride == 2 ? KATSU_F16_CONV_DX2 : KATSU_F16_CONV, md, p, plan_dx, partial_dx, (long long)dx_count));
            if (plan_dx.splits > 1)
                KATSU_TRY(katsu_f16_fold(ctx, p.raw, partial_dx, dx, dx_count, plan_dx.splits, accumulate, nullptr, 1, 1, 0));
        }
        if (dw) {
            KatsuF16Problem p = {};
            pixel_fields(&p, g, box_dw);
            p.a_bytes = 2 * 64 * 128;
            p.call = call;
            p.info_a = info;
            p.info_b = ig;
            p.a_second = prestaged ? 1 : 0;
            p.gscale = gscale;
            p.gfactor = gfactor;
            p.m_total = (long long)dw_lanes;
            p.f32_terms = regular(g) ? 0 : 1;  // the direct kernel's sums over pixels are split into short ones
            p.n_total = (int)k;
            p.col_stride = (long long)dw_lanes;
            p.in_step = (int)stride;
            p.lower_h = -(int)pad;
            p.groups = (int)(r * gpr);
            p.groups_per_row = (int)gpr;
            p.a_pairs = a_pairs;
            p.b_pairs = b_pairs;
            KATSU_TRY(katsu_f16_launch(ctx, KATSU_F16_CONV_DW, mw, p, plan_dw, partial_dw, (long long)dw_count));
            KATSU_TRY(katsu_prepare_kernel(ctx, (const void *)f16_dw_fold_kernel, 0));
            KATSU_TRY(katsu_launch_chained(ctx, f16_dw_fold_kernel, (unsigned)katsu_div_up(dw_count, (size_t)32), 256, 0, 1,
                                           raw_of(KatsuF16Raw::DW, x, gr, g, false, gscale, gfactor), partial_dw, dw, (int)k, (int)c, (int)r, (int)s, (int)cp, (int)gpr, plan_dw.splits,
                                           accumulate));
        }
    }
    return KATSU_OK;
}
