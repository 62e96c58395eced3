// Operands of the fp16 tensor-core path: f32 tensors as one or two fp16 planes with a common power-of-two scale.
//
// A tensor v is held as v * 2^exp ~ hi + lo with hi = fp16(v * 2^exp) and lo = fp16(v * 2^exp - hi), both rounded to
// nearest; exp places the largest magnitude in [2^14, 2^15).  hi alone carries the 11 significand bits of TF32, hi + lo
// carry 22, what the two TF32 parts of 3xTF32 carry (there both parts are truncated), and the tensor core multiplies
// fp16 at twice the rate of TF32 from half the bytes.  Products of fp16 values are exact in the f32 accumulator, and
// 2^-(exp_a + exp_b) is applied to the f32 sums, so the scale itself costs no rounding.
//
// What fp16 lacks is range.  Below 2^-14 it goes subnormal: an element's error never exceeds 2^-25 of the scaled
// range = 2^-39 of the tensor's largest magnitude (so one plane has its 11 bits down to 2^-28 of it).  An output that
// depends on small elements alone (a column of b, an input channel of w, a dim region of an image) would lose what TF32
// parts keep, so the pass that finds the largest magnitude also finds the SMALLEST maximum over groups of elements that
// are not all zero, along both axes of the tensor: up to 128 neighbours in a row, and up to 16 rows of a column (a row of
// a matrix, of weights [k][c * r * s], or a channel's plane of an image).  A tensor counts as narrow only if every group's
// maximum is within 2^17 of the tensor's (two planes) or 2^28 (one plane): then no element's error exceeds 2^-22 (2^-11)
// of the largest magnitude around it in its row, and in its column.  Within such a neighbourhood of 16 x 128 elements of
// mixed sizes the small ones do have fewer bits than TF32 parts would give them.  (Groups of single elements would keep
// those too, but every normally distributed tensor of more than a few thousand elements holds one below 2^-17.)
//
// If one operand of a call has a wider range, or holds infinities or NaNs, all of the call's operands are written as
// bf16 planes instead: each the leading 8 significand bits of what the planes before it left, three of them (two in
// TF32 mode), no scale.  bf16 has the exponents of f32, and three planes hold all 24 bits.  The products kept are
// those down to 2^-16 (six; three in TF32 mode).  The choice is made on the device, by every kernel of the call from the
// same KatsuF16Info values; no value crosses to the host.  Such calls take about twice the time in 3xTF32 mode (4096^3 685 us
// against 366, 256 channels 128 x 56 x 56 forward 2193 against 1206, 64 channels 8 x 56 x 56 39 against 29) and in TF32 mode
// (396 against 182, 1263 against 712, 31 against 25): the products, and three (two) planes of operand fill for two (one).
// TF32 parts, which have f32's range, take 600 / 2045 / 40 and 202 / 857 / 34 us on the same layers, wide or not.
//
// In a call with an infinity or NaN every plane but the last is cut strictly below the value, so that each part of a nonzero
// value is nonzero and of its sign, and an infinity is one in every plane: its products with the other operand's parts are
// then all the infinity of the product, where 0 * inf would be NaN.
#pragma once

#include <cuda_fp16.h>

#include "common.cuh"

// What the magnitude pass finds of an operand, as f32 bit patterns: the largest magnitude, and 0x7fffffff minus the
// smallest maximum of a group (so that both grow from zero and both are plain atomic maxima).
struct KatsuF16Info {
    unsigned most, inverted_least;
};

// The operands of one call (unused entries null) and the range that counts as narrow in its mode: 2^span.
struct KatsuF16Call {
    const KatsuF16Info *info[3];
    int span;
    // factors of the results, of a call whose first operand meets the others
    const float *gscale;  // device scalar or null
    float gfactor;
};

// 2^-48 .. 2^48 keeps the product of two operands' scales inside f32.
__device__ __forceinline__ bool katsu_f16_narrow(KatsuF16Info info, int span) {
    const int top = int(info.most >> 23), low = int((0x7fffffffu - info.inverted_least) >> 23);
    return info.most == 0 || (top >= 127 - 48 && top <= 127 + 48 && top - low < span);
}

__device__ __forceinline__ int katsu_f16_exp(KatsuF16Info info) {  // of a narrow operand
    return info.most == 0 ? 0 : 14 - (int(info.most >> 23) - 127);
}

__device__ __forceinline__ KatsuF16Info katsu_f16_load(const KatsuF16Info *info) {
    const uint2 v = *reinterpret_cast<const uint2 *>(info);
    return KatsuF16Info{v.x, v.y};
}

__device__ __forceinline__ bool katsu_f16_wide(const KatsuF16Call &call) {
    KatsuF16Info v[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) v[i] = call.info[i] ? katsu_f16_load(call.info[i]) : KatsuF16Info{0, 0};
    if (!(katsu_f16_narrow(v[0], call.span) && katsu_f16_narrow(v[1], call.span) && katsu_f16_narrow(v[2], call.span))) return true;
    if (call.gscale == nullptr && call.gfactor == 1.f) return false;
    // The sums are multiplied by the factors and the operands' scales as one f32, which has to be a normal number.
    const float factor = call.gscale ? call.gfactor * __ldg(call.gscale) : call.gfactor;
    const int e = int((__float_as_uint(factor) >> 23) & 255) - 127, e0 = katsu_f16_exp(v[0]), e1 = katsu_f16_exp(v[1]), e2 = katsu_f16_exp(v[2]);
    return e - e0 - max(e1, e2) < -100 || e - e0 - min(e1, e2) > 100;
}

__device__ __forceinline__ bool katsu_f16_finite(KatsuF16Info info) { return info.most < 0x7f800000u; }
__device__ __forceinline__ bool katsu_f16_finite(const KatsuF16Call &call) {
    unsigned most = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i)
        if (call.info[i]) most = max(most, katsu_f16_load(call.info[i]).most);
    return most < 0x7f800000u;
}

// Whether a wide call needs planes of its own for an operand of which a copy has been made by itself: the copy holds fp16
// planes, or planes that are not made to stand beside an infinity.
__device__ __forceinline__ bool katsu_f16_own_copy(const KatsuF16Call &call, KatsuF16Info info) {
    return katsu_f16_narrow(info, call.span) || (katsu_f16_finite(info) && !katsu_f16_finite(call));
}

// One operand whose magnitude is to be found: matrices [images][rows][cols], none of the sizes 0.
struct KatsuAmaxJob {
    const float *src;
    unsigned images, rows, cols;
    bool columns;  // groups along columns too
    KatsuF16Info *info;
};

static inline KatsuAmaxJob katsu_amax_matrix(const float *src, size_t rows, size_t cols, KatsuF16Info *info) {
    return {src, 1, (unsigned)rows, (unsigned)cols, true, info};
}

// An image tensor [n][c][pixels]; without pixels beside each other a matrix [n][c].  With one channel a group along a
// column would be a single pixel.
static inline KatsuAmaxJob katsu_amax_planes(const float *src, size_t n, size_t c, size_t pixels, KatsuF16Info *info) {
    if (pixels == 1) return katsu_amax_matrix(src, n, c, info);
    return {src, (unsigned)n, (unsigned)c, (unsigned)pixels, c > 1, info};
}

enum KatsuStageKind { KATSU_STAGE_NHWC, KATSU_STAGE_ROWS, KATSU_STAGE_WEIGHTS };

// Fp16 planes of a tensor: plane i starts i * stride elements behind the first.  Room for one more than the mode's
// narrow form needs.
struct KatsuF16Planes {
    __half *base;
    size_t stride;
};

// One operand to be written as planes.
//   NHWC     src [n][c][h * w] -> [n][h][w + gap][cp], channels padded with zeros to cp (a multiple of 8), `gap` zero
//            pixels behind every row and in front of the first; `tail` more zero elements behind the last row.
//            (n = 1, h = 1, gap = 0 is a transposed matrix.)
//   ROWS     src [n][c] -> [n][cp]
//   WEIGHTS  src [k][c][r][s] -> [r][rows][width]; backward = 0: rows are k and column kx * cp + c is tap kx;
//            backward = 1: rows are c and the columns of x-parity class j start at col_begin[j], tap t of the class
//            (kx = kx_last[j] - t * stride) holding cp columns, channel k innermost;
//            backward = 2 (stride 2): -> [span_h][(py, c, px)][width], class_cols rows to a py, column t * cp + k of a row in
//            plane dy is tap (py + pad - 2 * (lower_h + dy), px + pad - 2 * (first_x + t)), zero where there is no such tap.
struct KatsuStageJob {
    int kind;
    const float *src;
    KatsuF16Planes to;
    const KatsuF16Info *info;
    KatsuF16Info *info_copy;  // where to leave a copy of it, or null
    int only_if_mixed;  // 1: a copy of this operand exists already; written only when the call is wide and cannot use it
    int n, c, h, w, gap, cp, tail;
    int k, r, s, width, backward, classes, stride;
    int col_begin[8], kx_last[8], class_taps[8];
    int class_cols, span_h, span_x, pad, lower_h, first_x;  // backward = 2
};

// Largest magnitude and usability of up to three operands, one launch.
int32_t katsu_f16_amax(katsu_cuda_ctx *ctx, const KatsuAmaxJob *jobs, int count);
// Writes up to KATSU_STAGE_JOBS operands' planes, one launch.
constexpr int KATSU_STAGE_JOBS = 4;
int32_t katsu_f16_stage(katsu_cuda_ctx *ctx, const KatsuF16Call &call, const KatsuStageJob *jobs, int count);

// Planes of the narrow form in the context's mode, and of room for either form.
static inline int katsu_f16_narrow_planes(const katsu_cuda_ctx *ctx) { return ctx->precision == KATSU_MODE_3XTF32 ? 2 : 1; }

// Device slots for the operands of one call.  There are two sets, used in turn: the staging pass of a call clears the
// other one for the next call.  katsu_f16_new_call picks the set and must come before the call's slots are taken.
enum { KATSU_INFO_A, KATSU_INFO_B, KATSU_INFO_G, KATSU_INFO_SLOTS };
void katsu_f16_new_call(katsu_cuda_ctx *ctx);
int32_t katsu_f16_drop_call(katsu_cuda_ctx *ctx);  // nothing was launched for it after all; KATSU_OK
KatsuF16Info *katsu_f16_slot(katsu_cuda_ctx *ctx, int slot);
KatsuF16Call katsu_f16_call(const katsu_cuda_ctx *ctx, const KatsuF16Info *a, const KatsuF16Info *b, const KatsuF16Info *c);

// Bump allocator over a scratch block; every piece is 256-byte aligned.
struct KatsuArena {
    char *base;
    size_t bytes;
    void *take(size_t n) {
        void *p = base + bytes;
        bytes += (n + 255) / 256 * 256;
        return p;
    }
    KatsuF16Planes planes(size_t n, int count) {
        KatsuF16Planes p;
        p.stride = (n + 127) / 128 * 128;
        p.base = static_cast<__half *>(take(p.stride * count * sizeof(__half)));
        return p;
    }
    float *floats(size_t n) { return static_cast<float *>(take(n * sizeof(float))); }
};

static inline size_t katsu_round_up(size_t n, size_t to) { return (n + to - 1) / to * to; }

// The fp16 path of matmul (f16_matmul.cu); *handled = 0 when the shape or mode is not one it takes.
int32_t katsu_f16_matmul_fwd(katsu_cuda_ctx *ctx, const float *a, const float *b, float *c, size_t m, size_t k, size_t n,
                             int *handled);
int32_t katsu_f16_matmul_bwd(katsu_cuda_ctx *ctx, const float *a, const float *b, const float *g, float *da, float *db,
                             size_t m, size_t k, size_t n, int accumulate, int *handled);

// The fp16 path of the convolutions (f16_conv.cu), *handled as above.
bool katsu_f16_conv_takes_copy(const katsu_cuda_ctx *ctx, size_t n, size_t c, size_t h, size_t w, size_t k, size_t r,
                               size_t s, size_t stride, size_t pad, size_t oh, size_t ow);
size_t katsu_f16_conv_staged_bytes(const katsu_cuda_ctx *ctx, size_t n, size_t c, size_t h, size_t w);
int32_t katsu_f16_conv_stage(katsu_cuda_ctx *ctx, const float *x, void *staged, size_t n, size_t c, size_t h, size_t w);
int32_t katsu_f16_conv_fwd(katsu_cuda_ctx *ctx, const float *x, const float *w, const float *bias, int relu, float *y,
                           size_t n, size_t c, size_t h, size_t wd, size_t k, size_t r, size_t s, size_t stride, size_t pad,
                           size_t oh, size_t ow, int *handled);
int32_t katsu_f16_conv_bwd(katsu_cuda_ctx *ctx, const float *x, const float *w, const float *gr, const float *gscale,
                           float gfactor, float *dx, float *dw, size_t n, size_t c, size_t h, size_t wd, size_t k, size_t r,
                           size_t s, size_t stride, size_t pad, size_t oh, size_t ow, int accumulate,
                           int *handled);
