// Convolution results that meet a value that is no number, and a product that the sum does not have.
//
// The tensor-core kernels multiply some terms that a sum does not have by zero: pixels of the padding, and at stride s the
// taps of other parity classes.  0 * inf is NaN, so a weight or gradient that is no number would reach results that do not
// depend on it.  Calls with such an operand therefore sum the results that have such products (`mixed`) again, from the f32
// operands, over exactly their own terms.  A sum ends when it is NaN, so a tensor full of NaNs costs little.
#pragma once

#include "common.cuh"

struct KatsuF16Raw {
    enum Form { NONE, FORWARD, DX, DW } form;  // NONE: nothing to do
    const float *a, *b;   // FORWARD: x, w; DX: g, w; DW: x, g
    int n, c, h, w, k, r, s, stride, pad, oh, ow;
    const float *gscale;  // every result is multiplied by gfactor and this device scalar (null: 1)
    float gfactor;
};

__device__ __forceinline__ bool katsu_is_number(float v) { return (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u; }

// (y, x): FORWARD and DX a pixel of the result, DW a tap.
__device__ __forceinline__ bool katsu_f16_mixed(const KatsuF16Raw &q, int y, int x) {
    if (q.form == KatsuF16Raw::FORWARD) {
        const int iy = y * q.stride - q.pad, ix = x * q.stride - q.pad;
        return iy < 0 || iy + q.r > q.h || ix < 0 || ix + q.s > q.w;
    }
    if (q.form == KatsuF16Raw::DX)
        return q.stride > 1 || y + q.pad - (q.r - 1) < 0 || y + q.pad >= q.oh || x + q.pad - (q.s - 1) < 0 || x + q.pad >= q.ow;
    // DW: output pixels whose tap is outside the image, or image rows that a box past the last output row reaches
    return y < q.pad || x < q.pad || (q.ow - 1) * q.stride + x - q.pad >= q.w || q.oh * q.stride + y - q.pad != q.h;
}

// One result in f32 multiply-adds, with the factors.  (i0, i1, y, x): FORWARD image, output channel; DX image, input channel;
// DW output channel, input channel.
static __device__ __noinline__ float katsu_f16_exact(const KatsuF16Raw &q, int i0, int i1, int y, int x) {
    float sum = 0.f;
    const size_t image = size_t(q.h) * q.w, plane = size_t(q.oh) * q.ow, taps = size_t(q.r) * q.s;
    if (q.form == KatsuF16Raw::FORWARD) {
        for (int c = 0; c < q.c && sum == sum; ++c) {
            const float *from = q.a + (size_t(i0) * q.c + c) * image, *w = q.b + (size_t(i1) * q.c + c) * taps;
            for (int ky = 0; ky < q.r; ++ky)
                for (int kx = 0; kx < q.s; ++kx) {
                    const int iy = y * q.stride + ky - q.pad, ix = x * q.stride + kx - q.pad;
                    if (iy >= 0 && iy < q.h && ix >= 0 && ix < q.w) sum = fmaf(from[size_t(iy) * q.w + ix], w[ky * q.s + kx], sum);
                }
        }
    } else if (q.form == KatsuF16Raw::DX) {
        for (int o = 0; o < q.k && sum == sum; ++o) {
            const float *g = q.a + (size_t(i0) * q.k + o) * plane, *w = q.b + (size_t(o) * q.c + i1) * taps;
            for (int ky = 0; ky < q.r; ++ky)
                for (int kx = 0; kx < q.s; ++kx) {
                    const int ty = y + q.pad - ky, tx = x + q.pad - kx;
                    if (ty < 0 || tx < 0 || ty % q.stride != 0 || tx % q.stride != 0) continue;
                    const int oy = ty / q.stride, ox = tx / q.stride;
                    if (oy < q.oh && ox < q.ow) sum = fmaf(g[size_t(oy) * q.ow + ox], w[ky * q.s + kx], sum);
                }
        }
    } else {
        for (int n = 0; n < q.n && sum == sum; ++n) {
            const float *from = q.a + (size_t(n) * q.c + i1) * image, *g = q.b + (size_t(n) * q.k + i0) * plane;
            for (int oy = 0; oy < q.oh; ++oy) {
                const int iy = oy * q.stride + y - q.pad;
                if (iy < 0 || iy >= q.h) continue;
                for (int ox = 0; ox < q.ow; ++ox) {
                    const int ix = ox * q.stride + x - q.pad;
                    if (ix >= 0 && ix < q.w) sum = fmaf(g[size_t(oy) * q.ow + ox], from[size_t(iy) * q.w + ix], sum);
                }
            }
        }
    }
    return sum * (q.gscale ? q.gfactor * __ldg(q.gscale) : q.gfactor);
}

// Element i of a FORWARD or DX result whose sum is s.
static __device__ __noinline__ float katsu_f16_exact_element(const KatsuF16Raw &q, size_t i, float s) {
    const bool forward = q.form == KatsuF16Raw::FORWARD;
    const int width = forward ? q.ow : q.w, height = forward ? q.oh : q.h, channels = forward ? q.k : q.c;
    const size_t row = i / width, plane = row / height;
    const int y = int(row - plane * height), x = int(i - row * width);
    return katsu_f16_mixed(q, y, x) ? katsu_f16_exact(q, int(plane / channels), int(plane % channels), y, x) : s;
}
