// Launch interface of the fp16 tensor-core kernel (f16_gemm.cu).
#pragma once

#include <cuda.h>

#include "f16_exact.cuh"
#include "f16_split.cuh"

constexpr int KATSU_F16_MAX_ROWS = 49;    // filter rows over all y-parity classes
constexpr int KATSU_F16_MAX_CLASSES = 8;  // parity classes per axis

enum KatsuF16Kind {
    KATSU_F16_GEMM,     // A and B are K-major matrices
    KATSU_F16_CONV,     // A is a convolution window over a channels-innermost tensor (forward, dX), B taps x rows
    KATSU_F16_CONV_DX2,  // CONV with the stores of dX at stride 2, whose code slows the others' epilogue
    KATSU_F16_CONV_DW,  // contraction over pixels, both operands MN-major
};

// out[lane offset + column * col_stride] = factor * sum_k A[lane][k] * B[column][k]; see f16_gemm.cu.
struct KatsuF16Problem {
    float *out;
    const float *bias;  // per column, or null
    int relu, accumulate;
    // Terms of one sum where TF32 parts would not do for 3xTF32 mode, because the shape can have f32 multiply-adds (rows that
    // are not whole 16-byte units, few channels); 0 elsewhere.
    long long f32_terms;
    KatsuF16Call call;
    const KatsuF16Info *info_a, *info_b;
    // A's planes come from the second set of maps when the copy made before the call is not one for it (katsu_f16_own_copy)
    int a_second;
    const float *gscale;  // device scalar or null, times gfactor
    float gfactor;
    KatsuF16Raw raw;
    long long m_total;    // lanes: matrix rows, pixels of the grid, or dW rows
    int n_total;          // columns
    long long col_stride;
    // ---- contraction: class (py, px) has rows row_begin[py] .. row_begin[py + 1] - 1, each of chunks[px] 64-wide
    // k-blocks, the last one of steps_last[px] 16-wide steps (a matrix product has one class and one row)
    int classes_y, classes_x;
    int row_begin[KATSU_F16_MAX_CLASSES + 1];
    short off_h[KATSU_F16_MAX_ROWS], b_row[KATSU_F16_MAX_ROWS];
    short off_w[KATSU_F16_MAX_CLASSES], steps_last[KATSU_F16_MAX_CLASSES];
    int chunks[KATSU_F16_MAX_CLASSES], b_col[KATSU_F16_MAX_CLASSES];
    int gemm_chunks;  // GEMM: k-blocks of the contraction (its chunks[0])
    // ---- pixels (conv kinds), in boxes of bw x bh pixels of nb images: box b is (b % blocks_x, b / blocks_x % blocks_y,
    // rest).  CONV: one box is the 128 lanes of a block (bw * bh * nb <= 128); grid pixel (jy, jx) reads operand rows
    // jy * in_step + lower_h + off_h and is output pixel (step * jy + py, step * jx + px).  CONV_DW: one box is a k-block
    // (bw * bh * nb == 64).
    int n_img, bw, bh, nb, blocks_x, blocks_y;
    long long blocks;
    int in_step, lower_h;
    int out_h, out_w, step;
    // CONV_DX2, step 2.  class_cols, if not 0: one contraction for all four parity classes, columns (py, channel, px),
    // class_cols to a py.  Else pair_x: the classes px = 0 and 1 are stored together (bn <= 128).  pair_vec: as float2.
    int class_cols, pair_x, pair_vec;
    long long img_stride;
    // ---- dW: lanes are 64-wide column groups, groups_per_row to a filter row
    int groups, groups_per_row;
    int a_pairs, b_pairs;  // the maps are of the `pairs` form: one load brings two column groups
    int a_bytes;  // bytes of one loaded A part of a k-block
    // filled in by the launcher
    int bn, m_tiles, n_tiles, splits, kb_per_split, drain, fine;
    long long split_stride;
    int *status;
};

// Tensor maps of the planes (the narrow form uses the leading ones).
struct KatsuF16Maps {
    CUtensorMap a[3], b[3], a_second[3];
};

// How a problem is cut: columns per tile and number of splits of the contraction.
struct KatsuF16Plan {
    int bn, splits;
};
KatsuF16Plan katsu_f16_plan(const katsu_cuda_ctx *ctx, KatsuF16Kind kind, long long m_total, int n_total,
                            long long kblocks, double out_floats, int most_bn = 256);

// Starts the kernel; with plan.splits > 1 the results go to `partial` (splits slabs of split_stride floats in the
// layout of `out`) and the caller folds them.
int32_t katsu_f16_launch(katsu_cuda_ctx *ctx, KatsuF16Kind kind, const KatsuF16Maps &maps, KatsuF16Problem p,
                         const KatsuF16Plan &plan, float *partial, long long split_stride);

// out[i] (+)= act(sum over splits of partial[split][i] + bias[(i / plane) % channels]).
int32_t katsu_f16_fold(katsu_cuda_ctx *ctx, const KatsuF16Raw &raw, const float *partial, float *out, size_t count, int splits,
                       int accumulate, const float *bias, size_t channels, size_t plane, int relu);

// Pixel boxes over a width x height x images grid: the factors of a box of at most `lanes` pixels (exactly `lanes`, in
// powers of two, when `exact`) that waste the fewest lanes.
struct KatsuF16Box {
    int bw, bh, nb;
    int blocks_x, blocks_y;
    long long blocks;
};
KatsuF16Box katsu_f16_box(int lanes, bool exact, int step_h, size_t width, size_t height, size_t images);

// Tensor maps over fp16 planes.  rows_map: [d2][rows][cols] with pitches in elements, box 64 x box_rows x 1, 128-byte
// swizzle.  window_map: {channels, width, height, images} with pitches in elements, box of box_channels x a pixel box whose
// rows are step_h apart.
// One map per plane.  `pairs` (channels a multiple of 64): the groups of 64 channels are a fifth dimension and a box holds
// two of them, one behind the other.
bool katsu_f16_rows_maps(CUtensorMap *maps, const KatsuF16Planes &planes, int count, size_t cols, size_t rows, size_t d2, size_t row_pitch,
                        size_t d2_pitch, int box_rows);
bool katsu_f16_window_maps(CUtensorMap *maps, const KatsuF16Planes &planes, long long offset, int count, size_t channels, size_t width, size_t height,
                          size_t images, size_t w_pitch, size_t h_pitch, size_t n_pitch, int step_h, int box_channels,
                          const KatsuF16Box &box, bool pairs = false);
