// The fp16 tensor-core kernel behind matmul and the convolutions in 3xTF32 and TF32 mode (operands: f16_split.cuh).
//
// Reference loops: Tensor::matmul and its VJP (crates/katsu-core/src/tensor.rs:265-273, 418-445), Conv2D forward and
// backward_buffers (crates/katsu-core/src/conv2d.rs:95-103, 232-262, 269-292).
//
// One kernel for three contractions; a result tile is 256 lanes x bn columns (bn = 32 .. 256) on a pair of thread blocks:
//
//   GEMM     C[j][i]        = sum_k  A[i][k] B[j][k]                 lanes i (contiguous in C), columns j
//   CONV     Y[n, o, pixel] = sum_ky sum_(kx, c) X[n, pixel + (ky, kx), c] W[ky][o][(kx, c)]    lanes pixels, columns o
//   CONV_DW  dW[ky, kx, c][o] = sum_pixel X[pixel + (ky, kx), c] G[pixel, o]                    lanes (ky, kx, c), columns o
//
// The lane index is the one that is contiguous in the result, so every store instruction of the epilogue writes whole
// 128-byte lines whatever the alignment, and NCHW comes out of a channels-innermost contraction without a pass.
//
// Convolution operands.  The staged tensor is [n][h][w + gap][cp]; the kx taps of a pixel are then ONE contiguous run of
// S * cp elements (the gap supplies the zeros left and right of a row).  The tensor map gives that run as its innermost
// dimension, overlapping from pixel to pixel, so k-blocks of 64 lose nothing to channel counts that are no multiple of 64:
// a filter row of 35 channels x 3 taps is 2 k-blocks, not 3.  Rows above and below the image are outside the tensor: zeros.
// Lanes are boxes of bw x bh pixels of nb images, chosen to waste few of them (56 x 56: 8 x 8 x 2, none).  TMA's im2col
// mode, which would waste none at any size, fetches a pixel in 8 clocks (16 bytes a clock; tiled boxes: 58): the wide
// layer's forward ran at 2 180 clocks a k-block with it.
//
// Passes.  Narrow operands (fp16): hi*hi in TF32 mode (NARROW = 1), lo*hi + hi*lo + hi*hi in 3xTF32 mode (NARROW = 2).
// Wide operands (bf16): the three largest products of two planes, or the six largest of three.  The tensor core's f32
// accumulation loses about 2e-8 of the sum per step, always towards zero, so the loss grows with the steps; in 3xTF32 mode
// eight epilogue warps fold an accumulator into f32 registers every p.drain k-blocks (katsu_f16_launch has the rule) while
// others fill.  A `fine` problem takes the small products of a k-block first, whose steps lose little, then the four steps of
// hi*hi, at 4 to 10 % more time than products in the order of the steps (which use A's rows twice in a row).
//
// What bounds it: at 256 x 256 a k-block is 12 (4) MMAs of 128 clocks against 64 (32) KiB of operand fill per block,
// the ratio of the TF32 kernels at twice their rate.
//
// Roles: warps 0-7 drain and store (lane quarter = warp % 4, alternate 32-column chunks by warp / 4), warp 8 issues the
// TMA loads, warp 9 of the leader block the MMAs.  Persistent over tiles x splits.  Every wait is bounded; both blocks of
// a pair always reach the cluster barrier at the end.
#include "f16_gemm.cuh"
#include "launch.cuh"
#include "sm100.cuh"
#include "sm100_pair.cuh"

using namespace sm100;

namespace {

constexpr int BM = 128, BK = 64;
constexpr int A_BYTES = BM * BK * 2;
constexpr int MAX_STAGES = 8;
constexpr int MAX_ACCS = 4;
constexpr int THREADS = 320;
constexpr uint32_t kLayoutSw64 = 4;
constexpr int RASTER_M = 16;
constexpr int SMEM_RING = 208 * 1024;
constexpr size_t SMEM = SMEM_RING + 1024;

struct Tile {
    int split, mt, nt;
};

// Bands of RASTER_M tile rows, column-major inside a band: blocks running together share operand tiles in L2.
__device__ __forceinline__ Tile tile_of(int item, const KatsuF16Problem &p) {
    Tile t;
    const int per_split = p.m_tiles * p.n_tiles;
    t.split = item / per_split;
    const int i = item - t.split * per_split;
    const int band_tiles = RASTER_M * p.n_tiles;
    const int band = i / band_tiles, r = i - band * band_tiles;
    const int rows = min(p.m_tiles - band * RASTER_M, RASTER_M);
    t.nt = r / rows;
    t.mt = band * RASTER_M + (r - t.nt * rows);
    return t;
}

// k-blocks [begin, end) of one class in one split.
__device__ __forceinline__ void k_range(const KatsuF16Problem &p, long long total, int split, int *begin, int *end) {
    const long long b = (long long)split * p.kb_per_split;
    const long long e = b + p.kb_per_split;
    *begin = int(b < total ? b : total);
    *end = int(e < total ? e : total);
}

template <KatsuF16Kind KIND>
__device__ __forceinline__ long long class_kblocks(const KatsuF16Problem &p, int py, int px) {
    if (KIND == KATSU_F16_CONV_DW) return p.blocks;
    if (KIND == KATSU_F16_GEMM) return p.gemm_chunks;
    return (long long)(p.row_begin[py + 1] - p.row_begin[py]) * p.chunks[px];
}

// First pixel of a box; past the last box an image that does not exist, which loads as zeros.
__device__ __forceinline__ void box_origin(const KatsuF16Problem &p, long long b, int *img, int *y, int *x) {
    if (b >= p.blocks) {
        *img = p.n_img;
        *y = *x = 0;
        return;
    }
    const unsigned q = unsigned(b) / unsigned(p.blocks_x);
    *x = int(unsigned(b) - q * p.blocks_x) * p.bw;
    const unsigned n = q / unsigned(p.blocks_y);
    *y = int(q - n * p.blocks_y) * p.bh;
    *img = int(n) * p.nb;
}

// One lane's values of columns col .. col + 31.  Few instructions a column: this runs on eight warps per block and sets the
// pace of layers with short contractions (with its branches inside the loop the small CNN's second dX took 0.58 ms).
// `bias` is column col + lane's, loaded before the accumulator was waited for; all lanes of the warp call this together.
__device__ __forceinline__ void store_columns(const KatsuF16Problem &p, float *d, bool valid, int col, const float (&v)[32],
                                              float factor, float bias) {
    const long long stride = p.col_stride;
    const int live = p.n_total - col;
    if (live >= 32 && !p.bias && !p.relu && !p.accumulate) {
        if (!valid) return;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            *d = v[i] * factor;
            d += stride;
        }
        return;
    }
    const float floor = p.relu ? 0.f : NAN;  // max(v, NaN) is v; max(NaN, 0) is 0: a ReLU cuts a NaN off, as in every kernel
#pragma unroll
    for (int i0 = 0; i0 < 32; i0 += 8) {
        float o[8];
        const bool all = live >= i0 + 8;
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = v[i0 + i] * factor + __shfl_sync(0xffffffffu, bias, i0 + i);
        if (p.accumulate && valid) {  // the loads of eight columns before the first store
            float old[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) old[i] = (all || i0 + i < live) ? d[i * stride] : 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] += old[i];
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            o[i] = fmaxf(o[i], floor);
            if (valid && (all || i0 + i < live)) *d = o[i];
            d += stride;
        }
    }
}

// The two neighbouring pixels of a stride-2 parity pair, for N channels from the one at `d` on: one 8-byte store where the
// result allows it.  Stored class by class, every 32-byte sector of dX went out half full twice, and these stores were
// half of the kernel's time (128 x 128 x 112 x 112: 981 us, 516 without them).
template <int N, int STEP>
__device__ __forceinline__ void store_pairs(const KatsuF16Problem &p, float *d, bool ok0, bool ok1, int live, const float *a,
                                            const float *b, float factor) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
        if (i < live) {
            float2 v = make_float2(a[i * STEP] * factor, b[i * STEP] * factor);
            if (p.pair_vec) {
                if (ok0) {
                    if (p.accumulate) {
                        const float2 old = *reinterpret_cast<const float2 *>(d);
                        v.x += old.x;
                        v.y += old.y;
                    }
                    *reinterpret_cast<float2 *>(d) = v;
                }
            } else {
                if (ok0) d[0] = p.accumulate ? d[0] + v.x : v.x;
                if (ok1) d[1] = p.accumulate ? d[1] + v.y : v.y;
            }
        }
        d += p.col_stride;
    }
}

// The mixed results (f16_exact.cuh) that this thread has stored, or left out (`left_out`), for the tile of its pixel (img, jy, jx).
__device__ __noinline__ void repair_tile(const KatsuF16Problem &p, int img, int jy, int jx, int n0, int group, bool left_out) {
    for (int py = 0; py < p.classes_y; ++py)
        for (int px = 0; px < p.classes_x; ++px)
            for (int i = 0; i < 128; ++i) {  // alternate 32-column chunks, as they are stored
                const int col = n0 + ((i >> 5) * 2 + group) * 32 + (i & 31);
                if (col >= n0 + p.bn) break;
                int channel = col, y = p.step * jy + py, x = p.step * jx + px;
                if (p.class_cols) {
                    const int q = col / p.class_cols;
                    if (q > 1) break;
                    channel = (col - q * p.class_cols) >> 1;
                    y += q;
                    x += col & 1;
                }
                if (channel >= p.n_total || y >= p.out_h || x >= p.out_w || !katsu_f16_mixed(p.raw, y, x)) continue;
                float *d = p.out + img * p.img_stride + (long long)y * p.out_w + x + channel * p.col_stride;
                if (!left_out && katsu_is_number(*d)) continue;
                float v = katsu_f16_exact(p.raw, img, channel, y, x);
                if (p.bias) v += __ldg(p.bias + channel);
                if (p.accumulate) v += *d;
                *d = p.relu ? fmaxf(v, 0.f) : v;
            }
}

template <int NARROW, KatsuF16Kind KIND>
__global__ void __launch_bounds__(THREADS, 1)
f16_pair_kernel(const __grid_constant__ KatsuF16Maps maps, const __grid_constant__ KatsuF16Problem p) {
    constexpr bool MN = KIND == KATSU_F16_CONV_DW, CONV = KIND == KATSU_F16_CONV || KIND == KATSU_F16_CONV_DX2;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ uint64_t full[MAX_STAGES], empty[MAX_STAGES], acc_full[MAX_ACCS], acc_empty[MAX_ACCS];
    __shared__ uint32_t tmem_slot;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const bool leader = rank == 0;
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int items = p.m_tiles * p.n_tiles * p.splits;
    const int half = p.bn >> 1;                 // B columns that this block loads
    const int b_bytes = half * BK * 2;
    launch_next();

    if (threadIdx.x == 0) {
        for (int s = 0; s < MAX_STAGES; ++s) {
            mbar_init(&full[s], 1);    // the leader's: its own expect_tx arrival, both blocks' bytes
            mbar_init(&empty[s], 1);   // each block's own copy, released by the leader's commit
        }
        for (int b = 0; b < MAX_ACCS; ++b) {
            mbar_init(&acc_full[b], 1);    // each block's own copy
            mbar_init(&acc_empty[b], 16);  // the leader's: eight epilogue warps of each block
        }
        mbar_init_fence();
    }
    if (warp == 9) {
        tmem_alloc_pair(&tmem_slot, 512);
        tmem_relinquish_pair();
    }
    if (warp == 8 && lane < 2 * NARROW) tma_prefetch_desc(lane < NARROW ? &maps.a[lane] : &maps.b[lane - NARROW]);
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();  // both blocks' barriers exist before anything is signalled across the pair
    tc_fence_after_sync();
    const uint32_t tmem_base = tmem_slot;
    launch_wait();
    const KatsuF16Info info_a = katsu_f16_load(p.info_a), info_b = katsu_f16_load(p.info_b);
    const bool wide = katsu_f16_wide(p.call);
    const int planes = NARROW + (wide ? 1 : 0);
    // Mixed results are summed again (f16_exact.cuh).  What is added to, or ends in a ReLU, cannot be told from what it should be
    // once it is stored, so such a call does not store them first.  Parts of a split contraction are looked at when they are folded.
    const bool repairs = CONV && p.raw.form != KatsuF16Raw::NONE && p.splits == 1 && !(katsu_f16_finite(info_a) && katsu_f16_finite(info_b));
    const bool left_out = repairs && (p.accumulate || p.relu);
    // k-blocks between two drains: in TF32 mode up to 12 288 accumulation steps (4e-4 of 2e-3)
    const int drain = NARROW == 2 ? (wide ? max(p.drain / 2, 1) : p.drain) : 1024;
    // accumulators that take turns; hand-over q is the one q & (2^acc_bits - 1), acc_cols columns apart
    const int acc_bits = NARROW == 2 && p.bn <= 128 ? 2 : 1, acc_mask = (1 << acc_bits) - 1, acc_cols = 512 >> acc_bits;
    const int b_off = planes * A_BYTES, stage_bytes = b_off + planes * b_bytes;
    const int stages = min(MAX_STAGES, SMEM_RING / stage_bytes);

    if (warp == 8 && lane == 0) {
        // ---- TMA producer: this block's lanes of A and half of B's columns; bytes counted on the leader's barrier ----
        const CUtensorMap *map_a = p.a_second && wide && katsu_f16_own_copy(p.call, info_a) ? maps.a_second : maps.a, *map_b = maps.b;
        bool ok = true;
        int s = 0;
        uint32_t phase = 1;  // a fresh barrier counts as released
        for (int item = pair; item < items && ok; item += pairs) {
            const Tile t = tile_of(item, p);
            const long long m0 = (2ll * t.mt + rank) * BM;
            const int n0 = t.nt * p.bn + int(rank) * half;
            int img = 0, jy = 0, jx = 0;  // CONV: first pixel of this block's lanes
            if (CONV) box_origin(p, 2ll * t.mt + rank, &img, &jy, &jx);
            // CONV_DW: this block's two column groups; past the last one an image that does not exist
            int group_y[2] = {0, 0}, group_x[2] = {0, 0};
            bool group_live[2] = {false, false};
            if (MN) {
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    const int group = (2 * t.mt + int(rank)) * 2 + g;
                    if (group >= p.groups) continue;
                    group_live[g] = true;
                    group_y[g] = group / p.groups_per_row;
                    group_x[g] = group - group_y[g] * p.groups_per_row;
                }
            }
            auto tma_a = [&](unsigned char *to, const CUtensorMap *map, uint32_t bar, int n, int y, int x) {
                if (p.a_pairs) {
                    tma_load_5d_pair(to, map, bar, 0, x, y + group_y[0], group_live[0] ? n : p.n_img, group_x[0]);
                } else {
#pragma unroll
                    for (int g = 0; g < 2; ++g)
                        tma_load_4d_pair(to + g * (A_BYTES / 2), map, bar, group_x[g] * 64, x, y + group_y[g],
                                         group_live[g] ? n : p.n_img);
                }
            };
            for (int py = 0; py < p.classes_y && ok; ++py)
                for (int px = 0; px < p.classes_x && ok; ++px) {
                    int kb0, kb1;
                    k_range(p, class_kblocks<KIND>(p, py, px), t.split, &kb0, &kb1);
                    const int chunks = MN ? 1 : KIND == KATSU_F16_GEMM ? p.gemm_chunks : p.chunks[px];
                    int row = 0, chunk = 0;
                    if (!MN && kb1 > kb0) {
                        row = kb0 / chunks;
                        chunk = kb0 - row * chunks;
                        row += p.row_begin[py];
                    }
                    for (int i = kb0; i < kb1; ++i) {
                        if (!mbar_wait(&empty[s], phase, p.status, 171)) { ok = false; break; }
                        if (leader) mbar_arrive_expect_tx(&full[s], 2 * planes * (p.a_bytes + b_bytes));
                        const uint32_t bar = map_to_rank(&full[s], 0);
                        unsigned char *st = smem + s * stage_bytes;
                        if (KIND == KATSU_F16_GEMM) {
                            for (int part = 0; part < planes; ++part) {
                                tma_load_3d_pair(st + part * A_BYTES, map_a + part, bar, i * BK, int(m0), 0);
                                tma_load_3d_pair(st + b_off + part * b_bytes, map_b + part, bar, i * BK, n0, 0);
                            }
                        } else if (CONV) {
                            for (int part = 0; part < planes; ++part) {
                                tma_load_4d_pair(st + part * A_BYTES, map_a + part, bar, chunk * BK, jx + p.off_w[px],
                                                 jy * p.in_step + p.lower_h + p.off_h[row], img);
                                tma_load_3d_pair(st + b_off + part * b_bytes, map_b + part, bar,
                                                 p.b_col[px] + chunk * BK, n0, p.b_row[row]);
                            }
                            if (++chunk == chunks) {
                                chunk = 0;
                                ++row;
                            }
                        } else {
                            int n, oy, ox;
                            box_origin(p, i, &n, &oy, &ox);
                            const int per_load = half >= 64 ? 64 : 32;
                            for (int part = 0; part < planes; ++part) {
                                tma_a(st + part * A_BYTES, map_a + part, bar, n, oy * p.in_step + p.lower_h, ox);
                                if (p.b_pairs) {
                                    tma_load_5d_pair(st + b_off + part * b_bytes, map_b + part, bar, 0, ox, oy, n, n0 >> 6);
                                } else {
                                    for (int c = 0; c < half; c += per_load)
                                        tma_load_4d_pair(st + b_off + part * b_bytes + c * BK * 2,
                                                         map_b + part, bar, n0 + c, ox, oy, n);
                                }
                            }
                        }
                        if (++s == stages) {
                            s = 0;
                            phase ^= 1;
                        }
                    }
                }
        }
    } else if (warp == 9 && leader) {
        // ---- MMA issue for the pair: whole warp in the loop, the elect.sync thread issues ----
        const bool issue = elect_one();
        const uint32_t idesc = idesc_f16(2 * BM, p.bn, MN, MN, wide);
        // K-major: 128-byte rows, a 16-element step is 32 bytes.  MN-major: 64 (or 32) columns to a row, a step is 16
        // rows; groups of 64 columns are A_BYTES / 2 apart.
        const uint32_t b_layout = MN && half < 64 ? kLayoutSw64 : kLayoutSw128;
        const uint32_t b_sbo = MN && half < 64 ? 512 : 1024;
        const uint32_t a_step = MN ? 2048 : 32, b_step = MN ? (half < 64 ? 1024 : 2048) : 32;
        const uint32_t lbo = MN ? A_BYTES / 2 : 16;
        bool ok = true;
        int s = 0, q = 0;  // q: accumulator hand-overs so far
        uint32_t phase = 0;
        for (int item = pair; item < items && ok; item += pairs) {
            const int split = item / (p.m_tiles * p.n_tiles);
            for (int py = 0; py < p.classes_y && ok; ++py)
                for (int px = 0; px < p.classes_x && ok; ++px) {
                    int kb0, kb1;
                    k_range(p, class_kblocks<KIND>(p, py, px), split, &kb0, &kb1);
                    const int chunks = MN ? 1 : KIND == KATSU_F16_GEMM ? p.gemm_chunks : p.chunks[px];
                    int chunk = (!MN && kb1 > kb0) ? kb0 % chunks : 0;
                    const int last = MN ? BK / 16 : p.steps_last[px];
                    for (int kb = kb0; kb < kb1 && ok; ++q) {
                        const int b = q & acc_mask;
                        if (!mbar_wait_warp_ready(&acc_empty[b], ((q >> acc_bits) & 1) ^ 1, p.status, 172)) { ok = false; break; }
                        tc_fence_after_sync();
                        const uint32_t acc = tmem_base + uint32_t(b * acc_cols);
                        const int kb_end = min(kb + drain, kb1);
                        bool first = true;
                        for (; kb < kb_end; ++kb) {
                            if (!mbar_wait_warp_ready(&full[s], phase, p.status, 173)) { ok = false; break; }
                            tc_fence_after_sync();
                            // descriptors differ in their address field only (16-byte units in the low word)
                            const uint32_t st = smem_u32(smem + s * stage_bytes);
                            const uint64_t a0 = smem_desc(st, lbo, 1024, kLayoutSw128);
                            const uint64_t b0 = smem_desc(st + b_off, lbo, b_sbo, b_layout);
                            const int steps = (!MN && chunk == chunks - 1) ? last : BK / 16;
                            if (issue) {
                                const uint32_t na = A_BYTES >> 4, nb = b_bytes >> 4;  // to the next plane
                                if (NARROW == 2 && p.fine) {
                                    // plane pa of A times plane pb of B, all steps of the k-block
                                    auto product = [&](uint32_t pa, uint32_t pb) {
#pragma unroll
                                        for (int j = 0; j < BK / 16; ++j)
                                            if (j < steps) {
                                                mma_f16_pair(acc, a0 + pa * na + j * (a_step >> 4), b0 + pb * nb + j * (b_step >> 4), idesc, !first);
                                                first = false;
                                            }
                                    };
                                    if (wide) {
                                        product(2, 0);
                                        product(1, 1);
                                        product(0, 2);
                                    }
                                    product(1, 0);
                                    product(0, 1);
                                    product(0, 0);
                                } else {
#pragma unroll
                                    for (int j = 0; j < BK / 16; ++j) {
                                        if (j < steps) {
                                            const uint64_t ad = a0 + j * (a_step >> 4), bd = b0 + j * (b_step >> 4);
                                            const bool add = !(first && j == 0);
                                            if (NARROW == 2) {
                                                if (wide) {
                                                    mma_f16_pair(acc, ad + 2 * na, bd, idesc, add);
                                                    mma_f16_pair(acc, ad + na, bd + nb, idesc, true);
                                                    mma_f16_pair(acc, ad, bd + 2 * nb, idesc, true);
                                                }
                                                mma_f16_pair(acc, ad + na, bd, idesc, add || wide);
                                                mma_f16_pair(acc, ad, bd + nb, idesc, true);
                                                mma_f16_pair(acc, ad, bd, idesc, true);
                                            } else {
                                                if (wide) {
                                                    mma_f16_pair(acc, ad + na, bd, idesc, add);
                                                    mma_f16_pair(acc, ad, bd + nb, idesc, true);
                                                }
                                                mma_f16_pair(acc, ad, bd, idesc, add || wide);
                                            }
                                        }
                                    }
                                }
                                // Every release goes to this block's barrier and to the peer's copy of it.  The accumulator's
                                // comes last: the blocks leave when it has been drained, and no arrival may be outstanding then.
                                mma_commit_both(&empty[s]);
                                if (kb == kb_end - 1) mma_commit_both(&acc_full[b]);
                            }
                            __syncwarp();
                            first = false;
                            if (!MN && ++chunk == chunks) chunk = 0;
                            if (++s == stages) {
                                s = 0;
                                phase ^= 1;
                            }
                        }
                    }
                }
        }
    } else if (warp < 8) {
        // ---- drains and epilogue: thread = lane of this block's half of the tile, alternate 32-column chunks ----
        const int quarter = warp & 3, group = warp >> 2;
        const int col_chunks = p.bn >> 5;
        float factor = p.gfactor;
        if (!wide) factor *= __uint_as_float(unsigned(127 - katsu_f16_exp(info_a) - katsu_f16_exp(info_b)) << 23);
        if (p.gscale) factor *= __ldg(p.gscale);
        int q = 0;
        bool alive = true;
        for (int item = pair; item < items && alive; item += pairs) {
            const Tile t = tile_of(item, p);
            const long long m = (2ll * t.mt + rank) * BM + quarter * 32 + lane;
            const int n0 = t.nt * p.bn;
            int img = 0, jy = 0, jx = 0;
            bool in_result = m < p.m_total;
            if (CONV) {
                const int r = quarter * 32 + lane;
                box_origin(p, 2ll * t.mt + rank, &img, &jy, &jx);
                const int q1 = r / p.bw, q2 = q1 / p.bh;
                jx += r - q1 * p.bw;
                jy += q1 - q2 * p.bh;
                img += q2;
                in_result = in_result && q2 < p.nb && img < p.n_img && !(KIND == KATSU_F16_CONV_DX2 && left_out);
            }
            const bool pairs_of_x = KIND == KATSU_F16_CONV_DX2 && p.pair_x;
            float run[4][32];  // sums of the drains; of pairs: [0, 1], and in [2, 3] those of the class px = 0 before
            for (int py = 0; py < p.classes_y && alive; ++py)
                for (int px = 0; px < p.classes_x && alive; ++px) {
                    int kb0, kb1;
                    k_range(p, class_kblocks<KIND>(p, py, px), t.split, &kb0, &kb1);
                    bool valid = in_result;
                    long long at = m;
                    int y = 0, x = 0;
                    if (CONV) {
                        y = p.step * jy + py, x = p.step * jx + px;
                        valid = valid && y < p.out_h && x < p.out_w;
                        if (KIND == KATSU_F16_CONV && left_out) valid = valid && !katsu_f16_mixed(p.raw, y, x);
                        at = img * p.img_stride + (long long)y * p.out_w + x;
                    }
                    float *dst = p.out + t.split * p.split_stride + at;
                    // columns n0 + c0 .. + 31 of this lane
                    auto put = [&](int c0, const float (&v)[32], float bias) {
                        const int col = n0 + c0;
                        if (KIND == KATSU_F16_CONV_DX2 && p.class_cols) {
                            // (a last column tile may reach past the classes)
                            const int q = col / p.class_cols, channel = (col - q * p.class_cols) >> 1;
                            const bool ok = in_result && q < 2 && y + q < p.out_h && x < p.out_w;
                            store_pairs<16, 2>(p, dst + q * p.out_w + channel * p.col_stride, ok, ok && x + 1 < p.out_w,
                                               p.n_total - channel, v, v + 1, factor);
                        } else {
                            store_columns(p, dst + col * p.col_stride, valid, col, v, factor, bias);
                        }
                    };
                    auto bias_of = [&](int c0) {
                        const int col = n0 + c0 + lane;
                        return p.bias && col < p.n_total ? __ldg(p.bias + col) : 0.f;
                    };
                    auto wait_acc = [&](int b) -> uint32_t {
                        alive = mbar_wait_warp(&acc_full[b], (q >> acc_bits) & 1, p.status, 174);
                        tc_fence_after_sync();
                        return tmem_base + (uint32_t(quarter * 32) << 16) + uint32_t(b * acc_cols);
                    };
                    auto release_acc = [&](int b) {
                        tc_fence_before_sync();
                        __syncwarp();
                        if (lane == 0) {
                            if (leader) mbar_arrive(&acc_empty[b]);
                            else mbar_arrive_cluster(map_to_rank(&acc_empty[b], 0));
                        }
                    };
                    if (!pairs_of_x && kb1 - kb0 <= drain) {
                        // one accumulator holds it all: 32 columns at a time, no sums in registers
                        float bias[4];
#pragma unroll
                        for (int c = 0; c < 4; ++c) bias[c] = bias_of((2 * c + group) * 32);
                        const uint32_t acc = kb1 > kb0 ? wait_acc(q & acc_mask) : 0;
                        if (!alive) break;
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            const int c0 = (2 * c + group) * 32;
                            if (c0 >= p.bn) break;
                            float v[32];
                            if (kb1 > kb0) {
                                tmem_ld_32x32(acc + c0, v);
                            } else {
#pragma unroll
                                for (int i = 0; i < 32; ++i) v[i] = 0.f;
                            }
                            put(c0, v, bias[c]);
                        }
                        if (kb1 > kb0) {
                            release_acc(q & acc_mask);
                            ++q;
                        }
                        continue;
                    }
#pragma unroll
                    for (int c = 0; c < 4; ++c)
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            if (c < 2) {
                                if (pairs_of_x) run[2 + c][i] = run[c][i];
                                run[c][i] = 0.f;
                            } else if (!pairs_of_x) {
                                run[c][i] = 0.f;
                            }
                        }
                    for (int kb = kb0; kb < kb1; kb += drain, ++q) {
                        const uint32_t acc = wait_acc(q & acc_mask);
                        if (!alive) break;
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            if (2 * c + group < col_chunks) {
                                float v[32];
                                tmem_ld_32x32(acc + (2 * c + group) * 32, v);
                                if (NARROW == 2 && 2 * c + group + 2 >= col_chunks) release_acc(q & acc_mask);
#pragma unroll
                                for (int i = 0; i < 32; ++i) run[c][i] += v[i];
                            }
                        }
                        if (NARROW == 1 || group >= col_chunks) release_acc(q & acc_mask);
                    }
                    if (!alive) break;
                    if (pairs_of_x) {
                        if (px == 0) continue;
                        const bool ok = in_result && y < p.out_h && x - 1 < p.out_w;
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            const int c0 = (2 * c + group) * 32;
                            if (c0 < p.bn)
                                store_pairs<32, 1>(p, dst - 1 + (n0 + c0) * p.col_stride, ok, valid, p.n_total - n0 - c0, run[2 + c],
                                                   run[c], factor);
                        }
                        continue;
                    }
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const int c0 = (2 * c + group) * 32;
                        if (c0 < p.bn) put(c0, run[c], bias_of(c0));
                    }
                }
        }
    }
    if (CONV && repairs && warp < 8) {
        // (behind the pipeline: no wait of the other warps runs out meanwhile)
        for (int item = pair; item < items; item += pairs) {
            const Tile t = tile_of(item, p);
            int img, jy, jx;
            box_origin(p, 2ll * t.mt + rank, &img, &jy, &jx);
            const int r = (warp & 3) * 32 + lane, q1 = r / p.bw, q2 = q1 / p.bh;
            if (q2 < p.nb && img + q2 < p.n_img)
                repair_tile(p, img + q2, jy + q1 - q2 * p.bh, jx + r - q1 * p.bw, t.nt * p.bn, warp >> 2, left_out);
        }
    }
    // Neither block leaves (or gives its tensor memory back) while the other may still signal its barriers,
    // read its half of B or hold accumulators: every path above ends here.
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();
    if (warp == 9) tmem_dealloc_pair(tmem_base, 512);
}

__global__ void __launch_bounds__(256)
f16_fold_kernel(const __grid_constant__ KatsuF16Raw raw, const float *__restrict__ partial, float *out, size_t count, int splits, int accumulate, const float *bias, size_t channels, size_t plane, int relu) {
    launch_next();
    launch_wait();
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += size_t(gridDim.x) * blockDim.x) {
        float s = 0.f;
#pragma unroll 8
        for (int q = 0; q < splits; ++q) s += __ldg(partial + size_t(q) * count + i);
        if (raw.form != KatsuF16Raw::NONE && !katsu_is_number(s)) s = katsu_f16_exact_element(raw, i, s);
        if (bias) s += __ldg(bias + (i / plane) % channels);
        if (relu) s = fmaxf(s, 0.f);
        out[i] = accumulate ? out[i] + s : s;
    }
}

template <int NARROW, KatsuF16Kind KIND>
int32_t launch(katsu_cuda_ctx *ctx, const KatsuF16Maps &maps, const KatsuF16Problem &p, unsigned pairs) {
    auto kernel = f16_pair_kernel<NARROW, KIND>;
    KATSU_TRY(katsu_prepare_kernel(ctx, (const void *)kernel, SMEM));
    return katsu_launch_chained(ctx, kernel, 2 * pairs, THREADS, SMEM, 2, maps, p);
}

}  // namespace

// Estimated clocks of every way to cut the problem; the cheapest wins.  A k-block costs the tensor pipe
// passes * 4 * bn / 2 clocks and the fill of (128 + bn / 2) * 128 bytes per part at about 60 bytes a clock; an item costs
// its pipeline start and its stores besides; splits pay for writing and folding their slabs.
KatsuF16Plan katsu_f16_plan(const katsu_cuda_ctx *ctx, KatsuF16Kind kind, long long m_total, int n_total,
                            long long kblocks, double out_floats, int most_bn) {
    const int parts = ctx->precision == KATSU_MODE_3XTF32 ? 2 : 1, passes = parts == 2 ? 3 : 1;
    const double pairs = ctx->num_sms / 2;
    const long long m_tiles = (m_total + 2 * BM - 1) / (2 * BM);
    KatsuF16Plan best = {0, 1};
    double best_cost = 0;
    for (int bn = 32; bn <= most_bn; bn += 32) {
        if (kind == KATSU_F16_CONV_DW && bn != 64 && bn != 128 && bn != 256) continue;
        const long long tiles = m_tiles * ((n_total + bn - 1) / bn);
        const double pipe = passes * 4 * bn / 2.0, fill = (BM + bn / 2) * 128.0 * parts / 60.0;
        const double per_kb = (pipe > fill ? pipe : fill) + 30;
        // unsplit, or as many splits as fill one to four waves
        for (int w = 0; w <= 4; ++w) {
            long long splits = w == 0 ? 1 : (long long)(w * pairs) / tiles;
            if (w > 0 && splits <= 1) continue;
            if (splits > kblocks / 2) splits = kblocks / 2;
            if (splits < 1) splits = 1;
            if (splits > 512) splits = 512;
            const long long kb = (kblocks + splits - 1) / splits;
            splits = (kblocks + kb - 1) / kb;
            const long long waves = (long long)((tiles * splits + pairs - 1) / pairs);
            double cost = waves * (kb * per_kb + 1200 + bn * 6);
            if (kind == KATSU_F16_CONV_DW) cost += splits * out_floats * 8 / 3000;
            else if (splits > 1) cost += (splits + 1) * out_floats * 4 / 2500 + 5000;
            if (best.bn == 0 || cost < best_cost) {
                best.bn = bn;
                best.splits = (int)splits;
                best_cost = cost;
            }
        }
    }
    return best;
}

int32_t katsu_f16_launch(katsu_cuda_ctx *ctx, KatsuF16Kind kind, const KatsuF16Maps &maps, KatsuF16Problem p,
                         const KatsuF16Plan &plan, float *partial, long long split_stride) {
    const int parts = katsu_f16_narrow_planes(ctx);
    p.bn = plan.bn;
    p.splits = plan.splits;
    p.m_tiles = (int)((p.m_total + 2 * BM - 1) / (2 * BM));
    p.n_tiles = ((p.class_cols ? 2 * p.class_cols : p.n_total) + plan.bn - 1) / plan.bn;
    long long most = 0;  // k-blocks of the longest class
    if (kind == KATSU_F16_CONV_DW) {
        most = p.blocks;
    } else if (kind == KATSU_F16_GEMM) {
        most = p.gemm_chunks;
    } else {
        for (int y = 0; y < p.classes_y; ++y)
            for (int x = 0; x < p.classes_x; ++x) {
                const long long kb = (long long)(p.row_begin[y + 1] - p.row_begin[y]) * p.chunks[x];
                if (kb > most) most = kb;
            }
    }
    // 3xTF32 mode: k-blocks to an accumulator, and with it the error against 64-bit sums of normally distributed values: 1 fine
    // 1.5e-7, 1 2.6e-7, 2 4.8e-7, 3 7e-7, 4 fine 6e-7 (plain 7e-7) in the small CNN's dX, 5 1.2e-6, 16 3.6e-6.  The lines lie where that is below the error of other arithmetic of this
    // mode's grade: kernels that cut operands into TF32 parts have 4.6e-7 to 8e-7 up to 8 k-blocks, 1.4e-6 and 1.6e-6 at 9
    // and 13, 4e-6 from 16 on, and 5e-7 to 4e-6 in dW; f32 multiply-adds 1.8e-8 times the root of their number (2.9e-7 for
    // 256 terms, 5.1e-7 for 800).  A drain costs more the shorter a tile's k-loop is (4096^3: 351 us with 16, 359 with 4, 375
    // with 2, 411 with 1; 64 channels, 8 x 56 x 56: 26.3, 27.9, 29.4, 31.4).
    // A contraction that one accumulator holds saves the sums in registers as well (that dX: 233 us, 300 in two parts).
    p.fine = p.f32_terms > 0 ? p.f32_terms < 256 : kind != KATSU_F16_CONV_DW && most == 4;
    if (p.f32_terms > 0) p.drain = p.f32_terms < 800 ? 1 : 2;
    else if (kind == KATSU_F16_CONV_DW) p.drain = 2;
    else p.drain = most == 4 ? 4 : most < 9 ? 3 : most < 16 ? 5 : 16;
    p.kb_per_split = (int)((most + plan.splits - 1) / plan.splits);
    if (p.kb_per_split < 1) p.kb_per_split = 1;
    p.split_stride = 0;
    if (plan.splits > 1 || kind == KATSU_F16_CONV_DW) {
        p.out = partial;
        p.split_stride = split_stride;
        p.accumulate = 0;
        p.bias = nullptr;
        p.relu = 0;
    }
    p.pair_vec = p.out_w % 2 == 0 && (reinterpret_cast<uintptr_t>(p.out) & 7) == 0;
    p.status = ctx->status;
    const long long items = (long long)p.m_tiles * p.n_tiles * p.splits;
    if (items > 0x3fffffff) return katsu_set_error(KATSU_ERR_UNSUPPORTED, "too many tiles");
    const unsigned pairs = (unsigned)(items < ctx->num_sms / 2 ? items : ctx->num_sms / 2);
    if (parts == 2) {
        if (kind == KATSU_F16_GEMM) return launch<2, KATSU_F16_GEMM>(ctx, maps, p, pairs);
        if (kind == KATSU_F16_CONV) return launch<2, KATSU_F16_CONV>(ctx, maps, p, pairs);
        if (kind == KATSU_F16_CONV_DX2) return launch<2, KATSU_F16_CONV_DX2>(ctx, maps, p, pairs);
        return launch<2, KATSU_F16_CONV_DW>(ctx, maps, p, pairs);
    }
    if (kind == KATSU_F16_GEMM) return launch<1, KATSU_F16_GEMM>(ctx, maps, p, pairs);
    if (kind == KATSU_F16_CONV) return launch<1, KATSU_F16_CONV>(ctx, maps, p, pairs);
    if (kind == KATSU_F16_CONV_DX2) return launch<1, KATSU_F16_CONV_DX2>(ctx, maps, p, pairs);
    return launch<1, KATSU_F16_CONV_DW>(ctx, maps, p, pairs);
}

int32_t katsu_f16_fold(katsu_cuda_ctx *ctx, const KatsuF16Raw &raw, const float *partial, float *out, size_t count, int splits,
                       int accumulate, const float *bias, size_t channels, size_t plane, int relu) {
    size_t blocks = katsu_div_up(count, (size_t)256);
    if (blocks > size_t(ctx->num_sms) * 8) blocks = size_t(ctx->num_sms) * 8;
    KATSU_TRY(katsu_prepare_kernel(ctx, (const void *)f16_fold_kernel, 0));
    return katsu_launch_chained(ctx, f16_fold_kernel, (unsigned)blocks, 256, 0, 1, raw, partial, out, count, splits, accumulate, bias,
                                channels, plane, relu);
}

bool katsu_f16_rows_maps(CUtensorMap *maps, const KatsuF16Planes &planes, int count, size_t cols, size_t rows, size_t d2,
                         size_t row_pitch, size_t d2_pitch, int box_rows) {
    katsu_tensor_map_encode_fn encode = katsu_tensor_map_encoder();
    if (encode == nullptr) return false;
    cuuint64_t dims[3] = {cols, rows, d2};
    cuuint64_t strides[2] = {row_pitch * 2, d2_pitch * 2};
    cuuint32_t box[3] = {(cuuint32_t)BK, (cuuint32_t)box_rows, 1}, estr[3] = {1, 1, 1};
    for (int i = 0; i < count; ++i)
        if (encode(maps + i, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, planes.base + i * planes.stride, dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return false;
    return true;
}

bool katsu_f16_window_maps(CUtensorMap *maps, const KatsuF16Planes &planes, long long offset, int count, size_t channels,
                           size_t width, size_t height, size_t images, size_t w_pitch, size_t h_pitch, size_t n_pitch,
                           int step_h, int box_channels, const KatsuF16Box &box, bool pairs) {
    katsu_tensor_map_encode_fn encode = katsu_tensor_map_encoder();
    if (encode == nullptr) return false;
    cuuint64_t dims[5] = {pairs ? 64 : channels, width, height, images, channels / 64};
    cuuint64_t strides[4] = {w_pitch * 2, h_pitch * 2, n_pitch * 2, 128};
    cuuint32_t gbox[5] = {(cuuint32_t)box_channels, (cuuint32_t)box.bw, (cuuint32_t)((box.bh - 1) * step_h + 1), (cuuint32_t)box.nb, 2};
    cuuint32_t estr[5] = {1, 1, (cuuint32_t)step_h, 1, 1};
    for (int i = 0; i < count; ++i)
        if (encode(maps + i, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, pairs ? 5 : 4, planes.base + offset + i * (long long)planes.stride, dims, strides,
                   gbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   box_channels == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return false;
    return true;
}

// Boxes narrower than 8 pixels (and than the grid) scatter the result over half-used 32-byte sectors and are taken only
// when they save a tenth of the lanes or more; among equals wide boxes of few images go first.
KatsuF16Box katsu_f16_box(int lanes, bool exact, int step_h, size_t width, size_t height, size_t images) {
    KatsuF16Box best = {0, 0, 0, 0, 0, 0};
    const unsigned w = (unsigned)width, h = (unsigned)height, n = (unsigned)images;
    const unsigned most_h = 255 / step_h + 1;  // a tensor map's box spans at most 256 rows of the tensor
    double best_cost = 0;
    auto consider = [&](unsigned bw, unsigned bh, unsigned nb) {
        if (bh > most_h) return;
        const unsigned bx = (w + bw - 1) / bw, by = (h + bh - 1) / bh, bn = (n + nb - 1) / nb;
        double cost = double(bx) * double(by) * double(bn);
        if (!exact && bw < 8 && bw < w) cost *= 1.1 * 8 / (bw + 7);
        if (best.bw == 0 || cost < best_cost) {
            best = {(int)bw, (int)bh, (int)nb, (int)bx, (int)by, (long long)bx * by * bn};
            best_cost = cost;
        }
    };
    if (exact) {
        for (int bw = lanes; bw >= 1; bw >>= 1)
            for (int bh = lanes / bw; bh >= 1; bh >>= 1) consider(bw, bh, lanes / (bw * bh));
        return best;
    }
    auto of_width = [&](unsigned bw) {
        if (bw > (unsigned)lanes) return;
        const unsigned rest = lanes / bw;
        auto of_height = [&](unsigned bh) {
            if (bh > rest || bh > h) return;
            const unsigned nb = rest / bh;
            consider(bw, bh, nb < n ? nb : n);
        };
        of_height(rest < h ? rest : h);
        for (unsigned parts = 1; parts <= 6 && parts <= h; ++parts) of_height((h + parts - 1) / parts);
        for (unsigned bh = 16; bh >= 1; bh >>= 1) of_height(bh);
    };
    for (unsigned parts = 1; parts <= 8 && parts <= w; ++parts) of_width((w + parts - 1) / parts);
    for (unsigned bw = 64; bw >= 4; bw >>= 1)
        if (bw <= w) of_width(bw);
    return best;
}
