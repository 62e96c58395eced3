// The passes in front of the fp16 tensor-core kernels: the largest magnitude of an operand with the range check, and
// the operand's fp16 planes in the layout its kernel loads (f16_split.cuh).
//
// Both are bound by HBM: the first reads the operand once (4 bytes an element), the second reads it again (from L2
// when the operand fits there) and writes 2 or 4 bytes an element.  Up to three operands share a launch, because in
// small calls a launch costs more than the pass.
#include "f16_split.cuh"
#include "launch.cuh"

namespace {

constexpr int THREADS = 256;
constexpr int STAGE_BLOCKS = 5;  // resident staging blocks per SM

// ---- largest magnitude ------------------------------------------------------------------------------------------
constexpr int AMAX_BLOCKS = 3;   // resident blocks per SM
constexpr int AMAX_ROWS = 16;    // rows of a strip at most

struct AmaxSegment {
    KatsuAmaxJob job;
    // Of a matrix.  The first `longer` strips have strip_rows + 1 rows, the others strip_rows: no strip of a row or two at the
    // end, whose elements would be groups by themselves.
    unsigned strips, strip_rows, longer, col_tiles;
    unsigned first_block, blocks;
    int vec;  // 128 columns to a tile, a float4 to a lane; else 32
};

struct AmaxParams {
    AmaxSegment seg[3];
    int segments;
};

__device__ __forceinline__ unsigned magnitude(float v) { return __float_as_uint(v) & 0x7fffffffu; }

// Magnitudes of ROWS rows of a tile, W columns to a lane, all loads in flight before the first use and no branch between
// them (with a range check around each load the compiler kept one in flight: 100 us for 103 M floats).  Rows past the last
// are the last one again, which changes no maximum.
template <int ROWS, int W>
__device__ __forceinline__ void amax_rows(const float *src, size_t pitch, unsigned rows, unsigned &most, unsigned &least,
                                          unsigned (&column)[W]) {
    unsigned v[ROWS][W];
#pragma unroll
    for (unsigned i = 0; i < ROWS; ++i) {
        const float *at = src + size_t(min(i, rows - 1)) * pitch;
        if (W == 4) {
            const float4 q = __ldg(reinterpret_cast<const float4 *>(at));
            v[i][0] = magnitude(q.x);
            v[i][W > 1 ? 1 : 0] = magnitude(q.y);
            v[i][W > 2 ? 2 : 0] = magnitude(q.z);
            v[i][W > 3 ? 3 : 0] = magnitude(q.w);
        } else {
            v[i][0] = magnitude(__ldg(at));
        }
    }
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
        unsigned m = v[i][0];
#pragma unroll
        for (int u = 0; u < W; ++u) {
            column[u] = max(column[u], v[i][u]);
            if (u) m = max(m, v[i][u]);
        }
        m = __reduce_max_sync(0xffffffffu, m);
        most = max(most, m);
        least = min(least, m ? m : 0x7fffffffu);
    }
}

template <int W>
__device__ __forceinline__ void amax_tiles(const AmaxSegment &sg, unsigned first, unsigned stride, unsigned &most, unsigned &least) {
    const KatsuAmaxJob &j = sg.job;
    const int lane = threadIdx.x & 31;
    const unsigned long long tiles = (unsigned long long)j.images * sg.strips * sg.col_tiles;
    unsigned least_column = 0x7fffffffu;
    // From the tensor's end to its front: the staging pass starts at the front, which then is what L2 holds.
    for (unsigned long long left = tiles - min((unsigned long long)first, tiles); left > 0; left -= min((unsigned long long)stride, left)) {
        const unsigned long long rest = (left - 1) / sg.col_tiles;
        const unsigned tile = unsigned(left - 1 - rest * sg.col_tiles);
        const unsigned long long image = rest / sg.strips;
        const unsigned strip = unsigned(rest - image * sg.strips);
        const unsigned row = strip * sg.strip_rows + min(strip, sg.longer), rows = sg.strip_rows + (strip < sg.longer ? 1 : 0);
        // the last tile reaches back so that it is a full one; lanes past a narrow row read its last columns again
        unsigned col = tile * (32 * W);
        if (col + 32 * W > j.cols) col = j.cols > 32 * W ? j.cols - 32 * W : 0;
        col = min(col + lane * W, j.cols - W);
        const float *src = j.src + (size_t(image) * j.rows + row) * j.cols + col;
        unsigned column[W] = {};
        if (rows <= 4) amax_rows<4, W>(src, j.cols, rows, most, least, column);
        else if (rows <= 8) amax_rows<8, W>(src, j.cols, rows, most, least, column);
        else amax_rows<AMAX_ROWS, W>(src, j.cols, rows, most, least, column);
#pragma unroll
        for (int u = 0; u < W; ++u) least_column = min(least_column, column[u] ? column[u] : 0x7fffffffu);
    }
    if (j.columns) least = min(least, __reduce_min_sync(0xffffffffu, least_column));
}

// Magnitudes compare as their bit patterns, which puts infinities and NaNs above every number.
__global__ void __launch_bounds__(THREADS, AMAX_BLOCKS) amax_kernel(const __grid_constant__ AmaxParams p) {
    launch_next();
    launch_wait();
    int si = 0;
    while (si + 1 < p.segments && blockIdx.x >= p.seg[si + 1].first_block) ++si;
    const AmaxSegment &sg = p.seg[si];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned first = (blockIdx.x - sg.first_block) * (THREADS / 32) + warp, stride = sg.blocks * (THREADS / 32);
    unsigned most = 0, least = 0x7fffffffu;
    if (sg.vec) amax_tiles<4>(sg, first, stride, most, least);
    else amax_tiles<1>(sg, first, stride, most, least);

    __shared__ unsigned sh_most[THREADS / 32], sh_least[THREADS / 32];
    if (lane == 0) {
        sh_most[warp] = most;
        sh_least[warp] = least;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int i = 1; i < THREADS / 32; ++i) {
        most = max(most, sh_most[i]);
        least = min(least, sh_least[i]);
    }
    // no result is waited for: the kernels behind this one read the slots when it has ended
    atomicMax(&sg.job.info->most, most);
    if (most) atomicMax(&sg.job.info->inverted_least, 0x7fffffffu - least);
}

__global__ void clear_kernel(KatsuF16Info *info) {
    if (threadIdx.x < KATSU_INFO_SLOTS) info[threadIdx.x] = KatsuF16Info{0, 0};
}

// ---- fp16 planes ------------------------------------------------------------------------------------------------
struct StageParams {
    KatsuF16Call call;
    int narrow_planes;
    KatsuF16Info *clear;  // the other set of slots, or null
    KatsuStageJob job[KATSU_STAGE_JOBS];
    unsigned first_block[KATSU_STAGE_JOBS], blocks[KATSU_STAGE_JOBS];
    int jobs;
};

// How the values of one job are written.
struct Writer {
    KatsuF16Planes to;
    float scale;
    int planes;  // planes of the form in use
    bool wide, finite;
};

// Two scaled values as packed hi and lo halves.  Two values to a conversion: with one each, the conversion pipe and not
// memory set the pace of these passes.
__device__ __forceinline__ void split_narrow(float a, float b, unsigned *hi, unsigned *lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
    *hi = *reinterpret_cast<const unsigned *>(&h);
    *lo = *reinterpret_cast<const unsigned *>(&l);
}

// The leading 8 significand bits of v as a bf16 pattern in the upper half of a word, and what is left of v.  `below`: of the
// largest value below v's.  An infinity or NaN is one in every plane.
__device__ __forceinline__ unsigned peel(float *v, bool below) {
    unsigned bits = __float_as_uint(*v);
    if ((bits & 0x7f800000u) == 0x7f800000u) {
        if (bits & 0x007fffffu) bits |= 0x00400000u;  // a NaN stays one without its lower bits
        return bits & 0xffff0000u;
    }
    if (below && (bits & 0x7fffffffu) != 0) bits -= 1;
    bits &= 0xffff0000u;
    *v -= __uint_as_float(bits);
    return bits;
}

__device__ __forceinline__ unsigned peel2(float *a, float *b, bool below) { return (peel(a, below) >> 16) | peel(b, below); }

// Eight consecutive elements at `at` (16-byte aligned).
__device__ __forceinline__ void write8(const Writer &w, size_t at, float (&v)[8]) {
    if (!w.wide) {
        uint4 hi, lo;
        split_narrow(v[0] * w.scale, v[1] * w.scale, &hi.x, &lo.x);
        split_narrow(v[2] * w.scale, v[3] * w.scale, &hi.y, &lo.y);
        split_narrow(v[4] * w.scale, v[5] * w.scale, &hi.z, &lo.z);
        split_narrow(v[6] * w.scale, v[7] * w.scale, &hi.w, &lo.w);
        *reinterpret_cast<uint4 *>(w.to.base + at) = hi;
        if (w.planes == 2) *reinterpret_cast<uint4 *>(w.to.base + w.to.stride + at) = lo;
    } else {
        for (int i = 0; i < w.planes; ++i) {
            const bool below = !w.finite && i + 1 < w.planes;
            uint4 o;
            o.x = peel2(&v[0], &v[1], below);
            o.y = peel2(&v[2], &v[3], below);
            o.z = peel2(&v[4], &v[5], below);
            o.w = peel2(&v[6], &v[7], below);
            *reinterpret_cast<uint4 *>(w.to.base + i * w.to.stride + at) = o;
        }
    }
}

__device__ __forceinline__ void zero8(const Writer &w, size_t at) {
    for (int i = 0; i < w.planes; ++i) *reinterpret_cast<uint4 *>(w.to.base + i * w.to.stride + at) = make_uint4(0, 0, 0, 0);
}

// CT channels x 4096 / CT pixels through shared memory: 16-byte reads along pixels, 16-byte writes along channels (8 fp16
// channels of a pixel to a thread).  The tile's columns are XORed with the channel group so that both sides are free of
// bank conflicts: a warp writes one or two channel rows, and reads 8 channel groups of 4 pixels (CT = 64) or 4 groups of
// 8 pixels (CT = 32).  Few instructions a value matter here: with a thread per channel pair, and a division per pixel and
// channel, this pass was bound by instruction issue (0.20 ms for 103 M values, 4.1 TB/s).
//
// A block walks over tiles `block`, `block + blocks` ..., the loads of the next one in flight while it writes the present
// one.  (One tile to a block, with its wait for the scale and for the loads in front of every store, took 164 us for 103 M
// values into two planes.)
template <int CT>
__device__ void stage_nhwc_tiles(const KatsuStageJob &j, const Writer &out, unsigned block, unsigned blocks, float *tile) {
    constexpr int PT = 4096 / CT, GROUPS = CT / 8, XOR = 32 / GROUPS;
    const int hw = j.h * j.w;
    const unsigned ptiles = (hw + PT - 1) / PT, ctiles = (j.c + CT - 1) / CT, tiles = unsigned(j.n) * ptiles * ctiles;
    const bool vec = (hw & 3) == 0 && (reinterpret_cast<uintptr_t>(j.src) & 15u) == 0;
    // vec: a float4 a thread, PT / 4 threads to a channel; else a float a thread, PT threads to a channel
    constexpr int VSTEP = THREADS / (PT / 4), STEP = THREADS / PT;
    const int quad = threadIdx.x % (PT / 4), vrow = threadIdx.x / (PT / 4);
    const int col0 = threadIdx.x % PT, row0 = threadIdx.x / PT;
    float v[16];
    unsigned n = 0;
    int p0 = 0, c0 = 0;
    auto load = [&](unsigned t) {
        n = t / (ptiles * ctiles);
        const unsigned rest = t - n * (ptiles * ctiles), pt = rest / ctiles;
        p0 = int(pt) * PT;
        c0 = int(rest - pt * ctiles) * CT;
        const float *src = j.src + (size_t(n) * j.c + c0) * hw + p0;
        const int channels = min(j.c - c0, CT), pixels = min(hw - p0, PT);
        if (vec) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int row = vrow + VSTEP * i;
                const float4 q = (row < channels && quad * 4 < pixels)
                                     ? __ldg(reinterpret_cast<const float4 *>(src + size_t(row) * hw) + quad)
                                     : make_float4(0.f, 0.f, 0.f, 0.f);
                v[4 * i] = q.x; v[4 * i + 1] = q.y; v[4 * i + 2] = q.z; v[4 * i + 3] = q.w;
            }
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int row = row0 + STEP * i;
                v[i] = (row < channels && col0 < pixels) ? __ldg(src + size_t(row) * hw + col0) : 0.f;
            }
        }
    };
    const int g = threadIdx.x % GROUPS, first = threadIdx.x / GROUPS;
    const float *column = tile + g * 8 * PT;
    constexpr int PSTEP = THREADS / GROUPS;
    unsigned t = block;
    if (t < tiles) load(t);
    for (; t < tiles; t += blocks) {
        if (vec) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int row = vrow + VSTEP * i;
                *reinterpret_cast<float4 *>(tile + row * PT + ((quad * 4) ^ ((row >> 3) * XOR))) =
                    make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int row = row0 + STEP * i;
                tile[row * PT + (col0 ^ ((row >> 3) * XOR))] = v[i];
            }
        }
        const int channel = c0 + g * 8, from0 = p0 + first, pixels = min(hw - p0, PT);
        const size_t image = size_t(n) * j.h;
        __syncthreads();
        if (t + blocks < tiles) load(t + blocks);
        if (channel < j.cp) {
            int y = from0 / j.w, x = from0 - y * j.w;
#pragma unroll
            for (int i = 0; i < PT / PSTEP; ++i) {
                const int p = first + PSTEP * i;
                if (p >= pixels) break;
                const float *from = column + (p ^ (g * XOR));
                float o[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) o[u] = from[u * PT];
                const size_t at = ((image + y) * (j.w + j.gap) + x) * j.cp + channel;
                write8(out, at, o);
                if (x == j.w - 1)
                    for (int q = 1; q <= j.gap; ++q) zero8(out, at + size_t(q) * j.cp);
                x += PSTEP;
                while (x >= j.w) {
                    x -= j.w;
                    ++y;
                }
            }
        }
        __syncthreads();
    }
}

// Channels to a tile: 32 where that many are all there are, or where 64 would leave half a tile or more empty.
__host__ __device__ inline int tile_channels(int c) { return ((c + 31) / 32) & 1 && c < 160 ? 32 : 64; }

// Up to 16 channels: a thread per pixel and 8 channels, no transposition needed for whole-sector writes.
__device__ void stage_nhwc_narrow(const KatsuStageJob &j, const Writer &out, unsigned block, unsigned blocks) {
    const int hw = j.h * j.w, eights = j.cp / 8;
    const size_t pixels = size_t(j.n) * hw, total = pixels * eights;
    for (size_t i = size_t(block) * THREADS + threadIdx.x; i < total; i += size_t(blocks) * THREADS) {
        const int e = int(i / pixels);
        const size_t q = i - size_t(e) * pixels;
        const int n = int(q / hw), p = int(q - size_t(n) * hw);
        const int y = p / j.w, x = p - y * j.w;
        const float *src = j.src + (size_t(n) * j.c + e * 8) * hw + p;
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = (e * 8 + u < j.c) ? __ldg(src + size_t(u) * hw) : 0.f;
        const size_t at = ((size_t(n) * j.h + y) * (j.w + j.gap) + x) * j.cp + e * 8;
        write8(out, at, v);
        if (x == j.w - 1)
            for (int q2 = 1; q2 <= j.gap; ++q2) zero8(out, at + size_t(q2) * j.cp);
    }
}

__device__ void stage_rows(const KatsuStageJob &j, const Writer &out, unsigned block, unsigned blocks) {
    const unsigned eights = j.cp / 8;
    const size_t total = size_t(j.n) * eights;
    const bool vec = (j.c & 3) == 0 && (reinterpret_cast<uintptr_t>(j.src) & 15u) == 0;
    for (size_t i = size_t(block) * THREADS + threadIdx.x; i < total; i += size_t(blocks) * THREADS) {
        const size_t row = i / eights;
        const int c0 = int(i - row * eights) * 8;
        const float *src = j.src + row * j.c + c0;
        float v[8];
        if (vec && c0 + 8 <= j.c) {
            const float4 a = __ldg(reinterpret_cast<const float4 *>(src)), b = __ldg(reinterpret_cast<const float4 *>(src) + 1);
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
            v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        } else {
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = c0 + u < j.c ? __ldg(src + u) : 0.f;
        }
        write8(out, i * 8, v);
    }
}

// Rows and planes of staged weights.
__host__ __device__ inline int weight_rows(const KatsuStageJob &j) {
    return j.backward == 2 ? 2 * j.class_cols : j.backward ? j.c : j.k;
}
__host__ __device__ inline int weight_planes(const KatsuStageJob &j) { return j.backward == 2 ? j.span_h : j.r; }

// Eight columns of one weight row to a thread; cp and every class's first column are multiples of 8.
__device__ void stage_weights(const KatsuStageJob &j, const Writer &out, unsigned block, unsigned blocks) {
    const int rows = weight_rows(j), inner = j.backward ? j.k : j.c;
    const unsigned eights = j.width / 8, taps = j.r * j.s;
    const size_t total = size_t(weight_planes(j)) * rows * eights;
    const size_t step = j.backward ? size_t(j.c) * taps : taps;  // between channels of the contraction
    for (size_t i = size_t(block) * THREADS + threadIdx.x; i < total; i += size_t(blocks) * THREADS) {
        const int col = int(i % eights) * 8;
        const size_t rest = i / eights;
        int row = int(rest % rows), ky = int(rest / rows);
        int kx, ch;
        bool live;
        if (j.backward == 2) {
            const int py = row / j.class_cols, px = row & 1, t = col / j.cp;
            row = (row - py * j.class_cols) >> 1;
            ch = col - t * j.cp;
            ky = py + j.pad - 2 * (j.lower_h + ky);
            kx = px + j.pad - 2 * (j.first_x + t);
            live = row < j.c && t < j.span_x && ky >= 0 && ky < j.r && kx >= 0 && kx < j.s;
            if (!live) ky = kx = row = 0;
        } else if (j.backward) {
            int q = 0;
            while (q + 1 < j.classes && col >= j.col_begin[q + 1]) ++q;
            const int t = (col - j.col_begin[q]) / j.cp;
            ch = (col - j.col_begin[q]) - t * j.cp;
            kx = j.kx_last[q] - t * j.stride;
            live = t < j.class_taps[q];
        } else {
            kx = col / j.cp;
            ch = col - kx * j.cp;
            live = true;
        }
        const float *src = j.src + (j.backward ? size_t(ch) * step + size_t(row) * taps : size_t(row) * j.c * taps + size_t(ch) * taps) +
                           ky * j.s + kx;
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = (live && ch + u < inner) ? __ldg(src + u * step) : 0.f;
        write8(out, i * 8, v);
    }
}

__global__ void __launch_bounds__(THREADS, STAGE_BLOCKS) stage_kernel(const __grid_constant__ StageParams p) {
    __shared__ __align__(16) float tile[4096];
    launch_next();
    launch_wait();
    int ji = 0;
    while (ji + 1 < p.jobs && blockIdx.x >= p.first_block[ji + 1]) ++ji;
    const KatsuStageJob &j = p.job[ji];
    const unsigned block = blockIdx.x - p.first_block[ji];
    Writer out;
    out.to = j.to;
    const KatsuF16Info own = katsu_f16_load(j.info);
    out.wide = katsu_f16_wide(p.call);
    out.finite = katsu_f16_finite(p.call);
    out.planes = p.narrow_planes + (out.wide ? 1 : 0);
    out.scale = out.wide ? 1.f : __uint_as_float(unsigned(127 + katsu_f16_exp(own)) << 23);
    if (p.clear && blockIdx.x == 0 && threadIdx.x < KATSU_INFO_SLOTS) p.clear[threadIdx.x] = KatsuF16Info{0, 0};
    if (block == 0 && threadIdx.x == 0 && j.info_copy) *j.info_copy = own;
    if (j.only_if_mixed && !(out.wide && katsu_f16_own_copy(p.call, own))) return;
    if (j.kind == KATSU_STAGE_NHWC) {
        if (block == 0) {
            // zero pixels in front of the first row, zeros behind the last
            for (int i = threadIdx.x * 8; i < j.gap * j.cp; i += THREADS * 8) {
                Writer front = out;
                front.to.base -= size_t(j.gap) * j.cp;
                zero8(front, i);
            }
            const size_t end = size_t(j.n) * j.h * (j.w + j.gap) * j.cp;
            for (int i = threadIdx.x * 8; i < j.tail; i += THREADS * 8) zero8(out, end + i);
        }
        if (j.c <= 16) stage_nhwc_narrow(j, out, block, p.blocks[ji]);
        else if (tile_channels(j.c) == 32) stage_nhwc_tiles<32>(j, out, block, p.blocks[ji], tile);
        else stage_nhwc_tiles<64>(j, out, block, p.blocks[ji], tile);
    } else if (j.kind == KATSU_STAGE_ROWS) {
        stage_rows(j, out, block, p.blocks[ji]);
    } else {
        stage_weights(j, out, block, p.blocks[ji]);
    }
}

}  // namespace

static KatsuF16Info *slots(const katsu_cuda_ctx *ctx, int set) {
    return reinterpret_cast<KatsuF16Info *>(static_cast<char *>(ctx->f16_state) + set * 64);
}

// Set 2 is that of captured calls, which clear it themselves: a graph is replayed with the set it was captured with, at
// any point between other calls.
void katsu_f16_new_call(katsu_cuda_ctx *ctx) {
    ctx->f16_captured = katsu_capturing(ctx);
    if (!ctx->f16_captured) ctx->f16_set ^= 1;
}

int32_t katsu_f16_drop_call(katsu_cuda_ctx *ctx) {
    if (!ctx->f16_captured) ctx->f16_set ^= 1;
    return KATSU_OK;
}

KatsuF16Info *katsu_f16_slot(katsu_cuda_ctx *ctx, int slot) { return slots(ctx, ctx->f16_captured ? 2 : ctx->f16_set) + slot; }

KatsuF16Call katsu_f16_call(const katsu_cuda_ctx *ctx, const KatsuF16Info *a, const KatsuF16Info *b, const KatsuF16Info *c) {
    return KatsuF16Call{{a, b, c}, ctx->precision == KATSU_MODE_3XTF32 ? 17 : 28, nullptr, 1.f};
}

int32_t katsu_f16_amax(katsu_cuda_ctx *ctx, const KatsuAmaxJob *jobs, int count) {
    AmaxParams p;
    p.segments = count;
    unsigned at = 0;
    for (int i = 0; i < count; ++i) {
        AmaxSegment &s = p.seg[i];
        s.job = jobs[i];
        s.vec = (jobs[i].cols & 3) == 0 && (reinterpret_cast<uintptr_t>(jobs[i].src) & 15u) == 0;
        s.strips = (jobs[i].rows + AMAX_ROWS - 1) / AMAX_ROWS;
        s.strip_rows = jobs[i].rows / s.strips;
        s.longer = jobs[i].rows % s.strips;
        s.col_tiles = (jobs[i].cols + (s.vec ? 127 : 31)) / (s.vec ? 128 : 32);
        size_t blocks = katsu_div_up(size_t(jobs[i].images) * s.strips * s.col_tiles, (size_t)(THREADS / 32));
        if (blocks > size_t(ctx->num_sms) * AMAX_BLOCKS) blocks = size_t(ctx->num_sms) * AMAX_BLOCKS;
        s.first_block = at;
        s.blocks = (unsigned)blocks;
        at += s.blocks;
    }
    if (ctx->f16_captured) KATSU_LAUNCH(ctx, clear_kernel, 1, 32, 0, katsu_f16_slot(ctx, 0));
    KATSU_TRY(katsu_prepare_kernel(ctx, (const void *)amax_kernel, 0));
    return katsu_launch_chained(ctx, amax_kernel, at, THREADS, 0, 1, p);
}

int32_t katsu_f16_stage(katsu_cuda_ctx *ctx, const KatsuF16Call &call, const KatsuStageJob *jobs, int count) {
    StageParams p;
    p.call = call;
    p.narrow_planes = katsu_f16_narrow_planes(ctx);
    p.clear = ctx->f16_captured ? nullptr : slots(ctx, ctx->f16_set ^ 1);
    p.jobs = count;
    size_t at = 0;
    for (int i = 0; i < count; ++i) {
        const KatsuStageJob &j = jobs[i];
        p.job[i] = j;
        size_t blocks;
        const size_t hw = size_t(j.h) * j.w;
        if (j.kind == KATSU_STAGE_NHWC && j.c > 16) {
            const size_t ct = tile_channels(j.c);
            blocks = size_t(j.n) * katsu_div_up(hw, 4096 / ct) * katsu_div_up((size_t)j.c, ct);
            if (blocks > 0x3fffffff) return katsu_set_error(KATSU_ERR_UNSUPPORTED, "operand too large to stage");
            if (blocks > size_t(ctx->num_sms) * STAGE_BLOCKS) blocks = size_t(ctx->num_sms) * STAGE_BLOCKS;
        } else {
            const size_t units = j.kind == KATSU_STAGE_NHWC ? size_t(j.n) * hw * (j.cp / 8)
                                 : j.kind == KATSU_STAGE_ROWS ? size_t(j.n) * (j.cp / 8)
                                                              : size_t(weight_planes(j)) * weight_rows(j) * (j.width / 8);
            blocks = katsu_div_up(units, (size_t)THREADS);
            if (blocks > size_t(ctx->num_sms) * 64) blocks = size_t(ctx->num_sms) * 64;
        }
        // (as many blocks would do nothing but start and end when the copy is not needed: 30 us for 25 000)
        if (j.only_if_mixed && blocks > (size_t)ctx->num_sms) blocks = (size_t)ctx->num_sms;
        p.first_block[i] = (unsigned)at;
        p.blocks[i] = (unsigned)blocks;
        at += blocks;
    }
    if (at > 0x7fffffffu) return katsu_set_error(KATSU_ERR_UNSUPPORTED, "operand too large to stage");
    KATSU_TRY(katsu_prepare_kernel(ctx, (const void *)stage_kernel, 0));
    return katsu_launch_chained(ctx, stage_kernel, (unsigned)at, THREADS, 0, 1, p);
}
