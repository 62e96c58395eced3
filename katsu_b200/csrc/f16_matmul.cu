// matmul and its VJP on the fp16 tensor-core kernel (operands: f16_split.cuh, kernel: f16_gemm.cu).
//
//   c[m,n]  = a b      lanes n (rows of b^T, staged transposed), columns m (rows of a)      tensor.rs:264-273
//   da[m,k] = g b^T    lanes k (rows of b),                      columns m (rows of g)      tensor.rs:425-434
//   db[k,n] = a^T g    lanes n (rows of g^T),                    columns k (rows of a^T)    tensor.rs:435-444
//
// Staging pads the contraction to the 16 bytes TMA needs and takes operands at any address, so every shape comes
// here that is large enough to pay for the two passes in front.
#include "f16_gemm.cuh"

namespace {

// Multiply-adds from which the path, three to six launches, pays against gemm_small_kernel on the CUDA cores.  Forward / both
// gradients in us, here against there: 3xTF32 mode 17.2 / 23.8 against 12.3 / 25.3 at 256 x 512 x 256 (3.4e7), 18.1 / 27.7
// against 21.3 / 42.1 at 512 x 512 x 256 (6.7e7).  In TF32 mode the times would meet at 3e7 (13.8 / 20.2 against 8.0 / 16.0 at
// 256^3, 14.5 / 21.1 against 14.5 / 30.1 at 320^3); the line stays at the smallest products that have had 11-bit parts there.
double least_macs(const katsu_cuda_ctx *ctx) { return ctx->precision == KATSU_MODE_3XTF32 ? 4e7 : 1.5e7; }

bool takes(const katsu_cuda_ctx *ctx, size_t m, size_t k, size_t n) {
    if (ctx->precision == KATSU_MODE_FP32 || ctx->f16_state == nullptr) return false;
    if (m > 0x3fffffff || n > 0x3fffffff || k > 0x3fffffff) return false;
    return double(m) * double(n) * double(k) >= least_macs(ctx);
}

KatsuStageJob rows_job(const float *src, size_t rows, size_t cols, const KatsuF16Planes &to, const KatsuF16Info *info) {
    KatsuStageJob j = {};
    j.kind = KATSU_STAGE_ROWS;
    j.src = src;
    j.to = to;
    j.info = info;
    j.n = (int)rows;
    j.c = (int)cols;
    j.cp = (int)katsu_round_up(cols, 8);
    j.h = j.w = 1;
    return j;
}

// src [rows][cols] -> [cols][rows padded to 8]
KatsuStageJob transposed_job(const float *src, size_t rows, size_t cols, const KatsuF16Planes &to, const KatsuF16Info *info) {
    KatsuStageJob j = rows_job(src, 1, rows, to, info);
    j.kind = KATSU_STAGE_NHWC;
    j.w = (int)cols;
    return j;
}

struct Product {
    KatsuF16Planes lanes, columns;  // K-major, pitch round_up(K, 8)
    const KatsuF16Info *info_lanes, *info_columns;
    size_t n_lanes, n_columns, k;
    float *out;
    int accumulate;
    bool regular;
    KatsuF16Plan plan;
};

int32_t run(katsu_cuda_ctx *ctx, const KatsuF16Call &call, const Product &q, float *partial) {
    const size_t kp = katsu_round_up(q.k, 8);
    KatsuF16Maps maps;
    const int planes = katsu_f16_narrow_planes(ctx) + 1;
    if (!katsu_f16_rows_maps(maps.a, q.lanes, planes, kp, q.n_lanes, 1, kp, kp * q.n_lanes, 128) ||
        !katsu_f16_rows_maps(maps.b, q.columns, planes, kp, q.n_columns, 1, kp, kp * q.n_columns, q.plan.bn / 2))
        return katsu_set_error(KATSU_ERR_CUDA, "cuTensorMapEncodeTiled failed for a matmul operand");
    KatsuF16Problem p = {};
    p.out = q.out;
    p.accumulate = q.accumulate;
    p.f32_terms = q.regular ? 0 : (long long)q.k;
    p.call = call;
    p.info_a = q.info_lanes;
    p.info_b = q.info_columns;
    p.gfactor = 1.f;
    p.a_bytes = 128 * 128;
    p.m_total = (long long)q.n_lanes;
    p.n_total = (int)q.n_columns;
    p.col_stride = (long long)q.n_lanes;
    p.classes_y = p.classes_x = 1;
    p.row_begin[1] = 1;
    p.gemm_chunks = (int)katsu_div_up(q.k, 64);
    p.steps_last[0] = (short)(katsu_div_up(q.k, 16) - 4 * (size_t(p.gemm_chunks) - 1));
    const size_t count = q.n_lanes * q.n_columns;
    KATSU_TRY(katsu_f16_launch(ctx, KATSU_F16_GEMM, maps, p, q.plan, partial, (long long)count));
    if (q.plan.splits > 1)
        KATSU_TRY(katsu_f16_fold(ctx, p.raw, partial, q.out, count, q.plan.splits, q.accumulate,
                                 nullptr, 1, 1, 0));
    return KATSU_OK;
}

// Products of matrices whose rows are whole 16-byte units at 16-byte addresses, and no sliver: those that TF32 parts suit.
bool regular(const float *a, const float *b, const float *c, size_t m, size_t n, size_t k) {
    const uintptr_t at = reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c);
    return (at & 15u) == 0 && m >= 64 && n >= 32 && k >= 32;
}

KatsuF16Plan plan_for(const katsu_cuda_ctx *ctx, size_t n_lanes, size_t n_columns, size_t k) {
    return katsu_f16_plan(ctx, KATSU_F16_GEMM, (long long)n_lanes, (int)n_columns, (long long)katsu_div_up(k, 64),
                          double(n_lanes) * double(n_columns));
}

size_t partial_floats(const Product &q) { return q.plan.splits > 1 ? size_t(q.plan.splits) * q.n_lanes * q.n_columns : 0; }

}  // namespace

int32_t katsu_f16_matmul_fwd(katsu_cuda_ctx *ctx, const float *a, const float *b, float *c, size_t m, size_t k, size_t n,
                             int *handled) {
    *handled = 0;
    if (!takes(ctx, m, k, n)) return KATSU_OK;
    const int planes = katsu_f16_narrow_planes(ctx) + 1;
    const size_t kp = katsu_round_up(k, 8);
    Product q = {};
    q.plan = plan_for(ctx, n, m, k);
    q.n_lanes = n;
    q.n_columns = m;
    q.k = k;
    q.out = c;
    q.regular = k % 4 == 0 && n % 4 == 0 && regular(a, b, c, m, n, k);
    katsu_f16_new_call(ctx);
    KatsuF16Info *ia = katsu_f16_slot(ctx, KATSU_INFO_A), *ib = katsu_f16_slot(ctx, KATSU_INFO_B);
    q.info_lanes = ib;
    q.info_columns = ia;
    KatsuArena arena = {nullptr, 0};
    for (int pass = 0; pass < 2; ++pass) {  // the first only adds up the sizes
        if (pass) {
            float *base = nullptr;
            if (katsu_scratch(ctx, arena.bytes / 4, &base) != KATSU_OK) return katsu_f16_drop_call(ctx);  // no room: the other kernels
            arena = {reinterpret_cast<char *>(base), 0};
        }
        q.lanes = arena.planes(n * kp, planes);
        q.columns = arena.planes(m * kp, planes);
        float *partial = arena.floats(partial_floats(q));
        if (!pass) continue;
        *handled = 1;
        const KatsuF16Call call = katsu_f16_call(ctx, ia, ib, nullptr);
        const KatsuAmaxJob amax[2] = {katsu_amax_matrix(a, m, k, ia), katsu_amax_matrix(b, k, n, ib)};
        KATSU_TRY(katsu_f16_amax(ctx, amax, 2));
        const KatsuStageJob jobs[2] = {transposed_job(b, k, n, q.lanes, ib), rows_job(a, m, k, q.columns, ia)};
        KATSU_TRY(katsu_f16_stage(ctx, call, jobs, 2));
        KATSU_TRY(run(ctx, call, q, partial));
    }
    return KATSU_OK;
}

int32_t katsu_f16_matmul_bwd(katsu_cuda_ctx *ctx, const float *a, const float *b, const float *g, float *da, float *db,
                             size_t m, size_t k, size_t n, int accumulate, int *handled) {
    *handled = 0;
    if (!takes(ctx, m, k, n)) return KATSU_OK;
    const int planes = katsu_f16_narrow_planes(ctx) + 1;
    katsu_f16_new_call(ctx);
    KatsuF16Info *ia = katsu_f16_slot(ctx, KATSU_INFO_A), *ib = katsu_f16_slot(ctx, KATSU_INFO_B), *ig = katsu_f16_slot(ctx, KATSU_INFO_G);
    Product qa = {}, qb = {};
    qa.plan = plan_for(ctx, k, m, n);
    qa.n_lanes = k; qa.n_columns = m; qa.k = n;
    qa.out = da; qa.accumulate = accumulate;
    qa.regular = n % 4 == 0 && regular(g, b, da, m, k, n);
    qa.info_lanes = ib; qa.info_columns = ig;
    qb.plan = plan_for(ctx, n, k, m);
    qb.n_lanes = n; qb.n_columns = k; qb.k = m;
    qb.out = db;
    qb.regular = k % 4 == 0 && n % 4 == 0 && regular(a, g, db, k, n, m);
    // da == db (the same parent on both edges): the second product adds to the first whatever `accumulate` says
    qb.accumulate = da != nullptr && da == db ? 1 : accumulate;
    qb.info_lanes = ig; qb.info_columns = ia;
    const size_t np = katsu_round_up(n, 8), mp = katsu_round_up(m, 8);
    KatsuArena arena = {nullptr, 0};
    for (int pass = 0; pass < 2; ++pass) {
        if (pass) {
            float *base = nullptr;
            if (katsu_scratch(ctx, arena.bytes / 4, &base) != KATSU_OK) return katsu_f16_drop_call(ctx);
            arena = {reinterpret_cast<char *>(base), 0};
        }
        float *partial_a = nullptr, *partial_b = nullptr;
        if (da) {
            qa.lanes = arena.planes(k * np, planes);
            qa.columns = arena.planes(m * np, planes);
            partial_a = arena.floats(partial_floats(qa));
        }
        if (db) {
            qb.lanes = arena.planes(n * mp, planes);
            qb.columns = arena.planes(k * mp, planes);
            partial_b = arena.floats(partial_floats(qb));
        }
        if (!pass) continue;
        *handled = 1;
        const KatsuF16Call call = katsu_f16_call(ctx, ig, da ? ib : nullptr, db ? ia : nullptr);
        KatsuAmaxJob amax[3];
        KatsuStageJob jobs[4];
        int na = 0, nj = 0;
        amax[na++] = katsu_amax_matrix(g, m, n, ig);
        if (da) {
            amax[na++] = katsu_amax_matrix(b, k, n, ib);
            jobs[nj++] = rows_job(b, k, n, qa.lanes, ib);
            jobs[nj++] = rows_job(g, m, n, qa.columns, ig);
        }
        if (db) {
            amax[na++] = katsu_amax_matrix(a, m, k, ia);
            jobs[nj++] = transposed_job(g, m, n, qb.lanes, ig);
            jobs[nj++] = transposed_job(a, m, k, qb.columns, ia);
        }
        KATSU_TRY(katsu_f16_amax(ctx, amax, na));
        KATSU_TRY(katsu_f16_stage(ctx, call, jobs, nj));
        if (da) KATSU_TRY(run(ctx, call, qa, partial_a));
        if (db) KATSU_TRY(run(ctx, call, qb, partial_b));
    }
    return KATSU_OK;
}
