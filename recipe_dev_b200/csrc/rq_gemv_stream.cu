// Launches of the streaming matrix-vector kernel (rq_gemv_stream.cuh): plain matvecs, sibling projections, gated pairs and the
// planned launches of expert banks.
#include "rq_gemv_stream.cuh"

using namespace rqstream;

static int dispatch_stream_type(int type, StreamParams& p, bool is_float, int sm_count, int vectors, cudaStream_t s) {
    switch (type) {
        case RQ_Q4_K: return dispatch_type<RQ_Q4_K>(p, is_float, sm_count, vectors, s);
        case RQ_Q6_K: return dispatch_type<RQ_Q6_K>(p, is_float, sm_count, vectors, s);
        case RQ_Q8_0: return dispatch_type<RQ_Q8_0>(p, is_float, sm_count, vectors, s);
        default: return dispatch_type<RQ_Q4_0>(p, is_float, sm_count, vectors, s);
    }
}

// Launches the streaming kernel over a segment table. `table` is device memory, or null with the
// segments in `inline_seg` (at most RQ_INLINE_SEGMENTS, one sub-row each).
// vectors_per_launch = 0: the activation vectors are the tokens (x + t * st); > 0: one token, that
// many slot vectors. Returns RQ_ERR_UNSUPPORTED (without error text) when the shape is not served.
int rq_launch_stream(rq_ctx* ctx, int type, int64_t cols, const RqSegment* table, const RqSegment* inline_seg, int n_segments, int subs,
                     int epilogue, int64_t total_rows, const float* x, int64_t sk, int64_t st, int tokens, int vectors_per_launch,
                     int64_t yn, int64_t yt, int act_mode, const uint8_t* act, int fuse_step, uint8_t* act_out, cudaStream_t s) {
    if (cols % 256 || subs < 1 || subs > RQ_MAX_SUB) return RQ_ERR_UNSUPPORTED;
    if ((!table && n_segments > RQ_INLINE_SEGMENTS) || n_segments < 1 || n_segments > RQ_MAX_SEGMENTS) return RQ_ERR_UNSUPPORTED;
    StreamParams p;
    memset(&p, 0, sizeof(p));
    p.table = table;
    if (!table) for (int i = 0; i < n_segments; ++i) p.inline_seg[i] = inline_seg[i];
    p.n_segments = n_segments; p.subs = subs; p.epilogue = epilogue;
    p.rows = total_rows; p.cols = (int)cols; p.units = (int)(cols / 256);
    p.x = x; p.sk = sk; p.st = st; p.act = act; p.yn = yn; p.yt = yt; p.tokens = tokens;
    p.fuse_step = act_mode == RQ_ACT_INT8 ? fuse_step : 0; p.act_out = act_out;
    p.error_flag = ctx->error_flag; p.wait_ns = ctx->wait_limit_ns;
    switch (type) {
        case RQ_Q4_K: p.unit_bytes = 144; p.scales_per_unit = 0; break;
        case RQ_Q6_K: p.unit_bytes = 208; p.scales_per_unit = 1; break;
        case RQ_Q8_0: p.unit_bytes = 256; p.scales_per_unit = 8; break;
        case RQ_Q4_0: p.unit_bytes = 128; p.scales_per_unit = 8; break;
        default: return RQ_ERR_UNSUPPORTED;
    }
    return dispatch_stream_type(type, p, act_mode == RQ_ACT_FLOAT, ctx->sm_count, vectors_per_launch, s);
}

// A launch whose segment table and counts a kernel wrote into `plan` (device memory): the host
// sizes the launch for the maxima. FLOAT activations only: vector v is x + v * st. plan_count > 1 runs
// that many planned launches as the grid rows of one: row y reads plan[y * plan_stride] and x + y * x_plan_stride.
int rq_launch_stream_plan(rq_ctx* ctx, int type, int64_t cols, const RqPlan* plan, int plan_count, int plan_stride, int max_segments, int max_subs,
                          int epilogue, int64_t max_rows, const float* x, int64_t x_plan_stride, int64_t sk, int64_t st, int vectors, int64_t yn, int64_t yt,
                          cudaStream_t s, bool side_by_side) {
    if (cols % 256 || max_subs < 1 || max_subs > RQ_MAX_SUB || max_segments < 1 || max_segments > RQ_MAX_SEGMENTS || vectors < 1) return RQ_ERR_UNSUPPORTED;
    StreamParams p;
    memset(&p, 0, sizeof(p));
    p.plan = plan; p.plan_count = plan_count; p.plan_stride = plan_stride; p.x_plan_stride = x_plan_stride;
    p.n_segments = max_segments; p.subs = max_subs; p.epilogue = epilogue;
    p.rows = max_rows; p.cols = (int)cols; p.units = (int)(cols / 256);
    p.x = x; p.sk = sk; p.st = st; p.yn = yn; p.yt = yt; p.tokens = 1;
    p.bank_group = side_by_side ? -1 : 0;
    p.error_flag = ctx->error_flag; p.wait_ns = ctx->wait_limit_ns;
    switch (type) {
        case RQ_Q4_K: p.unit_bytes = 144; p.scales_per_unit = 0; break;
        case RQ_Q6_K: p.unit_bytes = 208; p.scales_per_unit = 1; break;
        case RQ_Q8_0: p.unit_bytes = 256; p.scales_per_unit = 8; break;
        case RQ_Q4_0: p.unit_bytes = 128; p.scales_per_unit = 8; break;
        default: return RQ_ERR_UNSUPPORTED;
    }
    return dispatch_stream_type(type, p, true, ctx->sm_count, vectors, s);
}

int rq_launch_gemv_stream(rq_ctx* ctx, const rq_weight* w, const float* x, int64_t sk, int64_t st, int tokens,
                          float* y, int64_t yn, int64_t yt, int act_mode, const uint8_t* act, int fuse_step, uint8_t* act_out, cudaStream_t s) {
    RqSegment seg;
    memset(&seg, 0, sizeof(seg));
    seg.row_begin = 0; seg.rows = (int)w->rows; seg.y = y;
    seg.main[0] = w->main; seg.scale[0] = w->scale; seg.act[0] = 0; seg.coef[0] = 1.0f;
    return rq_launch_stream(ctx, w->type, w->cols, nullptr, &seg, 1, 1, RQ_EPI_PLAIN, w->rows, x, sk, st, tokens, 0, yn, yt, act_mode, act, fuse_step, act_out, s);
}
