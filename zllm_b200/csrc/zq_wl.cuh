// Host-side interface of the work-list decode kernel (zq_gemv_wl.cu): a list of independent projections, each
// y[m, rows] = x[m, cols] W^T (+ residual), or silu(x gate^T) * (x up^T) when `w_up` is given, run in as few launches as
// their (weight type, row count, plain / gated) classes allow: one for a list of plain jobs of up to 4 rows, whatever their types, that needs few
// activation records per CTA.
#pragma once
#include "zq_common.cuh"

namespace zq {

constexpr int kWlMaxJobs = 32;  // jobs per launch (the job table travels as a kernel parameter)

struct WlHostJob {
    const zq_weight *w;
    const zq_weight *w_up;  // gated pair, or null
    const void *x;          // [m, cols]
    size_t m;               // 1..16
    void *y;                // [m, rows]
    const void *residual;   // [m, rows] in the output dtype, or null
    int y_dtype;            // output dtype of this job, or -1 for the call's
};

// True when the job can ride in a work-list launch (Q4_K / Q5_K / Q6_K / Q4_0 / IQ4_NL / Q8_0, up to 16 activation rows).
bool gemv_wl_supported(const zq_ctx *ctx, const WlHostJob &job);
// True when one gated pair (supported) is better dealt out by this kernel than launched on gemv_i8_kernel.
bool gated_prefers_worklist(const zq_ctx *ctx, const zq_weight *gate, size_t m);
// An RMSNorm in front of the list: every job's input is norm(x), and the jobs' own `x` is only the name of that one input.
struct WlNorm {
    const void *x;
    const float *weight;
    int x_dtype;
    float eps, weight_offset;
};
int launch_gemv_wl(zq_ctx *ctx, const WlHostJob *jobs, size_t n_jobs, int x_dtype, int y_dtype, zq_error *err, const WlNorm *norm = nullptr, bool own_scratch = false);
// norm(x) as activation records of the K-quant and / or block-32 format (zq_norm.cu); null: format not wanted.
int launch_rmsnorm_records(zq_ctx *ctx, const WlNorm &norm, size_t m, size_t cols, uint8_t *rec_k, uint8_t *rec_b, zq_error *err);

}  // namespace zq
