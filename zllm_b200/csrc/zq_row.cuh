// Host-side interface of the one-row decode kernels, resident and streamed (zq_gemv_row.cu).
#pragma once
#include "zq_wl.cuh"

namespace zq {

constexpr int kRowMaxJobs = 4;  // zq_rmsnorm_linear fills three; with room for three alone every call takes 0.4 us longer (one projection 3.6 us, 4.0)
struct RowHostJob {
    const zq_weight *w, *w_up;  // w_up: gated pair
    void *y;
    const void *residual;
    int y_dtype;
};
// Projections of one input row, all plain or one gated pair; norm: an RMSNorm in front.
struct RowCall {
    RowHostJob jobs[kRowMaxJobs];
    int n_jobs;
    const void *x;
    int x_dtype;
    const WlNorm *norm;
};
int launch_gemv_row(zq_ctx *ctx, const RowCall &c, bool &taken, zq_error *err);

}  // namespace zq
