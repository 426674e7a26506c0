// RMSNorm in front of a quantized projection: Backend::rmsnorm_linear / rmsnorm_dual_linear
// (src/backend/mod.rs:455-464) = rmsnorm (src/kernel/cpu/rmsnorm.rs:7-41), then the linear layer(s).
//   out[i] = x[i] * (1 / sqrt(mean(x^2) + eps)) * (w[i] + weight_offset)     (offset 1 = the "Gemma" form)
// One CTA per activation row.  Two forms of the result:
//   f32 rows in a context buffer, for projections that take their input as it is (more than 16 rows, other kernels)
//   activation records (zq_i8.cuh) of one or both record formats, what the work-list decode kernel reads: the record pass, its
//   launch and the trip of the normalised row through memory disappear
// The projection that follows is launched with programmatic dependent launch, so its weight prefetch runs under this kernel.
// The operation order of the scaling is the reference's (x * inv_rms, then * weight); the sum of squares is a tree sum, which
// differs from the reference's 8-lane running sums in the last bits only.
//
// Latency bounds it (a row is a few KB and everything behind it waits): all loads of a row and of the norm weights, 8
// consecutive columns per thread and turn, are in flight together, and the values stay in registers between the sum and the
// scaling.  With a scalar load per turn and a second read of the row, 3840 columns took 16 us; now 3 to 4 us with the records.
#include "zq_i8.cuh"
#include "zq_wl.cuh"

namespace zq {

struct NormArgs {
    const void *x;
    const float *weight;
    int x_dtype, cols;
    float eps, weight_offset;
    bool x_wide, w_wide;    // 16-byte aligned rows / weights: vector loads
    float *out;             // f32 rows, or null
    uint8_t *rec_k, *rec_b; // records of the K-quant / block-32 format, [unit][row], each or null
};

constexpr int kNormThreads = 512, kNormHeld = 4;  // 4 x 8 columns per thread stay in registers: rows up to 16 384 columns

// Columns 8 c .. 8 c + 7 of a row that starts at element `base` (zeros past the row: rows are whole 32-column blocks).
__device__ __forceinline__ void norm_load(const NormArgs &a, size_t base, int c, float (&v)[8]) {
    const bool valid = 8 * c < a.cols;
    if (a.x_wide) {
        load_act8(a.x, a.x_dtype, base + 8 * (size_t)c, valid, v);
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = valid ? load_as_f32(a.x, a.x_dtype, base + 8 * (size_t)c + j) : 0.f;
    }
}
__device__ __forceinline__ void norm_weights(const NormArgs &a, int c, float (&w)[8]) {
    const bool valid = 8 * c < a.cols;
    if (a.w_wide) {
        load_act8(a.weight, ZQ_F32, 8 * (size_t)c, valid, w);
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) w[j] = valid ? a.weight[8 * c + j] : 0.f;
    }
}
template <uint32_t TYPE> __device__ __forceinline__ void norm_store_record(uint8_t *dst, const float (&v)[8], int lane) {
    const RecLane o = quantize_record<TYPE>(v, lane);
    *reinterpret_cast<uint4 *>(dst + o.slot) = make_uint4(o.ph0, o.ph1, o.pl0, o.pl1);
    if (is_kclass(TYPE) && (lane & 7) == 0) *reinterpret_cast<uint2 *>(dst + kRecSums + (lane >> 3) * 8) = make_uint2(o.sw0, o.sw1);
    if (lane == 0) *reinterpret_cast<float *>(dst + kRecScale) = o.scale;
}

__global__ void __launch_bounds__(kNormThreads) rmsnorm_kernel(const __grid_constant__ NormArgs a) {
    pdl_launch_dependents();
    pdl_wait_prior_grid();  // the input belongs to the previous kernel until it completes, the record buffer to its readers
    __shared__ float partial[kNormThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const size_t base = (size_t)blockIdx.x * a.cols;
    const int turns = ((a.cols + 255) / 256 * 32 + kNormThreads - 1) / kNormThreads;  // a warp's turn is a 256-column unit
    float v[kNormHeld][8], w[kNormHeld][8];
#pragma unroll
    for (int i = 0; i < kNormHeld; ++i) {
        if (i < turns) {
            norm_load(a, base, tid + i * kNormThreads, v[i]);
            norm_weights(a, tid + i * kNormThreads, w[i]);
        }
    }
    float acc = 0.f;
#pragma unroll
    for (int i = 0; i < kNormHeld; ++i) {
        if (i < turns) {
#pragma unroll
            for (int j = 0; j < 8; ++j) acc = fmaf(v[i][j], v[i][j], acc);
        }
    }
    for (int i = kNormHeld; i < turns; ++i) {
        float u[8];
        norm_load(a, base, tid + i * kNormThreads, u);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc = fmaf(u[j], u[j], acc);
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, s);
    if (lane == 0) partial[warp] = acc;
    __syncthreads();
    float total = partial[lane & (kNormThreads / 32 - 1)];
#pragma unroll
    for (int s = kNormThreads / 64; s > 0; s >>= 1) total += __shfl_xor_sync(0xFFFFFFFFu, total, s);
    const float inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(total, (float)a.cols), a.eps)));
    auto finish = [&](int c, float (&x)[8], const float (&wt)[8]) {  // c - lane is a multiple of 32: the warp holds one unit
        if (c - lane >= (a.cols + 255) / 256 * 32) return;  // warp-uniform
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = __fmul_rn(__fmul_rn(x[j], inv), a.weight_offset == 0.0f ? wt[j] : __fadd_rn(a.weight_offset, wt[j]));
        if (a.out) {
            if (8 * c < a.cols) {
                float4 *dst = reinterpret_cast<float4 *>(a.out + base + 8 * (size_t)c);
                dst[0] = make_float4(x[0], x[1], x[2], x[3]);
                dst[1] = make_float4(x[4], x[5], x[6], x[7]);
            }
            return;
        }
        if (8 * c >= a.cols) {  // past the row: zeros (an infinite inv would make them NaN)
#pragma unroll
            for (int j = 0; j < 8; ++j) x[j] = 0.f;
        }
        const size_t rec = ((size_t)(c >> 5) * gridDim.x + blockIdx.x) * kRec;
        if (a.rec_k) norm_store_record<ZQ_Q4_K>(a.rec_k + rec, x, lane);
        if (a.rec_b) norm_store_record<ZQ_Q4_0>(a.rec_b + rec, x, lane);
    };
#pragma unroll
    for (int i = 0; i < kNormHeld; ++i) {
        if (i < turns) finish(tid + i * kNormThreads, v[i], w[i]);
    }
    for (int i = kNormHeld; i < turns; ++i) {
        float u[8], wt[8];
        norm_load(a, base, tid + i * kNormThreads, u);
        norm_weights(a, tid + i * kNormThreads, wt);
        finish(tid + i * kNormThreads, u, wt);
    }
}

static int launch_norm(zq_ctx *ctx, size_t m, NormArgs &a, zq_error *err) {
    a.x_wide = (reinterpret_cast<uintptr_t>(a.x) & 15) == 0;  // rows are multiples of 64 bytes
    a.w_wide = (reinterpret_cast<uintptr_t>(a.weight) & 15) == 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)m);
    cfg.blockDim = dim3(kNormThreads);
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ctx->disable_pdl ? 0 : 1;
    ZQ_CUDA_CHECK(cudaLaunchKernelEx(&cfg, rmsnorm_kernel, a), err);
    ctx->launches++;
    return ZQ_OK;
}

int launch_rmsnorm(zq_ctx *ctx, const void *x, int x_dtype, size_t m, size_t cols, const float *weight, float eps, float weight_offset, float *out, zq_error *err) {
    NormArgs a = {x, weight, x_dtype, (int)cols, eps, weight_offset, false, false, out, nullptr, nullptr};
    return launch_norm(ctx, m, a, err);
}

int launch_rmsnorm_records(zq_ctx *ctx, const WlNorm &norm, size_t m, size_t cols, uint8_t *rec_k, uint8_t *rec_b, zq_error *err) {
    NormArgs a = {norm.x, norm.weight, norm.x_dtype, (int)cols, norm.eps, norm.weight_offset, false, false, nullptr, rec_k, rec_b};
    return launch_norm(ctx, m, a, err);
}

}  // namespace zq

// ---------------------------------------------------------------------------------------------------------------
// Arg-max over the columns of every row: the greedy token choice behind an LM-head projection, left on the device so
// that the logits (vocabulary x 4 bytes per row) never travel to the host.  Ties go to the lower index; NaN entries are
// never chosen (a row of nothing but NaN yields index 0).  One CTA per row.
// ---------------------------------------------------------------------------------------------------------------
namespace zq {

__global__ void __launch_bounds__(1024) argmax_rows_kernel(const void *__restrict__ x, int dtype, int cols, uint32_t *__restrict__ out) {
    pdl_launch_dependents();
    pdl_wait_prior_grid();
    const size_t row = blockIdx.x;
    float best = -INFINITY;
    int best_i = 0x7fffffff;
    for (int c = threadIdx.x; c < cols; c += blockDim.x) {
        const float v = load_as_f32(x, dtype, row * cols + c);
        if (v > best || (v == best && c < best_i)) { best = v; best_i = c; }
    }
    __shared__ float s_best[32];
    __shared__ int s_idx[32];
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
        if (ov > best || (ov == best && oi < best_i)) { best = ov; best_i = oi; }
    }
    if ((threadIdx.x & 31) == 0) {
        s_best[threadIdx.x >> 5] = best;
        s_idx[threadIdx.x >> 5] = best_i;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const int warps = (blockDim.x + 31) / 32;
        best = threadIdx.x < warps ? s_best[threadIdx.x] : -INFINITY;
        best_i = threadIdx.x < warps ? s_idx[threadIdx.x] : 0x7fffffff;
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
            if (ov > best || (ov == best && oi < best_i)) { best = ov; best_i = oi; }
        }
        if (threadIdx.x == 0) out[row] = best_i == 0x7fffffff ? 0u : (uint32_t)best_i;
    }
}

}  // namespace zq

extern "C" int zq_argmax_rows(zq_ctx *ctx, const void *dev_x, int dtype, size_t rows, size_t cols, uint32_t *dev_ids, zq_error *err) {
    using namespace zq;
    if (!ctx || !dev_x || !dev_ids) return set_error(err, ZQ_ERR_ARG, "zq_argmax_rows: null argument");
    if (dtype != ZQ_F32 && dtype != ZQ_F16 && dtype != ZQ_BF16) return set_error(err, ZQ_ERR_ARG, "zq_argmax_rows: unknown dtype %d", dtype);
    if (rows == 0 || cols == 0 || cols > (size_t)INT32_MAX || rows > (size_t)INT32_MAX) return set_error(err, ZQ_ERR_SHAPE, "zq_argmax_rows: shape [%zu, %zu]", rows, cols);
    int rc = use_device(ctx, err);
    if (rc) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)rows);
    cfg.blockDim = dim3(1024);
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ctx->disable_pdl ? 0 : 1;
    ZQ_CUDA_CHECK(cudaLaunchKernelEx(&cfg, argmax_rows_kernel, dev_x, dtype, (int)cols, dev_ids), err);
    ctx->launches++;
    return ZQ_OK;
}

// LM head: logits = W x into a context buffer (f32), then the arg-max of every row.
extern "C" int zq_lm_head_argmax(zq_ctx *ctx, const zq_weight *head, const void *dev_x, int x_dtype, size_t m, uint32_t *dev_ids, zq_error *err) {
    using namespace zq;
    if (!ctx || !head || !dev_x || !dev_ids) return set_error(err, ZQ_ERR_ARG, "zq_lm_head_argmax: null argument");
    if (m == 0) return set_error(err, ZQ_ERR_SHAPE, "zq_lm_head_argmax: no rows");
    int rc = ensure_scratch_norm(ctx, m * head->rows * sizeof(float) + 256, err);  // the logits share the buffer of the normalised rows
    if (rc) return rc;
    rc = zq_linear(ctx, head, dev_x, x_dtype, m, ctx->norm, ZQ_F32, nullptr, err);
    if (rc) return rc;
    return zq_argmax_rows(ctx, ctx->norm, ZQ_F32, m, head->rows, dev_ids, err);
}
