// Decode of one activation row through a small matrix: everything a CTA needs lies in shared memory, one pass, no ring, no cluster.
//
// A projection of a few MB streams from HBM in a microsecond, and with programmatic dependent launch its weights arrive under the kernel before
// it.  What is left is the chain from that kernel's end to this one's: 1536 -> 1536 in Q4_K took gemv_i8_kernel 4.7 us in a chain of its like, of
// which (clock(), at 1.9 GHz) load and quantisation of the row 1.3, the integer MMAs of one unit per warp 0.9, two cluster barriers and the K slices' sums
// through distributed shared memory 1.7.  A chain of kernels that only wait for one another takes 0.6 us per launch, with a load and a store 1.3,
// with two cluster barriers 2.4.  So here:
//   * a CTA holds whole rows: groups of 16 outputs (gated: of gate and of up), all of K, copied by one bulk copy per row, whose pitch in
//     shared memory is free and keeps the fragment loads off one another's banks;
//   * K lies over the warps: a warp quantises the units (256 columns) that it multiplies, for itself, and needs no barrier in between; with few units
//     more warps stand side by side over the groups and quantise the same units again;
//   * the warps' sums meet once, in shared memory; an RMSNorm in front costs one barrier more (every CTA computes it, a row is a few KB out of L2).
// The arithmetic is that of gemv_i8_kernel (zq_gemv_i8.cu): 16-bit integer activations, exact integer sums per unit, f32 across units.
// us per launch, gemv_i8_kernel or the work list and this kernel, 32 and more launches of different weights back to back:
//   Q4_K  512 -> 8192 3.5 / 2.9   1536 -> 1536 4.7 / 2.7   1536 -> 3840 4.9 / 2.9   3840 -> 1536 5.1 / 3.0   3840 -> 3840 5.9 / 4.1   5120 -> 3840 6.6 / 4.7
//   Q8_0  1536 -> 1536 4.6 / 2.7   2560 -> 3840 5.7 / 3.4   3840 -> 3840 6.4 / 4.7   5120 -> 3840 7.2 / 5.5
//   gated Q4_K  1536 -> 3840 5.8 / 3.8   2560 -> 3840 6.7 / 4.7   3840 -> 3840 7.7 / 6.8;   norm and 1536 -> 1536, 512, 512 6.6 / 3.6, of two types 7.3 / 3.5
#include <algorithm>

#include "zq_i8.cuh"
#include "zq_row.cuh"

namespace zq {

constexpr int kRowWarps = 16;      // most warps of a CTA
constexpr int kRowMaxGroups = 16;  // most groups of 16 weight rows of a CTA
constexpr int kRowTurns = 4;       // most units per warp
constexpr int kRowMaxSmem = 232448 - 1024;  // opt-in maximum minus static shared memory

struct RowJob {
    const uint8_t *w, *w_up;  // resident rows
    void *y;                  // [n_out]
    const void *residual;
    int n_out;
    int cta0;                 // first CTA of the job
    int y_dtype;
    uint32_t type;
};
struct RowArgs {
    RowJob jobs[kRowMaxJobs];
    int n_jobs;
    const void *x;
    int x_dtype, cols, units;
    int groups;            // groups of 16 outputs per CTA
    int lanes_k, lanes_g;  // warps side by side along K, and over the groups
    int turns;             // most units per warp
    int off_rec, off_red;  // shared memory: weights at 0, records [warp][turn], partial sums [warp along K][group][16]
    const float *norm_weight;
    float eps, weight_offset;
    bool x_wide, w_wide;
    uint32_t *status;
};

__host__ __device__ inline int row_unit_bytes(uint32_t type) { return type == ZQ_Q8_0 ? 272 : type == ZQ_Q6_K ? 224 : type == ZQ_Q5_K ? 176 : 144; }
// Bytes between rows in shared memory: whole 128-byte lines and a quarter (K-quants: eight-byte fragment loads of four rows) or a half (16-byte
// ones of two) of one more, which spreads the rows that one access touches over the banks.
__host__ __device__ inline int row_smem_pitch(uint32_t type, int units) { return ((units * row_unit_bytes(type) + 127) & ~127) + (type == ZQ_Q4_K || type == ZQ_Q5_K ? 32 : 64); }

template <uint32_t TYPE, bool GATED>
__global__ void __launch_bounds__(kRowWarps * 32, 1) gemv_row_kernel(const __grid_constant__ RowArgs a) {
    constexpr bool MIX = TYPE == 0;
    constexpr int PARTS = GATED ? 2 : 1;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    float *red = reinterpret_cast<float *>(smem + a.off_red);
    __shared__ uint64_t s_bar[kRowMaxGroups];  // a group's weights have arrived (gated: gate and up rows)
    __shared__ int s_abort;
    __shared__ float s_partial[kRowWarps];
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    int j = 0;
    while (j + 1 < a.n_jobs && a.jobs[j + 1].cta0 <= (int)blockIdx.x) ++j;
    const RowJob &jb = a.jobs[j];
    const uint32_t type = MIX ? jb.type : TYPE;
    const int ub = MIX ? row_unit_bytes(type) : Fmt<MIX ? (uint32_t)ZQ_Q4_K : TYPE>::unit_bytes;
    const int row0 = ((int)blockIdx.x - jb.cta0) * 16 * a.groups;
    const int rows = jb.n_out - row0 < 16 * a.groups ? jb.n_out - row0 : 16 * a.groups, groups = (rows + 15) >> 4;
    const uint32_t row_bytes = (uint32_t)(a.units * ub);
    const int pitch = row_smem_pitch(type, a.units);
    if (warp == 0) {
        if (lane < groups) mbar_init(&s_bar[lane], 1);
        if (lane == 0) s_abort = 0;
        fence_mbar_init();
        if (lane < groups) mbar_expect_tx(&s_bar[lane], (uint32_t)((rows - 16 * lane < 16 ? rows - 16 * lane : 16) * PARTS) * row_bytes);
        __syncwarp();
        for (int i = lane; i < 16 * PARTS * groups; i += 32) {  // rows of a group: 16 (gated: 16 of gate, 16 of up)
            const int grp = i / (16 * PARTS), r = 16 * grp + (i & 15);
            if (r < rows) bulk_load_1d(smem + i * pitch, (GATED && (i & 16) ? jb.w_up : jb.w) + (size_t)(row0 + r) * row_bytes, row_bytes, &s_bar[grp]);
        }
    }
    pdl_launch_dependents();
    __syncthreads();

    int ul = warp, ug = 0;
    for (; ul >= a.lanes_k; ul -= a.lanes_k) ++ug;
    const int g = lane >> 2, t = lane & 3;
    uint8_t *const rec_mine = smem + a.off_rec + warp * a.turns * kRec;
    auto store_rec = [&](int k, const float (&v)[8]) {
        uint8_t *dst = rec_mine + k * kRec;
        auto put = [&](auto kclass) {
            constexpr uint32_t T = decltype(kclass)::value ? (uint32_t)ZQ_Q4_K : (uint32_t)ZQ_Q4_0;
            const RecLane o = quantize_record<T>(v, lane);
            *reinterpret_cast<uint4 *>(dst + o.slot) = make_uint4(o.ph0, o.ph1, o.pl0, o.pl1);
            if (is_kclass(T) && (lane & 7) == 0) *reinterpret_cast<uint2 *>(dst + kRecSums + (lane >> 3) * 8) = make_uint2(o.sw0, o.sw1);
            if (lane == 0) *reinterpret_cast<float *>(dst + kRecScale) = o.scale;
        };
        if (MIX ? is_kclass(type) : is_kclass(TYPE)) put(std::true_type());
        else put(std::false_type());
    };

    pdl_wait_prior_grid();
    if (!GATED && a.norm_weight) {  // the arithmetic of rmsnorm_kernel (zq_norm.cu)
        float v[kRowTurns][8], w[kRowTurns][8];
        auto load = [&](const void *p, int dtype, bool wide, int k0, float (&o)[8]) {
            if (wide) {
                load_act8(p, dtype, (size_t)k0, k0 < a.cols, o);
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e) o[e] = k0 < a.cols ? load_as_f32(p, dtype, (size_t)k0 + e) : 0.f;
            }
        };
        float acc = 0.f;
#pragma unroll
        for (int k = 0; k < kRowTurns; ++k) {
            const int u = ul + k * a.lanes_k;
            if (u >= a.units) break;
            load(a.x, a.x_dtype, a.x_wide, u * kUnitWeights + 8 * lane, v[k]);
            load(a.norm_weight, ZQ_F32, a.w_wide, u * kUnitWeights + 8 * lane, w[k]);
        }
#pragma unroll
        for (int k = 0; k < kRowTurns; ++k) {
            if (ul + k * a.lanes_k >= a.units) break;
#pragma unroll
            for (int e = 0; e < 8; ++e) acc = fmaf(v[k][e], v[k][e], acc);
        }
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, s);
        if (lane == 0) s_partial[warp] = acc;
        __syncthreads();
        float total = (lane & 15) < a.lanes_k ? s_partial[lane & 15] : 0.f;
#pragma unroll
        for (int s = 8; s > 0; s >>= 1) total += __shfl_xor_sync(0xFFFFFFFFu, total, s);
        const float inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(total, (float)a.cols), a.eps)));
#pragma unroll
        for (int k = 0; k < kRowTurns; ++k) {
            const int u = ul + k * a.lanes_k;
            if (u >= a.units) break;
            const bool valid = u * kUnitWeights + 8 * lane < a.cols;
#pragma unroll
            for (int e = 0; e < 8; ++e) v[k][e] = valid ? __fmul_rn(__fmul_rn(v[k][e], inv), a.weight_offset == 0.0f ? w[k][e] : __fadd_rn(a.weight_offset, w[k][e])) : 0.f;
            store_rec(k, v[k]);
        }
    } else {
        float v[8];
        int k0 = ul * kUnitWeights + 8 * lane;
        load_act8(a.x, a.x_dtype, (size_t)k0, k0 < a.cols, v);
        store_rec(0, v);
        for (int k = 1; ul + k * a.lanes_k < a.units; ++k) {
            k0 += a.lanes_k * kUnitWeights;
            load_act8(a.x, a.x_dtype, (size_t)k0, k0 < a.cols, v);
            store_rec(k, v);
        }
    }
    __syncwarp();

    const uint32_t rec0 = smem_u32(rec_mine), xoff = (uint32_t)(16 * t + 8 * (g & 1));
    const int items = PARTS * groups;
    float *const red_mine = red + ul * PARTS * a.groups * 16 + g;
    for (int i = ug; i < items; i += a.lanes_g) {  // gated: gate and up of a group in turn
        i8_wait_or_abort(&s_bar[GATED ? i >> 1 : i], 0, &s_abort, a.status);
        uint32_t w_at = smem_u32(smem) + (uint32_t)((16 * i + g) * pitch + ul * ub), ru = rec0;
        float yacc[1][2] = {{0.f, 0.f}};
        for (int u = ul; u < a.units; u += a.lanes_k) {
            const uint32_t wq0 = w_at, wq1 = wq0 + (uint32_t)(8 * pitch);
            const uint32_t rec[1] = {ru}, srec[1] = {ru};
            if constexpr (MIX) {
                switch (type) {
                case ZQ_Q4_K: consume_q4k_i8<1, false>(wq0, wq1, t, rec, srec, xoff, yacc); break;
                case ZQ_Q5_K: consume_q4k_i8<1, true>(wq0, wq1, t, rec, srec, xoff, yacc); break;
                case ZQ_Q6_K: consume_q6k_i8<1>(wq0, wq1, t, rec, srec, xoff, yacc); break;
                case ZQ_Q4_0: consume_b32_i8<ZQ_Q4_0, 1>(wq0, wq1, t, rec, srec, xoff, yacc); break;
                case ZQ_IQ4_NL: consume_b32_i8<ZQ_IQ4_NL, 1>(wq0, wq1, t, rec, srec, xoff, yacc); break;
                default: consume_b32_i8<ZQ_Q8_0, 1>(wq0, wq1, t, rec, srec, xoff, yacc); break;
                }
            } else if constexpr (TYPE == ZQ_Q6_K) consume_q6k_i8<1>(wq0, wq1, t, rec, srec, xoff, yacc);
            else if constexpr (is_kclass(TYPE)) consume_q4k_i8<1, TYPE == ZQ_Q5_K>(wq0, wq1, t, rec, srec, xoff, yacc);
            else consume_b32_i8<MIX ? (uint32_t)ZQ_Q8_0 : TYPE, 1>(wq0, wq1, t, rec, srec, xoff, yacc);
            w_at += (uint32_t)(a.lanes_k * ub);
            ru += kRec;
        }
        if (t == 0) {
            red_mine[16 * i] = yacc[0][0];
            red_mine[16 * i + 8] = yacc[0][1];
        }
    }
    __syncthreads();
    for (int i = tid; i < rows; i += blockDim.x) {
        const int o = row0 + i;
        float res = 0.f;
        if (!GATED && jb.residual) res = load_as_f32(jb.residual, jb.y_dtype, (size_t)o);
        auto total_of = [&](int at) {
            const float *p = red + at;
            const int stride = PARTS * a.groups * 16;
            float s = 0.f;
            for (int w = 0; w < a.lanes_k; w += 4) {
                float q[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) q[e] = w + e < a.lanes_k ? p[(w + e) * stride] : 0.f;
                s = (s + (q[0] + q[1])) + (q[2] + q[3]);  // as the work-list kernel adds chunks of two units that are a CTA each
            }
            return s;
        };
        float v;
        if (GATED) {
            const float gate = total_of(32 * (i >> 4) + (i & 15)), up = total_of(32 * (i >> 4) + 16 + (i & 15));
            v = (gate / (1.0f + expf(-gate))) * up;
        } else {
            v = total_of(i) + res;
        }
        store_from_f32(jb.y, jb.y_dtype, (size_t)o, v);
    }
}

// Takes a call where its weights fit into the shared memory of the SMs.  Two CTAs per SM where registers and shared memory let them: the
// groups spread more evenly, and one copies while the other multiplies; else one CTA, up to 200 KB.  Two against one, us: Q4_K 512 -> 8192 2.9 / 3.2,
// 2560 -> 8192 4.6 / 5.8, gated 1536 -> 3840 3.8 / 4.5, 2560 -> 3840 4.7 / 6.0; where the second does not fit beside the first (3840 -> 3840, 15 warps) 5.8 / 4.1.
// What does not fit is a matter of bandwidth and stays with the ring kernels: Q4_K 3840 -> 8192 (17.7 MB) 7.7 there, 6.7 here; 5120 -> 8192 (23.6 MB) 8.9 and 8.7.
template <uint32_t TYPE, bool GATED> static int launch_row_one(zq_ctx *ctx, const RowCall &c, bool &taken, zq_error *err) {
    constexpr size_t PARTS = GATED ? 2 : 1;
    auto kernel = gemv_row_kernel<TYPE, GATED>;
    static size_t warp_regs[64] = {};
    size_t &regs = warp_regs[ctx->device & 63];
    if (!regs) {
        cudaFuncAttributes fa;
        ZQ_CUDA_CHECK(cudaFuncGetAttributes(&fa, kernel), err);
        ZQ_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kRowMaxSmem), err);
        regs = (size_t)((fa.numRegs + 7) & ~7) * 32;
    }
    const size_t units = c.jobs[0].w->units_per_row, turns = (units + kRowWarps - 1) / kRowWarps, lanes_k = (units + turns - 1) / turns;
    if (turns > (size_t)kRowTurns) return ZQ_OK;
    // Gated pairs of many outputs from few columns, and IQ4_NL's of more than 16 units, are as fast or faster where a K slice is a CTA: IQ4_NL 1024 -> 8192 5.8 there,
    // 6.3 here, 8192 -> 512 6.9 / 7.3; Q6_K 512 -> 8192 4.3 / 4.4.
    if (GATED && (c.jobs[0].w->rows >= 8 * c.jobs[0].w->cols || (TYPE == ZQ_IQ4_NL && turns > 1))) return ZQ_OK;
    size_t row = 0, all = 0;
    for (int i = 0; i < c.n_jobs; ++i) {
        row = std::max(row, (size_t)row_smem_pitch(c.jobs[i].w->type, (int)units));
        all += (c.jobs[i].w->rows + 15) / 16;
    }
    RowArgs ra;
    size_t grid = 0, warps = 0, smem = 0;
    for (size_t per_sm = 2; per_sm >= 1 && !taken; --per_sm) {
        const size_t ctas = (size_t)ctx->sm_count * per_sm;
        size_t groups = (all + ctas - 1) / ctas;
        for (; groups <= (size_t)kRowMaxGroups; ++groups) {  // every job starts on a CTA of its own
            grid = 0;
            for (int i = 0; i < c.n_jobs; ++i) grid += ((c.jobs[i].w->rows + 15) / 16 + groups - 1) / groups;
            if (grid <= ctas) break;
        }
        if (groups > (size_t)kRowMaxGroups) continue;
        size_t lanes_g = 1;
        while (2 * lanes_g * lanes_k <= (size_t)kRowWarps && 2 * lanes_g <= groups * PARTS && per_sm * 2 * lanes_g * lanes_k * regs <= 65536) lanes_g *= 2;
        warps = lanes_k * lanes_g;
        const size_t w_bytes = 16 * groups * PARTS * row, rec = warps * turns * kRec;
        smem = w_bytes + rec + lanes_k * groups * PARTS * 16 * sizeof(float) + 128;
        if (per_sm * warps * regs > 65536 || smem > (per_sm == 2 ? (size_t)kRowMaxSmem / 2 - 1024 : (size_t)200 << 10)) continue;
        ra.groups = (int)groups;
        ra.lanes_k = (int)lanes_k;
        ra.lanes_g = (int)lanes_g;
        ra.turns = (int)turns;
        ra.off_rec = (int)w_bytes;
        ra.off_red = (int)(w_bytes + rec);
        taken = true;
    }
    if (!taken) return ZQ_OK;
    grid = 0;
    for (int i = 0; i < c.n_jobs; ++i) {
        const zq_weight *w = c.jobs[i].w;
        ra.jobs[i] = {w->data, GATED ? c.jobs[i].w_up->data : nullptr, c.jobs[i].y, c.jobs[i].residual, (int)w->rows, (int)grid, c.jobs[i].y_dtype, w->type};
        grid += ((w->rows + 15) / 16 + ra.groups - 1) / ra.groups;
    }
    ra.n_jobs = c.n_jobs;
    ra.x = c.x;
    ra.x_dtype = c.x_dtype;
    ra.cols = (int)c.jobs[0].w->cols;
    ra.units = (int)units;
    ra.norm_weight = c.norm ? c.norm->weight : nullptr;
    ra.eps = c.norm ? c.norm->eps : 0.f;
    ra.weight_offset = c.norm ? c.norm->weight_offset : 0.f;
    ra.x_wide = (reinterpret_cast<uintptr_t>(c.x) & 15) == 0;
    ra.w_wide = c.norm && (reinterpret_cast<uintptr_t>(c.norm->weight) & 15) == 0;
    ra.status = ctx->status_dev;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)(32 * warps));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ctx->disable_pdl ? 0 : 1;
    ZQ_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, ra), err);
    ctx->launches++;
    return ZQ_OK;
}

int launch_gemv_row(zq_ctx *ctx, const RowCall &c, bool &taken, zq_error *err) {
    taken = false;
    if (c.n_jobs < 1 || c.n_jobs > kRowMaxJobs) return ZQ_OK;
    const bool gated = c.jobs[0].w_up != nullptr;
    uint32_t type = c.jobs[0].w->type;
    for (int i = 0; i < c.n_jobs; ++i) {
        const zq_weight *w = c.jobs[i].w;
        if (!has_i8_decode(w->type) || w->units_per_row != c.jobs[0].w->units_per_row || w->row_pitch != w->units_per_row * (size_t)row_unit_bytes(w->type)) return ZQ_OK;
        if (w->type != type) type = 0;
    }
#define ZQ_ROW_CASE(T) case T: return gated ? launch_row_one<T, true>(ctx, c, taken, err) : launch_row_one<T, false>(ctx, c, taken, err)
    switch (type) {
        ZQ_ROW_CASE(ZQ_Q4_K);
        ZQ_ROW_CASE(ZQ_Q5_K);
        ZQ_ROW_CASE(ZQ_Q6_K);
        ZQ_ROW_CASE(ZQ_Q4_0);
        ZQ_ROW_CASE(ZQ_IQ4_NL);
        ZQ_ROW_CASE(ZQ_Q8_0);
    default: return launch_row_one<0, false>(ctx, c, taken, err);
    }
#undef ZQ_ROW_CASE
}

}  // namespace zq
