// Decode of one activation row: whole rows of the weight per CTA, K over its warps, no cluster and nothing shared between CTAs.  Small matrices lie in
// shared memory at once (gemv_row_kernel), larger ones go through a ring of row groups (gemv_row_stream_kernel).
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
constexpr int kRowSums = 4;        // groups whose sums may wait to be added up
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
    int groups;            // groups of 16 outputs per CTA; streamed: stages of the ring
    int all_groups, stage_bytes;  // streamed: groups of all jobs (cta0: a job's first group), bytes of a stage
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

// The records of the units that this warp multiplies (unit ul, ul + lanes_k, ..), one after the other in its own place; with a norm in front all `threads` of
// these warps meet once.
template <uint32_t TYPE, bool GATED> __device__ __forceinline__ void row_records(const RowArgs &a, uint32_t type, uint8_t *rec_mine, int ul, int warp, int lane, int threads, float *s_partial) {
    constexpr bool MIX = TYPE == 0;
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
        asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
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
}

// One unit of 16 rows: wq0 is fragment row g of it, `pitch` bytes between rows.
template <uint32_t TYPE> __device__ __forceinline__ void row_unit(uint32_t type, uint32_t wq0, int pitch, int t, uint32_t ru, uint32_t xoff, float (&yacc)[1][2]) {
    const uint32_t wq1 = wq0 + (uint32_t)(8 * pitch);
    const uint32_t rec[1] = {ru}, srec[1] = {ru};
    if constexpr (TYPE == 0) {
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
    else consume_b32_i8<TYPE, 1>(wq0, wq1, t, rec, srec, xoff, yacc);
}

// The sum of one output over the warps along K, `stride` floats apart: pairs in turn.  That is the order of the cluster and work-list kernels where each chunk of two
// units is a CTA's there; where a CTA has several chunks they keep one running sum per half of a unit pair, and here a warp of several units (more
// than 16 of a row) adds its own first, so that f32 sums differ in their last bits.
__device__ __forceinline__ float row_total(const float *p, int lanes_k, int stride) {
    float s = 0.f;
    for (int w = 0; w < lanes_k; w += 4) {
        float q[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) q[e] = w + e < lanes_k ? p[(w + e) * stride] : 0.f;
        s = (s + (q[0] + q[1])) + (q[2] + q[3]);
    }
    return s;
}

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
    pdl_wait_prior_grid();
    row_records<TYPE, GATED>(a, type, rec_mine, ul, warp, lane, (int)blockDim.x, s_partial);
    __syncwarp();

    const uint32_t rec0 = smem_u32(rec_mine), xoff = (uint32_t)(16 * t + 8 * (g & 1));
    const int items = PARTS * groups;
    float *const red_mine = red + ul * PARTS * a.groups * 16 + g;
    for (int i = ug; i < items; i += a.lanes_g) {  // gated: gate and up of a group in turn
        i8_wait_or_abort(&s_bar[GATED ? i >> 1 : i], 0, &s_abort, a.status);
        uint32_t w_at = smem_u32(smem) + (uint32_t)((16 * i + g) * pitch + ul * ub), ru = rec0;
        float yacc[1][2] = {{0.f, 0.f}};
        for (int u = ul; u < a.units; u += a.lanes_k) {
            row_unit<TYPE>(type, w_at, pitch, t, ru, xoff, yacc);
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
        const int stride = PARTS * a.groups * 16;
        float v;
        if (GATED) {
            const float gate = row_total(red + 32 * (i >> 4) + (i & 15), a.lanes_k, stride), up = row_total(red + 32 * (i >> 4) + 16 + (i & 15), a.lanes_k, stride);
            v = (gate / (1.0f + expf(-gate))) * up;
        } else {
            v = row_total(red + i, a.lanes_k, stride) + res;
        }
        store_from_f32(jb.y, jb.y_dtype, (size_t)o, v);
    }
}

// The same for matrices past the SMs' shared memory: one CTA per SM walks an equal share of the groups through a ring of groups (gated: of gate
// and up rows in turn).  A producer warp copies, the warps along K multiply their units of every group, a warp of its own adds up and stores; nobody
// meets anybody but at the stages' barriers.  Unlike the ring kernels it cuts no tile, quantises the row once per CTA and shares no result between CTAs.
template <uint32_t TYPE, bool GATED>
__global__ void __launch_bounds__((kRowWarps + 2) * 32, 1) gemv_row_stream_kernel(const __grid_constant__ RowArgs a) {
    constexpr bool MIX = TYPE == 0;
    constexpr int PARTS = GATED ? 2 : 1;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    float *red = reinterpret_cast<float *>(smem + a.off_red);  // [buffer][part][warp along K][16]
    __shared__ uint64_t s_full[kRowMaxGroups], s_empty[kRowMaxGroups], s_sums[kRowSums], s_free[kRowSums];
    __shared__ int s_abort;
    __shared__ float s_partial[kRowWarps];
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int consumers = a.lanes_k * a.lanes_g, S = a.groups;
    const int g0 = (int)((long long)blockIdx.x * a.all_groups / gridDim.x), g1 = (int)((long long)(blockIdx.x + 1) * a.all_groups / gridDim.x);
    if (tid == 0) {
        for (int i = 0; i < S; ++i) {
            mbar_init(&s_full[i], 1);
            mbar_init(&s_empty[i], (uint32_t)a.lanes_k);
        }
        for (int i = 0; i < kRowSums; ++i) {
            mbar_init(&s_sums[i], (uint32_t)(PARTS * a.lanes_k));
            mbar_init(&s_free[i], 1);
        }
        fence_mbar_init();
        s_abort = 0;
    }
    pdl_launch_dependents();
    __syncthreads();
    int j = 0;
    auto job_of = [&](int g) -> const RowJob & {  // cta0: the job's first group
        while (j + 1 < a.n_jobs && a.jobs[j + 1].cta0 <= g) ++j;
        return a.jobs[j];
    };
    if (warp == consumers) {
        // ------------------------------------------------ copies: a row per lane
        int s = 0;
        uint32_t ph = 0;
        bool fresh = true;
        for (int g = g0; g < g1; ++g) {
            const RowJob &jb = job_of(g);
            const int ub = MIX ? row_unit_bytes(jb.type) : Fmt<MIX ? (uint32_t)ZQ_Q4_K : TYPE>::unit_bytes, pitch = row_smem_pitch(MIX ? jb.type : TYPE, a.units);
            const uint32_t row_bytes = (uint32_t)(a.units * ub);
            const int row0 = (g - jb.cta0) * 16, rows = jb.n_out - row0 < 16 ? jb.n_out - row0 : 16;
#pragma unroll
            for (int part = 0; part < PARTS; ++part) {
                if (!fresh) {
                    i8_wait_or_abort(&s_empty[s], ph ^ 1u, &s_abort, a.status);
                    if (i8_warp_aborts(&s_abort)) return;  // never start a copy nobody will wait for
                }
                if (lane == 0) mbar_expect_tx(&s_full[s], (uint32_t)rows * row_bytes);
                __syncwarp();
                if (lane < rows) bulk_load_1d(smem + s * a.stage_bytes + lane * pitch, (part ? jb.w_up : jb.w) + (size_t)(row0 + lane) * row_bytes, row_bytes, &s_full[s]);
                if (++s == S) {
                    s = 0;
                    ph ^= 1u;
                    if (fresh) pdl_wait_prior_grid();  // weights are constants; but no bounded wait may count while an earlier kernel still runs
                    fresh = false;
                }
            }
        }
        return;
    }
    pdl_wait_prior_grid();
    if (warp == consumers + 1) {
        // ------------------------------------------------ sums over the warps, epilogue
        int b = 0;
        uint32_t ph = 0;
        for (int g = g0; g < g1; ++g) {
            const RowJob &jb = job_of(g);
            const int o = (g - jb.cta0) * 16 + (lane & 15);
            const bool mine = lane < 16 && o < jb.n_out;
            const float res = !GATED && mine && jb.residual ? load_as_f32(jb.residual, jb.y_dtype, (size_t)o) : 0.f;
            i8_wait_or_abort(&s_sums[b], ph, &s_abort, a.status);
            if (i8_warp_aborts(&s_abort)) return;
            // gated: lanes 0..15 add gate, lanes 16..31 up
            float v = row_total(red + ((b * PARTS + (GATED ? lane >> 4 : 0)) * a.lanes_k) * 16 + (lane & 15), a.lanes_k, 16);
            if (GATED) {
                const float up = __shfl_down_sync(0xffffffffu, v, 16);
                v = (v / (1.0f + expf(-v))) * up;
            } else {
                v += res;
            }
            if (mine) store_from_f32(jb.y, jb.y_dtype, (size_t)o, v);
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_free[b]);
            if (++b == kRowSums) {
                b = 0;
                ph ^= 1u;
            }
        }
        return;
    }
    // ---------------------------------------------------- warps along K
    int ul = warp, ug = 0;
    for (; ul >= a.lanes_k; ul -= a.lanes_k) ++ug;
    const int g = lane >> 2, t = lane & 3;
    uint8_t *const rec_mine = smem + a.off_rec + warp * a.turns * kRec;
    const uint32_t type0 = MIX ? job_of(g0).type : TYPE;
    uint32_t rec_type = type0;
    row_records<TYPE, GATED>(a, rec_type, rec_mine, ul, warp, lane, consumers * 32, s_partial);
    __syncwarp();
    const uint32_t rec0 = smem_u32(rec_mine), xoff = (uint32_t)(16 * t + 8 * (g & 1));
    int s = ug;
    uint32_t ph = 0;
    for (int i = ug; i < PARTS * (g1 - g0); i += a.lanes_g) {
        const int n = GATED ? i >> 1 : i, part = GATED ? i & 1 : 0, b = n & (kRowSums - 1);
        const RowJob &jb = job_of(g0 + n);
        const uint32_t type = MIX ? jb.type : TYPE;
        const int ub = MIX ? row_unit_bytes(type) : Fmt<MIX ? (uint32_t)ZQ_Q4_K : TYPE>::unit_bytes, pitch = row_smem_pitch(type, a.units);
        i8_wait_or_abort(&s_full[s], ph, &s_abort, a.status);
        uint32_t w_at = smem_u32(smem) + (uint32_t)(s * a.stage_bytes + g * pitch + ul * ub), ru = rec0;
        float yacc[1][2] = {{0.f, 0.f}};
        for (int u = ul; u < a.units; u += a.lanes_k) {
            row_unit<TYPE>(type, w_at, pitch, t, ru, xoff, yacc);
            w_at += (uint32_t)(a.lanes_k * ub);
            ru += kRec;
        }
        if (n >= kRowSums) i8_wait_or_abort(&s_free[b], (uint32_t)(n / kRowSums - 1) & 1u, &s_abort, a.status);
        if (i8_warp_aborts(&s_abort)) return;
        if (t == 0) {
            float *at = red + ((b * PARTS + part) * a.lanes_k + ul) * 16 + g;
            at[0] = yacc[0][0];
            at[8] = yacc[0][1];
        }
        __syncwarp();
        if (lane == 0) {
            mbar_arrive(&s_empty[s]);  // behind the stores of the sums, whose MMAs have waited for all loads from the stage: an arrival may overtake queued loads (zq_gemm.cu)
            mbar_arrive(&s_sums[b]);
        }
        s += a.lanes_g;
        if (s >= S) {
            s -= S;
            ph ^= 1u;
        }
    }
}

// Whether matrices past the SMs' shared memory are streamed here, `all` groups of 16 outputs, n of them on the busiest SM.  Against the work list (a norm in
// front) this form starts 2 us earlier and costs more per group, which shows where rows are short; us, work list / streamed:
//   Q4_K  3840 -> 3 x 3840 12.5/8.5   3840 -> 32768 (n = 14) 19.4/18.4   3840 -> 50000 (n = 22) 23.8/25.9   2560 -> 16384 (n = 7) 11.5/9.0   2560 -> 32768 15.2/15.6   1536 -> 32768 12.0/13.9
//   Q8_0  3840 -> 3 x 3840 14.6/11.3  3840 -> 32768 28.4/24.5  3840 -> 50000 36.5/34.5  2048 -> 50000 23.7/22.8  1536 -> 32768 15.4/15.0  1536 -> 50000 18.5/21.0
//   Q6_K  3840 -> 50000 34.9/33.2  2560 -> 32768 19.8/18.5  2560 -> 50000 25.3/26.3  2048 -> 32768 17.1/18.4;   IQ4_NL  3840 -> 32768 26.1/25.1  5120 -> 32768 32.6/33.4
// Against gemv_i8_kernel (one matrix, one pair) what counts is the busiest SM: its tiles of 128 rows cut along K as far as SMs are idle, in rounds of whole
// slices, against n groups; rows times units there and here:
//   Q4_K  5120 -> 11008 (0.63) 11.5/9.8  3840 -> 28672 (0.76) 18.8/17.0  5120 -> 28672 (0.81) 23.9/19.8  3840 -> 14336 (0.82) 9.8/10.3  3840 -> 17408 (0.94) 10.6/11.6  2048 -> 28672 (0.81) 12.6/14.0
//   Q8_0  3072 -> 28672 (0.81) 22.1/18.3  3072 -> 14336 (0.88) 11.7/11.3  3840 -> 17408 (0.94) 15.1/15.4
//   gated Q4_K  3840 -> 15360 (0.82) 20.3/17.1  3840 -> 17408 (0.94) 21.1/18.4  3072 -> 17408 (1.0) 18.7/18.2  2048 -> 14336 (0.88) 12.8/14.0;   IQ4_NL  3840 -> 15360 27.2/24.0  3840 -> 8192 (0.94) 14.6/14.7
static bool row_stream_pays(const zq_ctx *ctx, const RowCall &c, uint32_t type, size_t units, size_t all) {
    const size_t sms = (size_t)ctx->sm_count, n = (all + sms - 1) / sms;
    if (c.norm) {
        size_t row_bytes = 0;  // of a list's average row, whatever its order
        bool look_ups = false;
        for (int i = 0; i < c.n_jobs; ++i) {
            row_bytes += (c.jobs[i].w->rows + 15) / 16 * units * row_unit_bytes(c.jobs[i].w->type);
            look_ups |= c.jobs[i].w->type == ZQ_IQ4_NL;
        }
        row_bytes /= all;
        const bool eight = type == ZQ_Q8_0;
        if (type == 0 && look_ups && n > 8) return false;  // Q8_0, IQ4_NL, IQ4_NL 3328 -> 3 x 9707 (n = 13) 22.8/24.9, Q6_K, IQ4_NL, Q4_0 4352 -> 13133, 6566, 6566 (n = 12) 27.2/29.1
        if (type == ZQ_IQ4_NL && units > (size_t)kRowWarps && n > 8) return false;
        return n <= 7 || (n <= 14 ? row_bytes >= 2000 || (eight && row_bytes >= 1600) : row_bytes >= 3300 || (eight && row_bytes >= 2100));
    }
    const zq_weight *w = c.jobs[0].w;
    const bool gated = c.jobs[0].w_up != nullptr;
    const size_t per_tile = gated ? kTileRows / 2 : kTileRows, tiles = (w->rows + per_tile - 1) / per_tile, chunks = (units + kChunkUnits - 1) / kChunkUnits;
    const size_t split = std::max<size_t>(1, std::min<size_t>(std::min<size_t>(sms / std::max<size_t>(tiles, 1), 8), chunks));
    const size_t there = (tiles * split + sms - 1) / sms * ((chunks + split - 1) / split) * kTileRows * kChunkUnits, here = n * 16 * (gated ? 2 : 1) * units;
    const auto within = [&](size_t percent) { return 100 * here <= percent * there; };
    if (gated) {
        // Few groups of few bytes do not pay for the ring's start: Q5_K 2304 -> 5553 (n = 3, 0.68) 7.7/8.3, 3328 -> 7514 (n = 4, 0.93) 11.0/12.2; Q4_0 3072 -> 5120 (n = 3, 0.75) 7.3/7.7, 3328 -> 7200
        // (n = 4, 0.93) 8.9/10.2.  Types of more bytes or more instructions do: Q8_0 2816 -> 5352 (n = 3, 0.69) 10.1/8.9, IQ4_NL 2816 -> 6496 10.8/10.1
        const bool few = (n == 3 || n == 4) && (type == ZQ_Q4_K || type == ZQ_Q5_K || type == ZQ_Q4_0);
        if (units < 12 + (few && type == ZQ_Q4_0)) return units >= 8 && !few && within(70);
        return within(type == ZQ_IQ4_NL || (few && type != ZQ_Q4_K) ? 90 : 95);
    }
    return (units >= 12 && within(type == ZQ_Q8_0 ? 90 : 70)) || (units >= 15 && within(81));
}

// Takes a call where its weights fit into the shared memory of the SMs, or else where streaming pays (above).  Two CTAs per SM where registers and shared memory let them: the
// groups spread more evenly, and one copies while the other multiplies; else one CTA, up to 200 KB.  Two against one, us: Q4_K 512 -> 8192 2.9 / 3.2,
// 2560 -> 8192 4.6 / 5.8, gated 1536 -> 3840 3.8 / 4.5, 2560 -> 3840 4.7 / 6.0; where the second does not fit beside the first (3840 -> 3840, 15 warps) 5.8 / 4.1.
template <uint32_t TYPE, bool GATED> static int launch_row_one(zq_ctx *ctx, const RowCall &c, bool &taken, zq_error *err) {
    constexpr size_t PARTS = GATED ? 2 : 1;
    auto kernel = gemv_row_kernel<TYPE, GATED>;
    static size_t warp_regs[64] = {};
    size_t &regs = warp_regs[ctx->device & 63];
    if (!regs) {
        cudaFuncAttributes fa;
        ZQ_CUDA_CHECK(cudaFuncGetAttributes(&fa, kernel), err);
        ZQ_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kRowMaxSmem), err);
        ZQ_CUDA_CHECK(cudaFuncSetAttribute(gemv_row_stream_kernel<TYPE, GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRowMaxSmem), err);
        regs = (size_t)((fa.numRegs + 7) & ~7) * 32;
    }
    // Warps that are resident at once: registers are a quarter of the SM's to each of its four schedulers.  Counted over the whole SM two CTAs of nine warps of 112
    // registers were planned side by side and ran one after the other: three types 2304 -> 3436, 1718, 1718 8.9 us, now 6.4; Q6_K 2304 -> 3001 5.2, now 3.7.
    const size_t slots = 4 * (16384 / regs);
    const size_t units = c.jobs[0].w->units_per_row, turns = (units + kRowWarps - 1) / kRowWarps, lanes_k = (units + turns - 1) / turns;
    if (turns > (size_t)kRowTurns) return ZQ_OK;
    // Gated pairs of many outputs from few columns, and IQ4_NL's of more than 16 units, are as fast or faster where a K slice is a CTA: IQ4_NL 1024 -> 8192 5.8 there,
    // 6.3 here, 8192 -> 512 6.9 / 7.3; Q6_K 512 -> 8192 4.3 / 4.4.
    const int form = ctx->row_form;  // 0: by the rules below; else what fits
    if (form == 0 && GATED && (c.jobs[0].w->rows >= 8 * c.jobs[0].w->cols || (TYPE == ZQ_IQ4_NL && turns > 1))) return ZQ_OK;
    size_t row = 0, all = 0;
    for (int i = 0; i < c.n_jobs; ++i) {
        row = std::max(row, (size_t)row_smem_pitch(c.jobs[i].w->type, (int)units));
        all += (c.jobs[i].w->rows + 15) / 16;
    }
    const bool one_round = (c.jobs[0].w->rows + (GATED ? kTileRows / 2 : kTileRows) - 1) / (GATED ? kTileRows / 2 : kTileRows) <= (size_t)ctx->sm_count;  // of gemv_i8_kernel's tiles
    bool streams = lanes_k >= 4;
    for (int i = 1; i < c.n_jobs; ++i) streams &= is_kclass(c.jobs[i].w->type) == is_kclass(c.jobs[0].w->type);  // a CTA's range may hold several jobs: one format of records
    const auto pays = [&]() { return form == 0 && streams && row_stream_pays(ctx, c, TYPE, units, all); };
    RowArgs ra;
    size_t grid = 0, warps = 0, smem = 0;
    for (size_t per_sm = 2; per_sm >= 1 && !taken && form != 2; --per_sm) {
        const size_t ctas = (size_t)ctx->sm_count * per_sm;
        size_t groups = (all + ctas - 1) / ctas;
        for (; groups <= (size_t)kRowMaxGroups; ++groups) {  // every job starts on a CTA of its own
            grid = 0;
            for (int i = 0; i < c.n_jobs; ++i) grid += ((c.jobs[i].w->rows + 15) / 16 + groups - 1) / groups;
            if (grid <= ctas) break;
        }
        if (groups > (size_t)kRowMaxGroups) continue;
        size_t lanes_g = 1;
        while (2 * lanes_g * lanes_k <= (size_t)kRowWarps && 2 * lanes_g <= groups * PARTS && per_sm * 2 * lanes_g * lanes_k <= slots) lanes_g *= 2;
        warps = lanes_k * lanes_g;
        const size_t w_bytes = 16 * groups * PARTS * row, rec = warps * turns * kRec;
        smem = w_bytes + rec + lanes_k * groups * PARTS * 16 * sizeof(float) + 128;
        if (per_sm * warps > slots || smem > (per_sm == 2 ? (size_t)kRowMaxSmem / 2 - 1024 : (size_t)200 << 10)) continue;
        // IQ4_NL's look-ups want more warps than two CTAs of six hold: 1536 -> 17408 7.5 us on gemv_i8_kernel, 8.6 here; gated 1024 -> 5120 5.3 / 5.9
        if (form == 0 && TYPE == ZQ_IQ4_NL && (GATED && lanes_k <= 4 ? groups > 1 : groups > 2 && per_sm * warps < (size_t)kRowWarps)) break;
        // One or two warps along K have all the look-ups and sums of many groups to themselves.  Norm in front, work list / here: 256 -> 18463 (6.2 groups) 5.4 / 4.4, 58465 (12.3) 6.9 / 9.3; 512 ->
        // 22000 (4.6) 5.6 / 5.5, 27228 (5.8) 6.3 / 6.5, 33709 (7.1) 5.7 / 6.9, 3 x 18058 (11.4) 7.4 / 10.0.  Plain, two units, against one round of tiles: 512 -> 17408 Q4_0 3.5 / 3.9, Q4_K 3.7 / 4.0, Q8_0 4.0 / 4.1
        if (form == 0 && c.norm && groups > (units == 1 ? 7 : 5) && units <= 2) break;
        if (form == 0 && !c.norm && units == 2 && groups >= 4 && one_round) break;
        // more than 150 KB of many groups in one CTA come too late against one round of tiles: Q5_K 2304 -> 15939 8.7 / 10.8, gated Q8_0 1536 -> 6462 6.2 / 6.9, Q4_K 3328 -> 6846 9.1 / 9.8;
        // not of few: Q6_K 3072 -> 8870 (four) 8.7 / 7.7
        if (form == 0 && !c.norm && per_sm == 1 && w_bytes > 150 * 1024 && groups * PARTS >= 5 && turns == 1 && one_round) break;
        // much to copy and a busiest SM with far more of it than its share: Q8_0 1536 -> 14336 6.3 / 7.2, gated 1536 -> 5120 5.8 / 6.1
        if (form == 0 && per_sm == 1 && w_bytes > 150 * 1024 && 100 * groups * ctx->sm_count > 112 * all) continue;
        if (form == 0 && per_sm == 1 && groups >= 5 && pays()) break;
        ra.groups = (int)groups;
        ra.lanes_k = (int)lanes_k;
        ra.lanes_g = (int)lanes_g;
        ra.turns = (int)turns;
        ra.off_rec = (int)w_bytes;
        ra.off_red = (int)(w_bytes + rec);
        taken = true;
    }
    bool stream = false;
    if (!taken && (form == 2 ? streams : pays())) {
        for (size_t lanes_g = 2; lanes_g >= 1 && !taken; --lanes_g) {
            if (lanes_g * lanes_k > (size_t)kRowWarps) continue;
            warps = lanes_g * lanes_k;
            const size_t rec = warps * turns * kRec, sums = kRowSums * PARTS * lanes_k * 16 * sizeof(float), stage = 16 * row;
            size_t stages = std::min<size_t>(kRowMaxGroups, (kRowMaxSmem - 1024 - rec - sums - 128) / stage);
            if (lanes_g == 2) stages &= ~size_t(1);  // a stage is always the same warps', so that their parities tell its phases apart
            if (stages < (GATED ? 4 : 3)) continue;  // a pair takes two of them
            ra.groups = (int)stages;
            ra.lanes_k = (int)lanes_k;
            ra.lanes_g = (int)lanes_g;
            ra.turns = (int)turns;
            ra.stage_bytes = (int)stage;
            ra.off_rec = (int)(stages * stage);
            ra.off_red = (int)(stages * stage + rec);
            smem = stages * stage + rec + sums + 128;
            taken = stream = true;
        }
    }
    if (!taken) return ZQ_OK;
    grid = 0;
    for (int i = 0; i < c.n_jobs; ++i) {
        const zq_weight *w = c.jobs[i].w;
        ra.jobs[i] = {w->data, GATED ? c.jobs[i].w_up->data : nullptr, c.jobs[i].y, c.jobs[i].residual, (int)w->rows, (int)grid, c.jobs[i].y_dtype, w->type};
        grid += stream ? (w->rows + 15) / 16 : ((w->rows + 15) / 16 + ra.groups - 1) / ra.groups;
    }
    if (stream) grid = std::min<size_t>(all, (size_t)ctx->sm_count);
    ra.all_groups = (int)all;
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
    cfg.blockDim = dim3((unsigned)(32 * (warps + (stream ? 2 : 0))));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ctx->disable_pdl ? 0 : 1;
    ZQ_CUDA_CHECK(cudaLaunchKernelEx(&cfg, stream ? gemv_row_stream_kernel<TYPE, GATED> : kernel, ra), err);
    ctx->launches++;
    return ZQ_OK;
}

int launch_gemv_row(zq_ctx *ctx, const RowCall &c, bool &taken, zq_error *err) {
    taken = false;
    if (c.n_jobs < 1 || c.n_jobs > kRowMaxJobs || ctx->row_form < 0) return ZQ_OK;
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
