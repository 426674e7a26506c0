// Decode GEMV over a work list: several independent projections (jobs) in ONE persistent launch.
//
// A decode step is a handful of matrices of 1..50 MB each.  At B200 bandwidth such a matrix streams in 1..8 us, about
// the cost of starting a kernel, filling its TMA ring and draining it again, so a launch per matrix leaves HBM idle
// between matrices.  Here the (job, 128-row tile, 2-unit chunk) items of all jobs form one sequence that is cut into
// equal contiguous ranges, one per SM ("stream-K"): every CTA streams its range through one TMA ring that never
// drains between tiles or matrices, all SMs stay busy whatever the tile counts of the single matrices are, and the
// launch cost is paid once.
//
//   wl_quantize_kernel   activation records (zq_i8.cuh) of every distinct input block of the list, once, into global
//                        memory; each ring stage then brings the records of its two units along with the weights
//   gemv_wl_kernel       integer-MMA decode (arithmetic of zq_gemv_i8.cu) over the CTA's range; in lists of plain jobs of up to 4 rows that
//                        need few records per CTA it makes these itself, in shared memory, an RMSNorm of one row included, and
//                        jobs of several types share the launch
//
// Tiles that a range boundary cuts are finished without any CTA waiting for another: each contributor leaves its
// partial tile in its own slot of the context's scratch and bumps the tile's arrival counter; whoever arrives last
// adds the partials in CTA order (a fixed order: results are deterministic), applies the epilogue and stores.
// A CTA has at most two such tiles (the first and the last of its range).
//
// Reference behaviour covered: ggml_quant::matvec / matvec_residual / gated_silu_matvec
// (src/kernel/cpu/ggml_quant.rs:189-277) for a list of weights, as Backend::dual_linear / triple_linear
// (src/backend/mod.rs:444-451) and the Metal backend's gguf_dual_gemv_q4k_f16 (src/kernel/metal/gguf/mod.rs:1787-1824)
// do for two or three.
#include <algorithm>

#include "zq_i8.cuh"
#include "zq_row.cuh"
#include "zq_wl.cuh"

namespace zq {

constexpr int kWlMaxSegs = 128;  // (tile, chunk range) pieces of one CTA's range kept in shared memory

struct WlJob {
    const CUtensorMap *map_a;  // device copy of the weight's tensor map: 128-row boxes, or (gated) gate, 64-row boxes
    const CUtensorMap *map_b;  // gated: up, 64-row boxes
    const uint8_t *xq;         // records of the job's activation block, [unit][row]
    void *y;                   // [m, n_out]
    const void *residual;      // [m, n_out] or null
    int m;                     // activation rows (1 .. 4 NT)
    int n_out;                 // output features
    int units;                 // 256-column units per weight row
    int chunks;                // ring items per tile = ceil(units / 2)
    int tiles;                 // row tiles
    int q_begin;               // first ring item of the job in the launch's (job, tile, chunk) order
    int y_dtype;               // output (and residual) dtype of this job
    uint16_t src;              // resident records: index into WlResArgs::src
    uint16_t type;             // GGUF type (mixed lists)
};

// Resident records: a distinct input block of the list in one record format.
struct WlSrc {
    const void *x;
    int m, cols;
    bool kclass;
};
// Resident records behind an RMSNorm: the one input row is norm(x).
struct WlNormArgs {
    const float *weight;  // null: no norm
    float eps, weight_offset;
    bool x_wide, w_wide;  // 16-byte aligned row / weights
};

struct WlArgs {
    WlJob jobs[kWlMaxJobs];
    int n_jobs;
    int q_total;       // ring items of the whole launch
    int chunk_words;   // 32-bit words per chunk of a weight row
    int y_dtype;
    int async_fix;     // 5..8 rows: the finisher warp completes cut tiles (otherwise the consumers together)
    float *partials;   // [2 * grid][kSlotFloats]: slot 2c + 1 = the tile CTA c begins, slot 2c = the tile it continues
    uint32_t *counters;  // [grid], zero at the start of the launch: arrivals at the cut tile that CTA c begins
    uint32_t *status;
};
struct WlResArgs : WlArgs {
    int stages, stage_stride, off_rec;  // ring stages, bytes of one, where the records start
    int n_src, x_dtype;
    WlSrc src[kWlMaxJobs];
    WlNormArgs norm;
};
template <bool RES> struct WlArgsOf { using type = WlArgs; };
template <> struct WlArgsOf<true> { using type = WlResArgs; };

struct WlQuantSrc {
    const void *x;
    int m, cols, units;
    int rec_begin;  // first record of the block in the record buffer
};
struct WlQuantArgs {
    WlQuantSrc src[kWlMaxJobs];
    int n_src, total, x_dtype;
    uint8_t *out;
    uint32_t *zero;  // arrival counters to set to zero for the launch behind this one, or null
    int n_zero;
};

// Records of every distinct activation block of the list: one warp per (block, unit, row).
template <uint32_t TYPE>
__global__ void __launch_bounds__(256) wl_quantize_kernel(const __grid_constant__ WlQuantArgs qa) {
    pdl_launch_dependents();
    pdl_wait_prior_grid();  // the record buffer may still be read by the previous launch
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i < qa.n_zero; i += 256) qa.zero[i] = 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rec = blockIdx.x * 8 + warp;
    if (rec >= qa.total) return;  // warp-uniform
    int s = 0;
    while (s + 1 < qa.n_src && qa.src[s + 1].rec_begin <= rec) ++s;
    const WlQuantSrc &q = qa.src[s];
    const int local = rec - q.rec_begin;
    const int unit = local / q.m, row = local - unit * q.m;
    const int k0 = unit * kUnitWeights + 8 * lane;
    float v[8];
    load_act8(q.x, qa.x_dtype, (size_t)row * q.cols + k0, k0 < q.cols, v);
    const RecLane o = quantize_record<TYPE>(v, lane);
    uint8_t *dst = qa.out + (size_t)rec * kRec;
    *reinterpret_cast<uint4 *>(dst + o.slot) = make_uint4(o.ph0, o.ph1, o.pl0, o.pl1);
    if (is_kclass(TYPE) && (lane & 7) == 0) *reinterpret_cast<uint2 *>(dst + kRecSums + (lane >> 3) * 8) = make_uint2(o.sw0, o.sw1);
    if (lane == 0) *reinterpret_cast<float *>(dst + kRecScale) = o.scale;
}

// Shared-memory plan of one instantiation: as many ring stages (up to 5) as fit beside the exchange buffers.
template <uint32_t TYPE, int NT> struct WlSmem {
    static constexpr int UB = Fmt<TYPE>::unit_bytes;
    static constexpr int PITCH = kChunkUnits * UB;
    static constexpr int STAGE_W = kTileRows * PITCH;
    static constexpr int MROWS = 4 * NT;                                  // activation rows a launch class holds
    static constexpr int STRIDE = STAGE_W + kChunkUnits * MROWS * kRec;   // weights, then the chunk's records
    static constexpr int XCH_FLOATS = 16 * 32 * NT * 2;                   // one buffer: [consumer warp][lane][accumulator]
    static constexpr int LIMIT = 232448 - 1024;                           // opt-in maximum minus static shared memory
    static constexpr int MISC = 2 * XCH_FLOATS * 4 + kWlMaxSegs * 16 + 128 + 128;  // exchange (2 buffers), segment list, barriers, slack
    static constexpr int STAGES = (LIMIT - MISC) / STRIDE > 5 ? 5 : (LIMIT - MISC) / STRIDE;
    static constexpr int OFF_XCH = STAGES * STRIDE;
    static constexpr int OFF_SEG = OFF_XCH + 2 * XCH_FLOATS * 4;
    static constexpr int OFF_BAR = OFF_SEG + kWlMaxSegs * 16;
    static constexpr int TOTAL = OFF_BAR + 128 + 128;
    static_assert(STAGES >= 2, "work-list decode kernel: fewer than two ring stages fit");
    static_assert(STRIDE % 128 == 0 && STAGE_W % 256 == 0, "ring stages must keep TMA destinations 128-byte aligned");
};

// Resident records (up to 4 rows, plain jobs): no record pass and no records in the ring.  Every CTA quantises the slices that its own
// range needs, each once, into shared memory, while the first weights are on their way; an RMSNorm in front of the list (one
// row) is computed there too, by every CTA for itself: a row is a few KB out of L2.  That takes a launch (of 4 to 5 us in a chain of
// small ones) and the records' way through memory off a decode step; lists of several types go out as one launch instead of one per
// type (TYPE 0).  Five Q4_K projections of five inputs: 38.7 us, now 37.9.  Norm lists of one row come here where the one-row kernels do not take them
// (zq_gemv_row.cu: past the SMs' shared memory and short rows in many groups, both record formats or fewer than four units; many groups of one or two units).
// The ring gets what the records leave, five stages at most.
template <uint32_t TYPE> struct WlResSmem {
    static constexpr int XCH_FLOATS = 16 * 32 * 2;
    static constexpr int LIMIT = 232448 - 2048;  // opt-in maximum minus static shared memory
    static constexpr int OFF_XCH = (LIMIT - (2 * XCH_FLOATS * 4 + kWlMaxSegs * 16 + 256)) & ~127;
    static constexpr int OFF_SEG = OFF_XCH + 2 * XCH_FLOATS * 4;
    static constexpr int OFF_BAR = OFF_SEG + kWlMaxSegs * 16;
    static constexpr int TOTAL = OFF_BAR + 128 + 128;
};

constexpr int kWlConsumers = kI8Threads;        // 16 consumer warps: 8 row sub-tiles x 2 units
constexpr int kWlThreads = kWlConsumers + 64;   // + the producer warp and the finisher warp
constexpr int kWlNormTurns = 4;                 // a norm inside the kernel holds its row in registers: up to 16 384 columns
// Named barriers (0 is left to __syncthreads, which this kernel never uses: the producer warp runs its own loop).
constexpr int kBarQuad = 1;    // 1..4: the four warps that hold gate and up sums of the same 16 output rows (gated tiles)
constexpr int kBarPair = 5;    // 5..12: the two warps (unit halves) of one row sub-tile
constexpr int kBarFix = 13;    // 13, 14: the 16 consumer warps hand a cut tile's partial sums to the finisher warp (first / second cut piece)
constexpr int kBarAll = 15;    // the 16 consumer warps among themselves (9..16 activation rows: they finish cut tiles on their own; resident records)

__device__ __forceinline__ void named_bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
// Release / acquire fence at GPU scope: orders this thread's (and, after a CTA barrier, its CTA's) earlier accesses before
// its later ones; lighter than the sequentially consistent fence __threadfence() stands for.
__device__ __forceinline__ void fence_acq_rel_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ void named_bar_arrive(int id, int threads) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// CTA that owns ring item q when Q items are cut into G ranges [floor(c Q / G), floor((c + 1) Q / G)).
__device__ __forceinline__ int wl_owner(long long q, long long G, long long Q) { return (int)(((q + 1) * G - 1) / Q); }

// Bounded mbarrier wait that reads the abort flag through its shared address.
__device__ __forceinline__ void wl_wait(uint64_t *bar, uint32_t parity, uint32_t abort_addr, uint32_t *status) {
    for (uint32_t i = 0; i < (1u << 22); ++i) {
        if (mbar_try_wait(bar, parity)) return;
        uint32_t f;
        asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(f) : "r"(abort_addr));
        if (f) return;
    }
    asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(abort_addr), "r"(1u));
    atomicMax(status, (uint32_t)kStatusTmaTimeout);
}

__device__ __forceinline__ int wl_unit_bytes(uint32_t type) { return type == ZQ_Q8_0 ? 272 : type == ZQ_Q6_K ? 224 : type == ZQ_Q5_K ? 176 : 144; }

// One record into shared memory (the warp's lanes hold 8 columns each).
template <bool KCLASS> __device__ __forceinline__ void wl_store_record(uint8_t *dst, const float (&v)[8], int lane) {
    constexpr uint32_t T = KCLASS ? (uint32_t)ZQ_Q4_K : (uint32_t)ZQ_Q4_0;
    const RecLane o = quantize_record<T>(v, lane);
    *reinterpret_cast<uint4 *>(dst + o.slot) = make_uint4(o.ph0, o.ph1, o.pl0, o.pl1);
    if (KCLASS && (lane & 7) == 0) *reinterpret_cast<uint2 *>(dst + kRecSums + (lane >> 3) * 8) = make_uint2(o.sw0, o.sw1);
    if (lane == 0) *reinterpret_cast<float *>(dst + kRecScale) = o.scale;
}

// The units of a source that a CTA needs: a range walks the chunks of a source's jobs from 0 to the end over and over, so it is one run of units
// that may go round from the last chunk to the first.  (Everything between the lowest and the highest unit, which is the whole row wherever a
// range goes on to the next tile: 4 x 17408 -> 5120 in Q4_K, one row, 42.7 us; a list of 2048 -> 300, 17408 -> 512, 1024 -> 9000 and 4096 -> 4096,
// two rows, 17.8 us.  The record pass: 40.8 and 12.5.)
struct WlRun {
    int first, count;  // units; count goes round at `around`
    int rec0;          // index of the first one's first record
    int around;        // units per row, rounded up to whole chunks
};
__device__ __forceinline__ int wl_run_place(const WlRun &r, int unit) { return unit < r.first ? unit - r.first + r.around : unit - r.first; }

// The records of this CTA's range, by the 16 consumer warps.
template <uint32_t TYPE> __device__ __forceinline__ void wl_resident_records(const WlResArgs &a, uint8_t *records, const WlRun *s_run, float *s_partial) {
    constexpr bool MIX = TYPE == 0;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto store = [&](const WlSrc &src, int rec, const float (&v)[8]) {
        uint8_t *dst = records + rec * kRec;
        if (MIX ? src.kclass : is_kclass(MIX ? (uint32_t)ZQ_Q4_K : TYPE)) wl_store_record<true>(dst, v, lane);
        else wl_store_record<false>(dst, v, lane);
    };
    if (a.norm.weight) {
        // the arithmetic of rmsnorm_kernel (zq_norm.cu), thread for thread: thread t holds columns 8 (t + 512 i)
        const WlSrc &s0 = a.src[0];
        float v[kWlNormTurns][8], w[kWlNormTurns][8];
        const int turns = ((s0.cols + 255) / 256 * 32 + kWlConsumers - 1) / kWlConsumers;
        auto load = [&](const void *p, int dtype, bool wide, int c, float (&o)[8]) {
            const bool valid = 8 * c < s0.cols;
            if (wide) {
                load_act8(p, dtype, 8 * (size_t)c, valid, o);
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) o[j] = valid ? load_as_f32(p, dtype, 8 * (size_t)c + j) : 0.f;
            }
        };
        float acc = 0.f;
#pragma unroll
        for (int i = 0; i < kWlNormTurns; ++i) {
            if (i < turns) {
                load(s0.x, a.x_dtype, a.norm.x_wide, tid + i * kWlConsumers, v[i]);
                load(a.norm.weight, ZQ_F32, a.norm.w_wide, tid + i * kWlConsumers, w[i]);
            }
        }
#pragma unroll
        for (int i = 0; i < kWlNormTurns; ++i) {
            if (i < turns) {
#pragma unroll
                for (int j = 0; j < 8; ++j) acc = fmaf(v[i][j], v[i][j], acc);
            }
        }
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, s);
        if (lane == 0) s_partial[warp] = acc;
        named_bar_sync(kBarAll, kWlConsumers);
        float total = s_partial[lane & 15];
#pragma unroll
        for (int s = 8; s > 0; s >>= 1) total += __shfl_xor_sync(0xFFFFFFFFu, total, s);
        const float inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(total, (float)s0.cols), a.norm.eps)));
#pragma unroll
        for (int i = 0; i < kWlNormTurns; ++i) {
            const int unit = warp + 16 * i;
            if (i >= turns) break;
            if (unit * kUnitWeights >= s0.cols) break;  // warp-uniform, as all of this
            bool scaled = false;
            for (int s = 0; s < a.n_src; ++s) {  // the same row in one or both record formats
                const WlRun run = s_run[s];
                const int place = wl_run_place(run, unit);
                if (place >= run.count) continue;
                if (!scaled) {
                    scaled = true;
#pragma unroll
                    for (int j = 0; j < 8; ++j) v[i][j] = 8 * (tid + i * kWlConsumers) < s0.cols ? __fmul_rn(__fmul_rn(v[i][j], inv), a.norm.weight_offset == 0.0f ? w[i][j] : __fadd_rn(a.norm.weight_offset, w[i][j])) : 0.f;
                }
                store(a.src[s], run.rec0 + place, v[i]);
            }
        }
    } else {
        for (int s = 0; s < a.n_src; ++s) {
            const WlSrc &src = a.src[s];
            const WlRun run = s_run[s];
            const int count = run.count * src.m;
            constexpr int kBatch = 4;  // all loads of four records first, so that their latencies overlap
            for (int base = warp; base < count; base += 16 * kBatch) {
                float v[kBatch][8];
#pragma unroll
                for (int b = 0; b < kBatch; ++b) {
                    const int k = base + 16 * b, place = k / src.m, row = k - place * src.m, unit = run.first + place < run.around ? run.first + place : run.first + place - run.around;
                    const int k0 = unit * kUnitWeights + 8 * lane;
                    load_act8(src.x, a.x_dtype, (size_t)row * src.cols + k0, k < count && k0 < src.cols, v[b]);
                }
#pragma unroll
                for (int b = 0; b < kBatch; ++b)
                    if (base + 16 * b < count) store(src, run.rec0 + base + 16 * b, v[b]);  // warp-uniform
            }
        }
    }
    named_bar_sync(kBarAll, kWlConsumers);
}

// Warp-specialised: warp 16 is the producer (it alone waits for free ring stages and issues the TMA copies, so no
// consumer ever stalls on another consumer's progress); warps 0..15 consume.  At the end of a tile only the warps
// that hold sums of the same output rows meet (named barriers of 64 or 128 threads): the two unit halves of a row
// sub-tile, plus the gate / up partners of a gated tile.  The accumulators of partner warps sit in the same lanes, so
// the exchange buffer is indexed by lane and the owning warp stores its 16 rows straight from its fragments.
// RES: resident records.  TYPE 0 (with RES): the jobs' types differ, each brings its own.
template <uint32_t TYPE, int NT, bool GATED, bool RES>
__global__ void __launch_bounds__(kWlThreads, 1) gemv_wl_kernel(const __grid_constant__ typename WlArgsOf<RES>::type a) {
    static_assert(!RES || (NT == 1 && !GATED), "resident records: up to 4 rows, plain jobs");
    constexpr bool MIX = TYPE == 0;
    using S = WlSmem<MIX ? (uint32_t)ZQ_Q4_K : TYPE, NT>;
    using R = WlResSmem<TYPE>;
    int STAGES = S::STAGES, STRIDE = S::STRIDE;
    if constexpr (RES) {
        STAGES = a.stages;
        STRIDE = a.stage_stride;
    }
    constexpr int STAGE_W = S::STAGE_W;  // not in a mixed list
    constexpr int OFF_XCH = RES ? R::OFF_XCH : S::OFF_XCH, OFF_SEG = RES ? R::OFF_SEG : S::OFF_SEG, OFF_BAR = RES ? R::OFF_BAR : S::OFF_BAR;
    constexpr int XCH_FLOATS = S::XCH_FLOATS, NACC = NT * 2;
    auto unit_bytes = [&](const WlJob &jb) -> int { return MIX ? wl_unit_bytes(jb.type) : S::UB; };
    constexpr int out_rows = GATED ? kTileRows / 2 : kTileRows;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    uint8_t *ws = smem;
    float *xch = reinterpret_cast<float *>(smem + OFF_XCH);
    int4 *segs = reinterpret_cast<int4 *>(smem + OFF_SEG);  // {job, tile, first chunk | end chunk << 16, first item (CTA-relative)}
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + OFF_BAR);
    uint64_t *empty = full + 8;
    __shared__ uint32_t s_abort;
    __shared__ int s_nseg, s_last, s_c0, s_cl;
    __shared__ WlRun s_run[RES ? kWlMaxJobs : 1];
    __shared__ float s_partial[16];
    // Up to 4 activation rows a cut tile's partial sums are a few KB and one warp adds them up beside the consumers; with 9..16
    // that warp would need longer than the consumers themselves, so they do it together (and wait for it); with 5..8 rows the host
    // decides by the length of the launch.
    const bool async_fix = NT < 2 || (NT == 2 && a.async_fix);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long G = gridDim.x, Q = a.q_total;
    const int bid = blockIdx.x;
    const int q0 = (int)(bid * Q / G), q1 = (int)((bid + 1) * Q / G);
    const int n_items = q1 - q0;

    // the tensor maps live in global memory: fetch them into the descriptor cache while thread 0 lays out the range
    if (tid >= 32 && tid < 32 + a.n_jobs) {
        tma_prefetch_desc(a.jobs[tid - 32].map_a);
        if (GATED) tma_prefetch_desc(a.jobs[tid - 32].map_b);
    }
    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], kWlConsumers / 32);
        }
        fence_mbar_init();
        s_abort = 0;
        // this CTA's range as (job, tile, chunk range) pieces
        int j = 0;
        while (j + 1 < a.n_jobs && a.jobs[j + 1].q_begin <= q0) ++j;
        const int rel = q0 - a.jobs[j].q_begin;
        int tile = rel / a.jobs[j].chunks, cb = rel - tile * a.jobs[j].chunks;
        int q = q0, n = 0;
        if constexpr (RES)
            for (int i = 0; i < a.n_src; ++i) s_run[i].first = s_run[i].count = 0;
        while (q < q1 && n < kWlMaxSegs && j < a.n_jobs) {
            const int chunks = a.jobs[j].chunks;
            int ce = chunks;
            if (q + (ce - cb) > q1) ce = cb + (q1 - q);
            if constexpr (RES) {  // first and count in chunks here
                WlRun &run = s_run[a.jobs[j].src];
                if (run.count == 0) run.first = cb;
                run.count += ce - cb;
            }
            segs[n++] = make_int4(j, tile, cb | (ce << 16), q - q0);
            q += ce - cb;
            cb = 0;
            if (ce == chunks && ++tile == a.jobs[j].tiles) {
                tile = 0;
                ++j;
            }
        }
        if (q < q1) atomicMax(a.status, (uint32_t)kStatusBadIndex);  // the host sizes launches so that this never happens
        if constexpr (RES) {
            int at = 0;
            for (int i = 0; i < a.n_src; ++i) {
                const int units = (a.src[i].cols + kUnitWeights - 1) / kUnitWeights, chunks = (units + kChunkUnits - 1) / kChunkUnits;
                const bool all = s_run[i].count >= chunks;
                const WlRun run = {all ? 0 : s_run[i].first * kChunkUnits, all ? units : s_run[i].count * kChunkUnits, at, chunks * kChunkUnits};
                s_run[i] = run;
                at += run.count * a.src[i].m;
            }
        }
        // Cut tiles first: a piece of a tile that a range boundary cuts (only the first and the last piece of a range can
        // be one) is finished by whichever contributor arrives last, so every CTA does its cut pieces at the start and
        // the hand-over completes under the streaming of the whole tiles instead of at the very end of the kernel.
        if (n >= 2) {
            const int4 last = segs[n - 1];
            const bool last_cut = !((last.z & 0xFFFF) == 0 && (last.z >> 16) == a.jobs[last.x].chunks);
            const int4 first = segs[0];
            const bool first_cut = !((first.z & 0xFFFF) == 0 && (first.z >> 16) == a.jobs[first.x].chunks);
            if (last_cut) {
                const int pos = first_cut ? 1 : 0;
                for (int k = n - 1; k > pos; --k) segs[k] = segs[k - 1];
                segs[pos] = last;
                int item = 0;
                for (int k = 0; k < n; ++k) {
                    segs[k].w = item;
                    item += (segs[k].z >> 16) - (segs[k].z & 0xFFFF);
                }
            }
        }
        s_nseg = n;
    }
    __syncthreads();  // the only CTA-wide barrier: before the roles part
    const int nseg = s_nseg;
    const int last_item = nseg ? segs[nseg - 1].w + ((segs[nseg - 1].z >> 16) - (segs[nseg - 1].z & 0xFFFF)) : 0;
    const int total_items = last_item < n_items ? last_item : n_items;
    const uint32_t abort_addr = smem_u32(&s_abort);

    if (warp == kWlConsumers / 32 + 1) {
        // ------------------------------------------------------------------------------------------ finisher warp
        // Completes the tiles this CTA shares with its neighbours, off the consumers' path: waits until the consumers
        // have stored a cut piece's partial sums, publishes them (fence + arrival count) and, if this CTA was the last
        // contributor, adds all partials in CTA order and stores the tile.
        pdl_launch_dependents();
        if (!async_fix) return;
        pdl_wait_prior_grid();  // outputs and the fix-up scratch belong to earlier kernels until they complete
        constexpr int G4 = 4 * NT;  // float4 groups per lane: 128 rows x (4 NT) activation rows / 4 / 32 lanes
        for (int k = 0; k < 2 && k < nseg; ++k) {
            const int4 sg = segs[k];
            const WlJob &jb = a.jobs[sg.x];
            const int tile = sg.y, cb = sg.z & 0xFFFF, ce = sg.z >> 16, M = jb.m;
            if (cb == 0 && ce == jb.chunks) break;  // cut pieces come first
            named_bar_sync(kBarFix + k, kWlConsumers + 32);  // the consumers have stored this piece's partial sums
            int last = 0, c0 = 0, cl = 0;
            if (lane == 0) {
                fence_acq_rel_gpu();
                const long long ts = (long long)jb.q_begin + (long long)tile * jb.chunks;
                c0 = wl_owner(ts, G, Q);
                cl = wl_owner(ts + jb.chunks - 1, G, Q);
                last = atomicAdd(&a.counters[c0], 1u) == (uint32_t)(cl - c0);
            }
            last = __shfl_sync(0xffffffffu, last, 0);
            c0 = __shfl_sync(0xffffffffu, c0, 0);
            cl = __shfl_sync(0xffffffffu, cl, 0);
            if (!last) continue;
            fence_acq_rel_gpu();
            // A slot is [activation row][128 tile rows] f32.  Lane L owns tile rows 4L..4L+3 (one float4) of every
            // activation row; up to 8 activation rows are summed at a time so that a contributor costs one round trip.
            constexpr int GB = G4 < 8 ? G4 : 8;
            for (int qb = 0; qb < G4 && qb < M; qb += GB) {
                float4 acc[GB];
#pragma unroll
                for (int i = 0; i < GB; ++i) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                for (int c = c0; c <= cl; ++c) {
                    const float4 *ps = reinterpret_cast<const float4 *>(a.partials + (size_t)(2 * c + (c == c0 ? 1 : 0)) * kSlotFloats);
                    float4 got[GB];
#pragma unroll
                    for (int i = 0; i < GB; ++i) got[i] = qb + i < M ? __ldcg(ps + lane + 32 * (qb + i)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int i = 0; i < GB; ++i) {
                        acc[i].x += got[i].x; acc[i].y += got[i].y; acc[i].z += got[i].z; acc[i].w += got[i].w;
                    }
                }
#pragma unroll
                for (int i = 0; i < GB; ++i) {
                    const int tok = qb + i;
                    if (tok >= M) break;  // warp-uniform
                    const float vv[4] = {acc[i].x, acc[i].y, acc[i].z, acc[i].w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int row = 4 * lane + e;  // row inside the 128-row slot
                        float v = vv[e];
                        if (GATED) {
                            const float up = __shfl_down_sync(0xffffffffu, v, 16);  // lanes 16..31 hold rows 64..127: the up sums
                            if (row >= out_rows) continue;
                            v = (v / (1.0f + expf(-v))) * up;
                        }
                        const int n = tile * out_rows + row;
                        if (n >= jb.n_out) continue;
                        const size_t o = (size_t)tok * jb.n_out + n;
                        if (jb.residual) v += load_as_f32(jb.residual, jb.y_dtype, o);
                        store_from_f32(jb.y, jb.y_dtype, o, v);
                    }
                }
            }
            if (lane == 0) a.counters[c0] = 0;  // ready for the next launch
        }
        return;
    }
    if (warp == kWlConsumers / 32) {
        // ------------------------------------------------------------------------------------------ producer warp
        if (lane == 0) {
            int psi = 0;
            auto locate = [&](int i) {
                while (psi + 1 < nseg && segs[psi + 1].w <= i) ++psi;
            };
            // What stands between a stage's release and its copies is dead time of the stage: an item's addresses are ready before the wait.
            const CUtensorMap *map_a = nullptr, *map_b = nullptr;
            const uint8_t *rec = nullptr;
            int x = 0, y = 0;
            uint32_t w_bytes = 0, rec_bytes = 0;
            auto prepare = [&](int i) {
                locate(i);
                const int4 sg = segs[psi];
                const WlJob &jb = a.jobs[sg.x];
                const int chunk = (sg.z & 0xFFFF) + (i - sg.w);
                map_a = jb.map_a;
                if (GATED) map_b = jb.map_b;
                y = sg.y * out_rows;
                if constexpr (RES) {
                    const int words = kChunkUnits * unit_bytes(jb) / 4;
                    w_bytes = (uint32_t)(kTileRows * words * 4);
                    x = chunk * words;
                } else {
                    int nu = jb.units - chunk * kChunkUnits;
                    if (nu > kChunkUnits) nu = kChunkUnits;
                    w_bytes = STAGE_W;
                    x = chunk * a.chunk_words;
                    rec = jb.xq + (size_t)chunk * kChunkUnits * jb.m * kRec;
                    rec_bytes = (uint32_t)(nu * jb.m * kRec);
                }
            };
            auto issue_w = [&](int stage) {
                uint8_t *dst = ws + (size_t)stage * STRIDE;
                mbar_expect_tx(&full[stage], w_bytes + rec_bytes);
                tma_load_2d(dst, map_a, &full[stage], x, y);
                if (GATED) tma_load_2d(dst + STAGE_W / 2, map_b, &full[stage], x, y);
            };
            auto issue_x = [&](int stage) { bulk_load_1d(ws + (size_t)stage * STRIDE + STAGE_W, rec, rec_bytes, &full[stage]); };
            const int pre = total_items < STAGES ? total_items : STAGES;
            for (int s = 0; s < pre; ++s) {
                prepare(s);
                issue_w(s);  // weights are constants: they may stream while the previous kernel still runs
            }
            pdl_launch_dependents();
            // The records belong to the record pass, which waits for everything before it; and no bounded wait may count while an
            // earlier kernel still runs (one that waits for another rank may take longer than any bound here).
            pdl_wait_prior_grid();
            if constexpr (!RES) {
                psi = 0;
                for (int s = 0; s < pre; ++s) {
                    prepare(s);
                    issue_x(s);
                }
            }
            int stage = 0;
            uint32_t phase = 0;
            for (int i = pre; i < total_items; ++i) {
                prepare(i);
                wl_wait(&empty[stage], phase, abort_addr, a.status);  // every consumer warp is done with the stage's previous item
                uint32_t f;
                asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(f) : "r"(abort_addr));
                if (f) break;  // never start a copy nobody will wait for
                issue_w(stage);
                if constexpr (!RES) issue_x(stage);
                if (++stage == STAGES) {
                    stage = 0;
                    phase ^= 1u;
                }
            }
        } else {
            pdl_launch_dependents();
        }
        return;
    }

    // ---------------------------------------------------------------------------------------------- consumer warps
    pdl_launch_dependents();
    pdl_wait_prior_grid();  // outputs and the fix-up scratch belong to earlier kernels until they complete
    const int g = lane >> 2, t = lane & 3;
    const int rs = warp & 7, ul = warp >> 3;
    const int r0 = 16 * rs + frag_row(g);
    int ub = S::UB;  // unit bytes of the piece's weight
    uint32_t w_first = smem_u32(ws) + (uint32_t)((r0 * kChunkUnits + ul) * S::UB);
    const uint32_t rec_base = smem_u32(ws) + STAGE_W;
    const uint32_t xoff = (uint32_t)(16 * t + 8 * (g & 1));
    if constexpr (RES) wl_resident_records<TYPE>(a, smem + a.off_rec, s_run, s_partial);

    float yacc[NT][2];
    uint32_t moff[NT], soff[NT];
    uint32_t jtype = TYPE;
    int si = -1, seg_end = 0, chunk = 0, units = 0, M = 1, buf = 0, cut_k = 0;
    uint32_t rec_unit = 0;  // byte offset of this warp's unit inside a stage's records
    WlRun run = {};         // resident records: where the piece's units lie
    int stage = 0;
    uint32_t phase = 0;
    for (int it = 0; it < total_items; ++it) {
        if (it == seg_end) {  // a new piece: its job's row count, fresh accumulators
            ++si;
            const int4 sg = segs[si];
            const WlJob &jb = a.jobs[sg.x];
            M = jb.m;
            units = jb.units;
            chunk = sg.z & 0xFFFF;
            seg_end = sg.w + ((sg.z >> 16) - chunk);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                int mb = 4 * nt + (g >> 1), ms = 4 * nt + t;  // B column / accumulator column rows, clamped to an existing row
                if (mb > M - 1) mb = M - 1;
                if (ms > M - 1) ms = M - 1;
                moff[nt] = (uint32_t)(mb * kRec);
                soff[nt] = (uint32_t)(ms * kRec);
                yacc[nt][0] = yacc[nt][1] = 0.f;
            }
            rec_unit = (uint32_t)(ul * M * kRec);
            if constexpr (RES) run = s_run[jb.src];
            if constexpr (MIX) {
                jtype = jb.type;
                ub = unit_bytes(jb);
                w_first = smem_u32(ws) + (uint32_t)((r0 * kChunkUnits + ul) * ub);
            }
        }
        wl_wait(&full[stage], phase, abort_addr, a.status);
        if (chunk * kChunkUnits + ul < units) {
            const uint32_t soffs = (uint32_t)(stage * STRIDE);
            const uint32_t wq0 = w_first + soffs, wq1 = wq0 + (uint32_t)(8 * kChunkUnits * ub);
            uint32_t rb = rec_base + soffs + rec_unit;
            if constexpr (RES) rb = smem_u32(smem) + (uint32_t)(a.off_rec + (run.rec0 + wl_run_place(run, chunk * kChunkUnits + ul) * M) * kRec);
            uint32_t rec[NT], srec[NT];
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                rec[nt] = rb + moff[nt];
                srec[nt] = rb + soff[nt];
            }
            if constexpr (MIX) {
                switch (jtype) {
                case ZQ_Q4_K: consume_q4k_i8<NT, false>(wq0, wq1, t, rec, srec, xoff, yacc); break;
                case ZQ_Q5_K: consume_q4k_i8<NT, true>(wq0, wq1, t, rec, srec, xoff, yacc); break;
                case ZQ_Q6_K: consume_q6k_i8<NT>(wq0, wq1, t, rec, srec, xoff, yacc); break;
                case ZQ_Q4_0: consume_b32_i8<ZQ_Q4_0, NT>(wq0, wq1, t, rec, srec, xoff, yacc); break;
                case ZQ_IQ4_NL: consume_b32_i8<ZQ_IQ4_NL, NT>(wq0, wq1, t, rec, srec, xoff, yacc); break;
                default: consume_b32_i8<ZQ_Q8_0, NT>(wq0, wq1, t, rec, srec, xoff, yacc); break;
                }
            } else if constexpr (TYPE == ZQ_Q6_K) consume_q6k_i8<NT>(wq0, wq1, t, rec, srec, xoff, yacc);
            else if constexpr (is_kclass(TYPE)) consume_q4k_i8<NT, TYPE == ZQ_Q5_K>(wq0, wq1, t, rec, srec, xoff, yacc);
            else consume_b32_i8<TYPE, NT>(wq0, wq1, t, rec, srec, xoff, yacc);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[stage]);
        if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
        }
        ++chunk;
        if (it + 1 == seg_end) {
            // ------------------------------------------------ end of a piece
            const int4 sg = segs[si];
            const WlJob &jb = a.jobs[sg.x];
            const int tile = sg.y, cb = sg.z & 0xFFFF, ce = sg.z >> 16;
            const bool whole = cb == 0 && ce == jb.chunks;  // the whole tile was this CTA's
            float *xb = xch + buf * XCH_FLOATS;
            buf ^= 1;  // a buffer is written again only two pieces later, behind the barrier of the piece in between
            const bool quad = GATED && whole;
            const bool owner = ul == 0 && (!quad || rs < 4);  // the warp that adds up and stores
            if (!owner) {
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    xb[(warp * 32 + lane) * NACC + 2 * nt] = yacc[nt][0];
                    xb[(warp * 32 + lane) * NACC + 2 * nt + 1] = yacc[nt][1];
                }
            }
            if (quad) named_bar_sync(kBarQuad + (rs & 3), 128);
            else named_bar_sync(kBarPair + rs, 64);
            auto finish = [&](int row, int tok, float v, float vup) {
                const int n = tile * out_rows + row;
                if (n >= jb.n_out || tok >= M) return;
                if (GATED) v = (v / (1.0f + expf(-v))) * vup;
                const size_t o = (size_t)tok * jb.n_out + n;
                if (jb.residual) v += load_as_f32(jb.residual, jb.y_dtype, o);
                store_from_f32(jb.y, jb.y_dtype, o, v);
            };
            if (whole) {
                if (owner) {
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {  // fragment rows g and g + 8
                            float v = yacc[nt][h] + xb[((warp + 8) * 32 + lane) * NACC + 2 * nt + h], vup = 0.f;
                            if (GATED) vup = xb[((warp + 4) * 32 + lane) * NACC + 2 * nt + h] + xb[((warp + 12) * 32 + lane) * NACC + 2 * nt + h];
                            finish(r0 + 8 * h, 4 * nt + t, v, vup);
                        }
                    }
                }
            } else {
                // a tile cut by a range boundary: leave the partial sums (all 128 rows) in this CTA's slot, count the arrival
                float *slot = a.partials + (size_t)(2 * bid + (cb == 0 ? 1 : 0)) * kSlotFloats;
                if (owner) {
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt) {
                        const int tok = 4 * nt + t;
                        if (tok < M) {
                            slot[tok * kTileRows + r0] = yacc[nt][0] + xb[((warp + 8) * 32 + lane) * NACC + 2 * nt];
                            slot[tok * kTileRows + r0 + 8] = yacc[nt][1] + xb[((warp + 8) * 32 + lane) * NACC + 2 * nt + 1];
                        }
                    }
                }
                if (async_fix) {
                    named_bar_arrive(kBarFix + cut_k, kWlConsumers + 32);  // over to the finisher warp; this warp goes on
                    ++cut_k;
                } else {
                    __threadfence();
                    named_bar_sync(kBarAll, kWlConsumers);
                    if (tid == 0) {
                        const long long ts = (long long)jb.q_begin + (long long)tile * jb.chunks;
                        const int c0 = wl_owner(ts, G, Q), cl = wl_owner(ts + jb.chunks - 1, G, Q);
                        const uint32_t old = atomicAdd(&a.counters[c0], 1u);
                        s_last = old == (uint32_t)(cl - c0);
                        s_c0 = c0;
                        s_cl = cl;
                    }
                    named_bar_sync(kBarAll, kWlConsumers);
                    if (s_last) {  // every contributor has arrived: add the partials in CTA order
                        __threadfence();
                        const int c0 = s_c0, cl = s_cl;
                        for (int i = tid; i < out_rows * M; i += kWlConsumers) {
                            const int row = i & (out_rows - 1), tok = i / out_rows;
                            float v = 0.f, vup = 0.f;
                            for (int c = c0; c <= cl; ++c) {
                                const float *ps = a.partials + (size_t)(2 * c + (c == c0 ? 1 : 0)) * kSlotFloats + tok * kTileRows;
                                v += __ldcg(ps + row);
                                if (GATED) vup += __ldcg(ps + out_rows + row);
                            }
                            finish(row, tok, v, vup);
                        }
                        if (tid == 0) a.counters[c0] = 0;  // ready for the next launch
                    }
                    named_bar_sync(kBarAll, kWlConsumers);  // s_last may be rewritten by the next cut tile only after everyone read it
                }
            }
        }
    }
}

template <uint32_t TYPE>
static int launch_wl_quantize(zq_ctx *ctx, const WlQuantArgs &qa, zq_error *err) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((qa.total + 7) / 8));
    cfg.blockDim = dim3(256);
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ctx->disable_pdl ? 0 : 1;
    ZQ_CUDA_CHECK(cudaLaunchKernelEx(&cfg, wl_quantize_kernel<TYPE>, qa), err);
    ctx->launches++;
    return ZQ_OK;
}

template <uint32_t TYPE, int NT, bool GATED, bool RES = false>
static int launch_wl_one(zq_ctx *ctx, const typename WlArgsOf<RES>::type &wa, zq_error *err) {
    constexpr int smem = RES ? WlResSmem<TYPE>::TOTAL : WlSmem<TYPE ? TYPE : (uint32_t)ZQ_Q4_K, NT>::TOTAL;
    auto kernel = gemv_wl_kernel<TYPE, NT, GATED, RES>;
    static bool configured[64] = {};
    if (!configured[ctx->device & 63]) {
        ZQ_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem), err);
        configured[ctx->device & 63] = true;
    }
    int grid = ctx->sm_count < wa.q_total ? ctx->sm_count : wa.q_total;  // every CTA gets at least one item
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(kWlThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ctx->disable_pdl ? 0 : 1;
    ZQ_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, wa), err);
    ctx->launches++;
    return ZQ_OK;
}

template <uint32_t TYPE>
static int launch_wl_type(zq_ctx *ctx, const WlArgs &wa, int nt, bool gated, zq_error *err) {
    if (nt == 1) return gated ? launch_wl_one<TYPE, 1, true>(ctx, wa, err) : launch_wl_one<TYPE, 1, false>(ctx, wa, err);
    if (nt == 2) return gated ? launch_wl_one<TYPE, 2, true>(ctx, wa, err) : launch_wl_one<TYPE, 2, false>(ctx, wa, err);
    return gated ? launch_wl_one<TYPE, 4, true>(ctx, wa, err) : launch_wl_one<TYPE, 4, false>(ctx, wa, err);
}

static int launch_wl_resident(zq_ctx *ctx, uint32_t type, const WlResArgs &wa, zq_error *err) {
    switch (type) {
    case 0: return launch_wl_one<0, 1, false, true>(ctx, wa, err);
    case ZQ_Q4_K: return launch_wl_one<ZQ_Q4_K, 1, false, true>(ctx, wa, err);
    case ZQ_Q5_K: return launch_wl_one<ZQ_Q5_K, 1, false, true>(ctx, wa, err);
    case ZQ_Q6_K: return launch_wl_one<ZQ_Q6_K, 1, false, true>(ctx, wa, err);
    case ZQ_Q4_0: return launch_wl_one<ZQ_Q4_0, 1, false, true>(ctx, wa, err);
    case ZQ_IQ4_NL: return launch_wl_one<ZQ_IQ4_NL, 1, false, true>(ctx, wa, err);
    default: return launch_wl_one<ZQ_Q8_0, 1, false, true>(ctx, wa, err);
    }
}

// A list of plain jobs of up to 4 rows in one launch with resident records; `taken` says whether it was.  It is where a CTA's range needs few
// records and they leave enough of a ring, and no result lies over an input (CTAs read inputs while others write results; the record pass reads
// them all first).  A launch less is worth 2.5 to 3 us in a chain of calls, and a record costs some 30 ns of every CTA, in which the
// ring stands still once it is full.  Record pass and resident records, us, calls back to back:
//   records of a CTA   4          24         60         90         120        148
//   Q4_K               14.8/11.9  14.0/12.3  20.6/19.3  21.8/21.1  21.2/22.9  41.3/46.3
//   IQ4_NL             15.0/12.3  14.6/13.0  27.1/25.8  27.6/27.6  27.9/28.8  55.2/56.0
// (8 of 1024 -> 512; 2048 -> 300, 17408 -> 512, 1024 -> 9000 and 4096 -> 4096 of 3 rows; 3840 -> 3840, 3840 -> 15360 and 15360 -> 3840 of 2, 3 and 4 rows; 4 of
// 17408 -> 5120 of 2 rows.)  Less of a ring than the two stages of Q8_0 that the record pass has as well loses by itself: 4 of 17408 -> 5120 in Q5_K, one row,
// three stages of 44 KB 49.0, four 47.9.  A list of one input without a norm keeps the record pass, whose two launches a
// test pins; what resident records would give there is not measured.
constexpr int kWlMostRecords = 96, kWlLeastRing = 136 << 10;
static int launch_gemv_wl_resident(zq_ctx *ctx, const WlHostJob *jobs, size_t n_jobs, int x_dtype, int y_dtype, const WlNorm *norm, bool &taken, zq_error *err) {
    taken = false;
    if (n_jobs > (size_t)kWlMaxJobs || (norm && (jobs[0].m != 1 || jobs[0].w->cols > (size_t)kWlNormTurns * kWlConsumers * 8))) return ZQ_OK;
    if (!norm && std::all_of(jobs, jobs + n_jobs, [&](const WlHostJob &j) { return j.x == jobs[0].x; })) return ZQ_OK;
    WlResArgs wa;
    wa.n_jobs = (int)n_jobs;
    wa.n_src = 0;
    uint32_t type = jobs[0].w->type;
    int unit_bytes = 0, min_chunks = INT32_MAX;
    long long q_total = 0;
    int src_units[kWlMaxJobs];
    for (size_t k = 0; k < n_jobs; ++k) {
        const WlHostJob &j = jobs[k];
        if (j.m > 4 || j.w_up) return ZQ_OK;
        if (j.w->type != type) type = 0;
        unit_bytes = std::max(unit_bytes, format_info(j.w->type).unit_bytes);
        const bool kclass = is_kclass(j.w->type);
        const void *x = norm ? norm->x : j.x;
        int s = 0;
        for (; s < wa.n_src; ++s)
            if (wa.src[s].x == x && wa.src[s].m == (int)j.m && wa.src[s].cols == (int)j.w->cols && wa.src[s].kclass == kclass) break;
        if (s == wa.n_src) {
            src_units[s] = (int)j.w->units_per_row;
            wa.src[wa.n_src++] = {x, (int)j.m, (int)j.w->cols, kclass};
        }
        const long long tiles = (long long)((j.w->rows + kTileRows - 1) / kTileRows), chunks = (long long)((j.w->units_per_row + kChunkUnits - 1) / kChunkUnits);
        if (q_total + tiles * chunks > (long long)INT32_MAX / 512) return ZQ_OK;
        WlJob &d = wa.jobs[k];
        d.map_a = d.map_b = j.w->d_maps;
        d.xq = nullptr;
        d.y = j.y;
        d.residual = j.residual;
        d.m = (int)j.m;
        d.n_out = (int)j.w->rows;
        d.units = (int)j.w->units_per_row;
        d.chunks = (int)chunks;
        d.tiles = (int)tiles;
        d.q_begin = (int)q_total;
        d.y_dtype = j.y_dtype >= 0 ? j.y_dtype : y_dtype;
        d.src = (uint16_t)s;
        d.type = (uint16_t)j.w->type;
        q_total += tiles * chunks;
        min_chunks = std::min(min_chunks, d.chunks);
    }
    const auto apart = [](const void *a, size_t an, const void *b, size_t bn) {
        const uintptr_t a0 = reinterpret_cast<uintptr_t>(a), b0 = reinterpret_cast<uintptr_t>(b);
        return a0 + an <= b0 || b0 + bn <= a0;
    };
    const size_t xe = dtype_size(norm ? norm->x_dtype : x_dtype);
    for (size_t k = 0; k < n_jobs; ++k) {
        const size_t y_bytes = (size_t)wa.jobs[k].m * wa.jobs[k].n_out * dtype_size(wa.jobs[k].y_dtype);
        for (int s = 0; s < wa.n_src; ++s)
            if (!apart(wa.jobs[k].y, y_bytes, wa.src[s].x, (size_t)wa.src[s].m * wa.src[s].cols * xe)) return ZQ_OK;
        if (norm && !apart(wa.jobs[k].y, y_bytes, norm->weight, (size_t)wa.src[0].cols * sizeof(float))) return ZQ_OK;
    }
    if (norm && n_jobs <= (size_t)kRowMaxJobs) {  // one row: the kernels of zq_gemv_row.cu where they fit and pay, norm included
        RowCall c;
        for (size_t k = 0; k < n_jobs; ++k) c.jobs[k] = {jobs[k].w, nullptr, jobs[k].y, jobs[k].residual, wa.jobs[k].y_dtype};
        c.n_jobs = (int)n_jobs;
        c.x = norm->x;
        c.x_dtype = norm->x_dtype;
        c.norm = norm;
        const int rc = launch_gemv_row(ctx, c, taken, err);
        if (rc || taken) return rc;
    }
    wa.q_total = (int)q_total;
    const int grid = ctx->sm_count < wa.q_total ? ctx->sm_count : wa.q_total, per_cta = (wa.q_total + grid - 1) / grid;
    if (per_cta / min_chunks + 3 > kWlMaxSegs) return ZQ_OK;
    // records a range can need: the sources of neighbouring jobs that one range reaches, but no more than two units of each item
    int most = 0;
    for (size_t i = 0; i < n_jobs; ++i) {
        int need = 0, between = 0, rows = 0;
        uint32_t seen = 0;
        for (size_t k = i; k < n_jobs && between < per_cta; ++k) {
            if (!(seen >> wa.jobs[k].src & 1)) need += src_units[wa.jobs[k].src] * wa.jobs[k].m;
            seen |= 1u << wa.jobs[k].src;
            rows = std::max(rows, wa.jobs[k].m);
            if (k > i) between += wa.jobs[k].tiles * wa.jobs[k].chunks;
        }
        most = std::max(most, (int)std::min<long long>(need, (long long)kChunkUnits * per_cta * rows));
    }
    wa.stage_stride = kTileRows * kChunkUnits * unit_bytes;
    const long long left = (long long)WlResSmem<0>::OFF_XCH - (long long)most * kRec;
    wa.stages = left < 0 ? 0 : (int)std::min<long long>(5, left / wa.stage_stride);
    if (most > kWlMostRecords || wa.stages * wa.stage_stride < kWlLeastRing) return ZQ_OK;
    wa.off_rec = wa.stages * wa.stage_stride;
    wa.chunk_words = 0;
    wa.y_dtype = y_dtype;
    wa.x_dtype = norm ? norm->x_dtype : x_dtype;
    wa.async_fix = 1;
    wa.norm = {};
    if (norm) wa.norm = {norm->weight, norm->eps, norm->weight_offset, (reinterpret_cast<uintptr_t>(norm->x) & 15) == 0, (reinterpret_cast<uintptr_t>(norm->weight) & 15) == 0};
    wa.partials = ctx->gemv_partials;
    wa.counters = ctx->gemv_counters;
    wa.status = ctx->status_dev;
    taken = true;
    return launch_wl_resident(ctx, type, wa, err);
}

static bool wl_type_ok(uint32_t t) { return t == ZQ_Q4_K || t == ZQ_Q4_0 || t == ZQ_Q8_0 || t == ZQ_IQ4_NL || t == ZQ_Q5_K || t == ZQ_Q6_K; }

bool gemv_wl_supported(const zq_ctx *ctx, const WlHostJob &j) {
    if (!j.w || !j.w->d_maps || !wl_type_ok(j.w->type) || j.m < 1 || j.m > (size_t)kMaxGemvRows) return false;
    if (j.w_up && (!j.w_up->d_maps || j.w_up->type != j.w->type || j.w_up->rows != j.w->rows || j.w_up->cols != j.w->cols)) return false;
    if ((j.w->units_per_row + kChunkUnits - 1) / kChunkUnits > 0xFFFF) return false;
    if ((size_t)2 * ctx->sm_count * kSlotFloats > ctx->gemv_partials_floats || (size_t)ctx->sm_count > ctx->gemv_counters_n) return false;
    return true;
}

// A gated decode launch of gemv_i8_kernel walks ceil(tiles * slices / SMs) rounds of whole slices; the work-list kernel deals the
// same ring items out evenly, for a record pass, a longer start and the hand-over of cut tiles, ~5 us together.  It is taken when
// the busiest SM would walk at least 216 KB of weights less, those 5 us at ~43 GB/s per SM; with 9..16 rows of Q4_K and Q5_K, where
// arithmetic sets the pace of both kernels and the longer hand-over is not hidden, at least 300 KB.  Measured, gemv_i8 -> work list:
// (one row comes here only where the one-row kernels of zq_gemv_row.cu do not take it)
//   5120 -> 10240 (20 items on the busiest SM against 11)  1 row: Q4_K 21.5 -> 18.7 us, Q5_K 25.4 -> 21.1, IQ4_NL 30.2 -> 23.5, Q8_0 28.1 -> 25.8;
//     8 rows: 26.4 -> 23.4, 29.5 -> 25.7, 35.5 -> 28.2, 33.9 -> 29.6;  16 rows: 36.9 -> 36.2, 40.9 -> 38.8, 45.1 -> 35.2, 42.0 -> 35.6, Q6_K 50.0 -> 40.8
//   3840 -> 10240 (16 against 9)  16 rows: Q4_K 29.8 and 31.0 (258 KB: not taken), Q5_K 33.0 and 33.1, Q4_0 30.0 -> 26.5, IQ4_NL 36.0 -> 29.8, Q8_0 34.2 -> 29.9
//   4096 -> 11008 (16 against 10, the smallest difference that passes in a 4-bit type)  1 row: Q4_K 17.8 -> 16.5, IQ4_NL 25.1 -> 21.0, Q8_0 23.3 -> 22.4;
//     4 rows: 21.1 -> 20.9, 28.1 -> 24.7, 28.6 -> 28.1;  16 rows: Q4_K 31.1 and 34.1, Q5_K 34.3 and 36.6 (not taken), Q4_0 31.1 -> 29.0, IQ4_NL 37.5 -> 33.0
//   3840 -> 15360 (16 against 13, not taken)  1 row: Q4_K 18.8 and 18.9, Q8_0 25.1 and 27.0
bool gated_prefers_worklist(const zq_ctx *ctx, const zq_weight *gate, size_t m) {
    const size_t sms = (size_t)ctx->sm_count, tiles = (gate->rows + kTileRows / 2 - 1) / (kTileRows / 2), chunks = (gate->units_per_row + kChunkUnits - 1) / kChunkUnits;
    size_t split = tiles ? sms / tiles : 1;
    if (split > 8) split = 8;
    if (split > chunks) split = chunks;
    if (split < 1) split = 1;
    const size_t single = (tiles * split + sms - 1) / sms * ((chunks + split - 1) / split), even = (tiles * chunks + sms - 1) / sms;
    return single > even && (single - even) * kTileRows * kChunkUnits * format_info(gate->type).unit_bytes >= (m > 8 && is_kclass(gate->type) ? 300 : 216) * 1024;
}

// Runs the jobs (all of them supported, see gemv_wl_supported) in as few launches as their classes allow: one launch with resident
// records where launch_gemv_wl_resident takes the list, else one record pass per record format, then one decode launch per (weight type,
// column-tile count, plain / gated) class.
// `own_scratch` (one job): records, partial tiles and counters are scratch of the call instead of context memory.  gemv_i8_kernel, the
// other route of a gated pair, uses no context memory up to 4 rows: such a call may be replayed from a graph after any later call
// and run on two streams of a context at once, on either route.
int launch_gemv_wl(zq_ctx *ctx, const WlHostJob *jobs, size_t n_jobs, int x_dtype, int y_dtype, zq_error *err, const WlNorm *norm, bool own_scratch) {
    if (n_jobs == 0) return ZQ_OK;
    if (own_scratch && (n_jobs != 1 || norm)) return set_error(err, ZQ_ERR_ARG, "decode work list: scratch of its own is for one job");
    if (!own_scratch) {
        bool taken = false;
        const int rc = launch_gemv_wl_resident(ctx, jobs, n_jobs, x_dtype, y_dtype, norm, taken, err);
        if (taken || rc) return rc;
    }
    // ---- records: one block per distinct (x, m, cols, record format)
    struct Src { const void *x; size_t m, cols; bool q4k; size_t rec_begin, units; };
    std::vector<Src> srcs;
    std::vector<size_t> src_of(n_jobs);
    size_t total_rec = 0;
    for (size_t i = 0; i < n_jobs; ++i) {
        const WlHostJob &j = jobs[i];
        const bool q4k = is_kclass(j.w->type);
        size_t s = 0;
        for (; s < srcs.size(); ++s)
            if (srcs[s].x == j.x && srcs[s].m == j.m && srcs[s].cols == j.w->cols && srcs[s].q4k == q4k) break;
        if (s == srcs.size()) {
            srcs.push_back({j.x, j.m, j.w->cols, q4k, total_rec, j.w->units_per_row});
            total_rec += j.m * j.w->units_per_row;
        }
        src_of[i] = s;
    }
    if (total_rec > (size_t)INT32_MAX / kRec) return set_error(err, ZQ_ERR_SHAPE, "decode work list: %zu activation records are too many for one call", total_rec);
    LaunchScratch scratch;
    uint8_t *xq = nullptr;
    float *partials = ctx->gemv_partials;
    uint32_t *counters = ctx->gemv_counters;
    int rc;
    if (own_scratch) {
        const size_t head = ((size_t)ctx->sm_count * sizeof(uint32_t) + 1023) & ~size_t(1023), slots = (size_t)2 * ctx->sm_count * kSlotFloats * sizeof(float);
        if ((rc = scratch.take(ctx, head + slots + total_rec * kRec, err))) return rc;
        uint8_t *at = reinterpret_cast<uint8_t *>(scratch.p);
        counters = reinterpret_cast<uint32_t *>(at);
        partials = reinterpret_cast<float *>(at + head);
        xq = at + head + slots;
    } else {
        if ((rc = ensure_xq(ctx, total_rec * kRec, err))) return rc;
        xq = reinterpret_cast<uint8_t *>(ctx->xq);
    }
    if (norm) {  // one input, at most one source per format: the norm kernel writes the records
        uint8_t *rec[2] = {nullptr, nullptr};
        for (const Src &s : srcs) rec[s.q4k ? 0 : 1] = xq + s.rec_begin * kRec;
        if ((rc = launch_rmsnorm_records(ctx, *norm, srcs[0].m, srcs[0].cols, rec[0], rec[1], err))) return rc;
    }
    for (int cls = 0; cls < 2 && !norm; ++cls) {
        WlQuantArgs qa;
        qa.x_dtype = x_dtype;
        qa.n_src = 0;
        qa.zero = own_scratch ? counters : nullptr;
        qa.n_zero = own_scratch ? ctx->sm_count : 0;
        auto flush = [&]() -> int {
            if (qa.n_src == 0) return ZQ_OK;
            // records of one launch are contiguous: the kernel's record index starts at the first block's
            const int first = qa.src[0].rec_begin;
            qa.out = xq + (size_t)first * kRec;
            for (int s = 0; s < qa.n_src; ++s) qa.src[s].rec_begin -= first;
            qa.total = qa.src[qa.n_src - 1].rec_begin + qa.src[qa.n_src - 1].m * qa.src[qa.n_src - 1].units;
            const int r = cls ? launch_wl_quantize<ZQ_Q4_0>(ctx, qa, err) : launch_wl_quantize<ZQ_Q4_K>(ctx, qa, err);
            qa.n_src = 0;
            return r;
        };
        size_t expect = 0;
        for (const Src &s : srcs) {
            if (s.q4k != (cls == 0)) continue;
            if (qa.n_src == kWlMaxJobs || (qa.n_src && s.rec_begin != expect)) {  // full, or a block of the other class lies between
                if ((rc = flush())) return rc;
            }
            qa.src[qa.n_src++] = {s.x, (int)s.m, (int)s.cols, (int)s.units, (int)s.rec_begin};
            expect = s.rec_begin + s.m * s.units;
        }
        if ((rc = flush())) return rc;
    }
    // ---- decode launches, one per class, in order of first appearance
    std::vector<char> done(n_jobs, 0);
    for (size_t i = 0; i < n_jobs; ++i) {
        if (done[i]) continue;
        const uint32_t type = jobs[i].w->type;
        const int nt = jobs[i].m <= 4 ? 1 : (jobs[i].m <= 8 ? 2 : 4);
        const bool gated = jobs[i].w_up != nullptr;
        WlArgs wa;
        wa.n_jobs = 0;
        wa.q_total = 0;
        wa.chunk_words = kChunkUnits * format_info(type).unit_bytes / 4;
        wa.y_dtype = y_dtype;
        wa.partials = partials;
        wa.counters = counters;
        wa.status = ctx->status_dev;
        int min_chunks = INT32_MAX, max_chunks = 0, max_m = 0;
        auto flush = [&]() -> int {
            if (wa.n_jobs == 0) return ZQ_OK;
            // pieces per CTA: at most one per tile boundary inside a range, plus the two ends
            const int grid = ctx->sm_count < wa.q_total ? ctx->sm_count : wa.q_total;
            const long long per_cta = (wa.q_total + grid - 1) / grid;
            if (per_cta / min_chunks + 3 > kWlMaxSegs) return set_error(err, ZQ_ERR_UNSUPPORTED, "decode work list: a CTA would walk more than %d tiles", kWlMaxSegs);
            // The finisher warp needs longer for more rows, and longer for a gated tile; behind it the CTA should have that much left
            // to stream once its cut pieces are done, i.e. its range less a tile.  In ring items, at 5 / 8 rows, consumers together -> finisher warp:
            //   Q4_K 3840 -> 15360 (6 items of 8-item tiles)  17.7 / 17.8 -> 20.2 / 22.9 us, two of them (12)  25.8 / 26.0 -> 25.2 / 26.8
            //   two 5120 -> 17408 (18 of 10)  32.6 / 32.8 -> 29.2 / 31.3; IQ4_NL 41.7 / 41.9 -> 38.5 / 40.2;  q, k, v, o, gate and up of 4096 (16 of 8)  33 / 31.5 -> 28.3 / 29.4
            //   gated 5120 -> 10240 (10 of 10)  23.2 / 23.4 -> 27.6 / 32.4, two 4096 -> 11008 (18 of 8)  33.5 / 34.1 -> 32.0 / 37.4, two 4096 -> 14336 (24 of 8)  40.0 / 40.3 -> 36.0 / 38.7
            wa.async_fix = wa.q_total / grid - max_chunks >= 2 * max_m - (gated ? 0 : 8);
            int r;
            switch (type) {
            case ZQ_Q4_K: r = launch_wl_type<ZQ_Q4_K>(ctx, wa, nt, gated, err); break;
            case ZQ_Q5_K: r = launch_wl_type<ZQ_Q5_K>(ctx, wa, nt, gated, err); break;
            case ZQ_Q6_K: r = launch_wl_type<ZQ_Q6_K>(ctx, wa, nt, gated, err); break;
            case ZQ_Q4_0: r = launch_wl_type<ZQ_Q4_0>(ctx, wa, nt, gated, err); break;
            case ZQ_IQ4_NL: r = launch_wl_type<ZQ_IQ4_NL>(ctx, wa, nt, gated, err); break;
            default: r = launch_wl_type<ZQ_Q8_0>(ctx, wa, nt, gated, err); break;
            }
            wa.n_jobs = 0;
            wa.q_total = 0;
            min_chunks = INT32_MAX;
            max_chunks = max_m = 0;
            return r;
        };
        for (size_t k = i; k < n_jobs; ++k) {
            const WlHostJob &j = jobs[k];
            const int nt_k = j.m <= 4 ? 1 : (j.m <= 8 ? 2 : 4);
            if (done[k] || j.w->type != type || nt_k != nt || (j.w_up != nullptr) != gated) continue;
            done[k] = 1;
            const int rows_per_tile = gated ? kTileRows / 2 : kTileRows;
            const long long tiles = (long long)((j.w->rows + rows_per_tile - 1) / rows_per_tile);
            const long long chunks = (long long)((j.w->units_per_row + kChunkUnits - 1) / kChunkUnits);
            if (wa.n_jobs == kWlMaxJobs || (long long)wa.q_total + tiles * chunks > (long long)INT32_MAX / 512) {
                if ((rc = flush())) return rc;
            }
            WlJob &d = wa.jobs[wa.n_jobs++];
            d.map_a = j.w->d_maps + (gated ? 1 : 0);
            d.map_b = gated ? j.w_up->d_maps + 1 : d.map_a;
            d.xq = xq + srcs[src_of[k]].rec_begin * kRec;
            d.y = j.y;
            d.residual = j.residual;
            d.m = (int)j.m;
            d.n_out = (int)j.w->rows;
            d.units = (int)j.w->units_per_row;
            d.chunks = (int)chunks;
            d.tiles = (int)tiles;
            d.q_begin = wa.q_total;
            d.y_dtype = j.y_dtype >= 0 ? j.y_dtype : y_dtype;
            d.src = 0;
            d.type = (uint16_t)type;
            wa.q_total += (int)(tiles * chunks);
            if ((int)chunks < min_chunks) min_chunks = (int)chunks;
            if ((int)chunks > max_chunks) max_chunks = (int)chunks;
            if (d.m > max_m) max_m = d.m;
        }
        if ((rc = flush())) return rc;
    }
    return ZQ_OK;
}

}  // namespace zq
