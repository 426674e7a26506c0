// Prefill GEMM for GGUF block-quantised weights on the 5th-generation tensor cores (tcgen05 + TMEM), sm_100a.
//
// Replaces the reference's prefill kernels gguf_kq_matmul_f16 / gated_linear_q4_k_silu_rows8_f16 and its
// "dequantise, then cuBLAS" Q4_0 path (src/kernel/cuda/linear.rs:94-138, 880-941, 1141-1166, 1345-1390); the
// arithmetic contract is ggml_quant::matmul / gated_silu_matmul (src/kernel/cpu/ggml_quant.rs:280-362):
// Y[token, row] = sum_k X[token, k] * dequant(W)[row, k], f32 accumulation.
//
// One kernel in two forms of the weight operand A (f16 [rows, K]; every value rounded once to f16, 2^-12 relative, which
// keeps layer outputs inside the 2e-3 bound; bf16 operands would not):
//   SRC = 0     A was dequantised to memory before (launch_dequantize_f16) and arrives by TMA
//   SRC = type  the packed rows arrive by TMA and dequantiser warps write A into the swizzled shared-memory tile or, SHORT, into tensor memory
//               (zq_gemm_dq.cuh): the weight crosses HBM once, packed, and no operand pass runs
// Tiles of up to 128 tokens (SHORT) put that operand into tensor memory instead: two units of 128 columns behind the two accumulators,
// so its way through shared memory (written once, read once, the larger part of that memory's traffic here) is gone and the ring holds
// two units instead of five quarters of one.  What set their pace was the warp that issues the MMAs: 540 cycles per 64-column k-block (a
// successful wait 180, four MMAs and a commit 360, at a fifth of its scheduler's issue slots) where its MMAs take 128 at 64 tokens.  It now
// waits and commits once per unit, sixteen MMAs.  5120 -> 17408 / 17408 -> 5120 at 48 tokens, us: Q4_K 23.5 / 29.4, now 20.3 / 26.2; Q6_K 34.0 / 38.1,
// now 26.7 / 31.2; Q8_0 26.4 / 29.6, now 20.3 / 28.2.  Over 500 random shapes of 17 to
// 128 tokens against the form before, with the cuts that go with each: Q4_K 0.91, Q5_K 0.88, Q6_K 0.87, Q4_0 0.87, IQ4_NL 0.95, Q8_0 0.88.  With 128 to 256 tokens (one accumulator, the epilogue no longer under the next tile)
// plain shapes stay as they are and gated ones take 10 to 20 % longer.
// Activations are f16 (exact for bf16 inputs in f16 range), converted before the kernel where they are not.
//
// The two SMs of a cluster work on one tile of 256 weight rows x up to 256 tokens (cta_group::2, M = 256): each holds half
// of the weight rows, half of the tokens' operand and the accumulator of its own rows (two of 256 TMEM columns, so the
// epilogue of a tile runs under the MMAs of the next).  Why a pair: an MMA of 128 rows x 256 tokens x 16 reads 12 KB of
// shared memory per 128 cycles and its operands take as much again to arrive, more than one SM's 128 B/clk; with the token
// operand split over the pair both figures fall to two thirds.
//
// Tiles are dealt whole to the pairs while there are many; what does not divide is cut along K into equal shares
// (256-column steps), and the SM that finishes a cut tile's last share adds the f32 partials in pair order (deterministic) and
// stores.  A gated tile is 64 gate and 64 up rows per SM (128 outputs per pair), 16 of one and 16 of the other in turn: gate and up of
// an output meet in one warp of the epilogue, and the accumulator still fits twice.
//
// Roles: warp 0 TMA (activations, and A when it is in memory), warp 1 MMA issue (first SM of the pair), warps 2..9 (Q6_K: 2..5 or 2..9)
// epilogue; SRC != 0: then a warp for the TMA of packed boxes and sixteen dequantisers.  Eight epilogue warps and not four, because a tile's epilogue is
// a chain of some 5 (gated: 50) instructions per element in each, which short tiles (few columns of K) do not hide and which the
// last tile of a pair shows in full: Q4_K gated 1536 -> 3840 at 256 tokens 95 us, now 26; 4096 -> 11008 at 256 tokens 75 us, now 47 (with the
// exchange of gate and up inside a warp; before, through shared memory and a barrier per 16 columns).  27 warps leave 72 registers each.  Q6_K,
// whose dequantisers set the pace of most tiles and need more, has four epilogue warps (23 warps, 80 registers) where the epilogue is cheap:
// plain, and gated up to 64 tokens per tile.  Eight and four, us: 11008 -> 4096 at 512 tokens 51.2 and 48.7, 4096 -> 11008 gated at 512 tokens 93.9 and 99.6; SHORT,
// gated at 24 / 64 / 128 tokens 5120 -> 17408 50.3 / 48.4 / 57 and 47.1 / 46.8 / 58, 2048 -> 8192 15.2 / 15.2 / 17.8 and 15.3 / 15.9 / 20.3.  Of the others Q5_K spills four registers there, and every form with wide tiles
// 18 (gated 25), in the epilogue and the way out of cut tiles.
// Every wait is bounded, counted from the end of the previous kernel; a wait that runs out sets the CTA's state, all roles fall
// through to the end, TMEM is released and the context status word reports it.
#include <algorithm>

#include "zq_gemm_dq.cuh"

namespace zq {

constexpr int kBM = 128;      // weight rows per SM (operand tile of one CTA)
constexpr int kPairM = 256;   // weight rows per pair
constexpr int kBN = kGemmTileTokens;      // 256: most tokens per MMA, and per tile of operands in memory
constexpr int kWideBN = kGemmWideTokens;  // 320: most tokens per wide tile (packed types): two MMAs (pieces) of up to 160 share a dequantised operand
constexpr int kChunk = 32, kChunks = 512 / kChunk;  // accumulator columns of wide tiles are given back in chunks of 32
constexpr int kShortBN = 128;  // most tokens per tile with the weight operand in tensor memory
constexpr int kShortA = 256;   // its two units of 128 columns there, behind the two accumulators
constexpr int kShortStages = 4;  // most units of tokens in shared memory (two of more than 64 tokens)
constexpr int kFormPlain = 0, kFormWide = 1, kFormShort = 2;  // FORM of gemm_kernel: what the tiles may be
constexpr int kBK = 64;       // K elements per ring stage (128 bytes of f16: one swizzle atom row)
constexpr int kStepK = 256;   // K elements per step: one packed unit, the grain in which tiles are cut
constexpr int kDqWarps = 16;  // thread = (row, k-block of a unit): four warps per k-block

struct GemmParams {
    void *y;
    const void *residual;
    uint32_t *status;
    int y_dtype;
    int m;       // tokens
    int n_out;   // output features (weight rows; gated: rows of gate)
    int k;       // input columns
    int bn;      // tokens per tile (multiple of 32, at most 256; wide tiles 320)
    int box_tok; // token rows of one activation box (half a tile's)
    int wide;    // tiles may have up to kWideBN tokens; those with more than kBN take two boxes of 80 token rows
    int a_tmem;  // host: the weight operand goes to tensor memory (tiles of at most kShortBN tokens)
    int cut_tiles, cut_pairs;  // the first cut_tiles tiles are cut along K into cut_pairs equal shares
    float *partials;           // [2 * pairs][2 SMs][bn columns][128 rows] f32
    uint32_t *counters;        // arrivals per (pair that begins a cut tile, SM), zero at the start of the launch
    // Grouped form (MoE prefill): the work list replaces the tile grid.  Item = {weight matrix z, first output row of the tile,
    // first token row, end of the tile's token rows}; tokens are rows of one activation operand shared by all matrices,
    // outputs are rows of y with n_out columns.
    const int4 *items;
    int n_items;
    const int *n_items_dev;  // when set, the item count is read from device memory (a plan kernel wrote it); n_items is then its upper bound
    // grouped form of a packed type: per-matrix tensor maps (device table indexed by z)
    const CUtensorMap *w_maps, *w2_maps;
};

// ---- tcgen05 wrappers (pairs of SMs) -------------------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc2(uint32_t *smem_dst, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish2() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc2(uint32_t taddr, uint32_t cols) { asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// arrives on the barrier at this shared offset in both SMs of the pair once the MMAs issued so far are done
__device__ __forceinline__ void tc_commit2(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}
// D[tmem of both SMs] (+)= A[smem of both] * B[smem of both], K-major, f16 inputs, f32 accumulate; issued by the first SM
__device__ __forceinline__ void umma2_f16_ss(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// the same with A in tensor memory: each SM's 128 rows in its own lanes, two K elements per column
__device__ __forceinline__ void umma2_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// Load and wait in one statement: between two the compiler may copy or spill the destination registers, which do not hold the
// values before the wait.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\ttcgen05.wait::ld.sync.aligned;"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
                   "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr)
                 : "memory");
}

// ---- pair plumbing
__device__ __forceinline__ uint32_t pair_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// cluster address of this shared address in the pair's first SM
__device__ __forceinline__ uint32_t pair_first(uint32_t local) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(local));
    return r;
}
__device__ __forceinline__ void pair_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Default (CTA) scope on purpose: what the arrival publishes is read by this SM's own tensor core (operands, behind
// fence.proxy.async) or was ordered by a tcgen05 fence (accumulators).  A release at cluster scope drains all of the thread's
// memory traffic first, which cost more than a k-block's MMAs at every stage.
__device__ __forceinline__ void pair_arrive(uint32_t cluster_bar) { asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory"); }
// Operand row of row r of a gated box (64 gate rows, then 64 up rows): 16 gate rows and the 16 up rows of the same outputs alternate, so
// that they meet in one epilogue warp.
__device__ __forceinline__ int gated_row(int r) { return ((r & 63) >> 4) * 32 + (r >> 6) * 16 + (r & 15); }
// The way back: the box's row behind operand row a.
__device__ __forceinline__ int box_row(int a) { return ((a >> 4) & 1) * 64 + (a >> 5) * 16 + (a & 15); }
// Loads into this SM's shared memory whose completion counts on a barrier of the pair's first SM.  No multicast.
__device__ __forceinline__ void tma_load_2d_pair(void *dst, const CUtensorMap *map, uint32_t cluster_bar, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)),
                 "r"(cluster_bar), "r"(x), "r"(y)
                 : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(void *dst, const CUtensorMap *map, uint32_t cluster_bar, int x, int y, int z) {
    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)),
                 "r"(cluster_bar), "r"(x), "r"(y), "r"(z)
                 : "memory");
}

// K-major operand tile in shared memory, rows of 128 bytes, 128-byte swizzle: 8-row groups are 1024 bytes apart.
__device__ __forceinline__ uint64_t make_sw128_desc(uint32_t smem_addr) {
    uint64_t desc = 0;
    desc |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);   // start address, 16-byte units
    desc |= (uint64_t)1 << 16;                         // leading byte offset: unused for swizzled K-major, 1 by convention
    desc |= (uint64_t)(1024 >> 4) << 32;               // stride byte offset between 8-row groups
    desc |= (uint64_t)1 << 46;                         // descriptor version of this architecture
    desc |= (uint64_t)2 << 61;                         // SWIZZLE_128B
    return desc;
}

// One lane of a converged warp, always the same one.  The single-issuer roles below run their loops with the whole warp and
// only issue under this predicate: loop state and descriptors then stay in uniform registers.  Inside `if (lane == 0)` every
// operand of every tcgen05 or TMA instruction was moved there one by one, about 1000 cycles per k-block for the MMA warp,
// more than its MMAs take.
__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r != 0;
}
// State of a CTA, read by every poll that fails: set up under the previous kernel, whose end it waits for (polls do not count yet);
// running; a bounded wait has run out.  A poll counts only while the previous kernel is over: the warps that run ahead of its
// end would otherwise give up because of it.  (Having them wait for its end themselves cost 3 of 65 us at 48 tokens.)
enum : uint32_t { kStateRun = 0, kStateAbort = 1, kStateAhead = 2 };
// `sleep_ns` > 0: roles that share a scheduler with working warps back off between polls (a bare poll loop re-issues
// every few tens of nanoseconds).
__device__ __forceinline__ bool wait_flag(uint64_t *bar, uint32_t parity, uint32_t state_addr, uint32_t *status, uint32_t code, unsigned sleep_ns = 0) {
    for (uint32_t i = 0; i < (1u << 23);) {
        if (mbar_try_wait(bar, parity)) return true;
        uint32_t state;
        asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(state) : "r"(state_addr));
        if (state == kStateAbort) return false;
        if (state == kStateRun) ++i;
        if (sleep_ns) __nanosleep(sleep_ns);
    }
    asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(state_addr), "r"((uint32_t)kStateAbort));
    atomicMax(status, code);
    return false;
}
// The same where warp-wide instructions follow (elect.sync, tcgen05.ld, .st and tcgen05.wait want the whole warp).  Lanes poll each for itself: one
// may see that the block gives up and another that the phase is complete, and with a way out of the loop between them nothing brings them together.
// Short form: 2 % on gated IQ4_NL, nothing or less on the others.
template <bool VOTE> __device__ __forceinline__ bool wait_warp(uint64_t *bar, uint32_t parity, uint32_t state_addr, uint32_t *status, uint32_t code, unsigned sleep_ns = 0) {
    const bool ok = wait_flag(bar, parity, state_addr, status, code, sleep_ns);
    return VOTE ? __all_sync(0xffffffffu, ok) : ok;
}

template <int DT> struct DtypeTag {
    static constexpr int value = DT;
};
// f32 bits -> one element of the output type, and an element's bits as they are loaded -> f32
template <int DT> __device__ __forceinline__ void store_as(uint8_t *at, uint32_t f32_bits) {
    if constexpr (DT == ZQ_F32) *reinterpret_cast<uint32_t *>(at) = f32_bits;
    else if constexpr (DT == ZQ_F16) *reinterpret_cast<__half *>(at) = __float2half_rn(__uint_as_float(f32_bits));
    else *reinterpret_cast<__nv_bfloat16 *>(at) = __float2bfloat16_rn(__uint_as_float(f32_bits));
}
template <int DT> __device__ __forceinline__ uint32_t load_raw(const uint8_t *at) {
    if constexpr (DT == ZQ_F32) return *reinterpret_cast<const uint32_t *>(at);
    else return *reinterpret_cast<const uint16_t *>(at);
}
template <int DT> __device__ __forceinline__ float raw_as_f32(uint32_t r) {
    if constexpr (DT == ZQ_F32) return __uint_as_float(r);
    else if constexpr (DT == ZQ_F16) return __half2float(__ushort_as_half((unsigned short)r));
    else return __uint_as_float(r << 16);
}

// Shared-memory plan: a ring stage is 16 KB of weights and half a tile's tokens (16 KB, WIDE 20 KB); packed boxes take what the stages leave.
// SHORT: the ring is 64 KB of tokens, units of half a tile's.
template <uint32_t SRC, int FORM, int EPI> struct GemmSmem {  // EPI: epilogue warps
    static constexpr bool WIDE = FORM == kFormWide, SHORT = FORM == kFormShort;
    static constexpr int unit_bytes = SRC == ZQ_Q8_0 ? 272 : SRC == ZQ_Q6_K ? 224 : SRC == ZQ_Q5_K ? 176 : 144;
    static constexpr int a_bytes = SHORT ? 0 : kBM * kBK * 2;
    static constexpr int stage_bytes = SHORT ? 16384 : a_bytes + (WIDE ? kWideBN : kBN) / 2 * kBK * 2;
    static constexpr int p_bytes = SRC ? kBM * unit_bytes : 0;  // one packed box
    static constexpr int pstages = SRC == 0 ? 0 : SHORT ? (unit_bytes <= 144 ? 6 : unit_bytes <= 176 ? 5 : 4) : unit_bytes <= 144 && !WIDE ? 3 : 2;
    static constexpr int stages = SRC == 0 ? 6 : SHORT ? kShortStages : SRC == ZQ_Q8_0 || (SRC == ZQ_Q6_K && WIDE) ? 4 : 5;
    static constexpr int off_p = stages * stage_bytes;
    static constexpr int off_bar = off_p + pstages * p_bytes;
    static constexpr int bar_bytes = 256 + (WIDE ? 2 * kChunks * 8 : 0);
    static constexpr int total = off_bar + bar_bytes + 1024;    // barriers, slack for 1024-byte alignment
    static constexpr int threads = (2 + EPI + (SRC ? 1 + kDqWarps : 0)) * 32;
    static_assert(total <= 232448 - 64, "prefill GEMM: shared memory");
    static_assert(off_p % 1024 == 0 && off_bar % 8 == 0, "prefill GEMM: alignment");
};

// SHORT: units of tokens in the ring, from the bytes of a k-block of one
template <class S> __device__ __forceinline__ int short_stages(uint32_t sub) {
    const int fit = (int)((uint32_t)S::off_p / (4 * sub));
    return fit < S::stages ? fit : S::stages;
}

constexpr int kTokGroup = 8;  // token tiles per raster group: a weight tile is reused by 8 token tiles while it is hot in L2

// A piece of work of one pair: K steps [k0, k1) of a tile.
struct GemmSeg {
    int row0, tok0, tok_end, z, k0, k1, tile;
};
// Walks a pair's share: first its part of the cut tiles, then its whole tiles.
struct GemmWalk {
    int q, q1, tile, stride, total, steps, row_tiles, tok_tiles, rows_per_tile;
    __device__ __forceinline__ GemmWalk(const GemmParams &p, int pair, int pairs, int rows_per_tile_) {
        rows_per_tile = rows_per_tile_;
        steps = (p.k + kStepK - 1) / kStepK;
        row_tiles = (p.n_out + rows_per_tile - 1) / rows_per_tile;
        tok_tiles = (p.m + p.bn - 1) / p.bn;
        total = p.items ? (p.n_items_dev ? *p.n_items_dev : p.n_items) : row_tiles * tok_tiles;
        stride = pairs;
        const long long cut = (long long)p.cut_tiles * steps;
        q = q1 = 0;
        if (pair < p.cut_pairs) {
            q = (int)(pair * cut / p.cut_pairs);
            q1 = (int)((pair + 1) * cut / p.cut_pairs);
        }
        tile = p.cut_tiles + pair;
    }
    __device__ __forceinline__ bool next(const GemmParams &p, GemmSeg &s) {
        if (q < q1) {
            s.tile = q / steps;
            s.k0 = q - s.tile * steps;
            s.k1 = s.k0 + (q1 - q) < steps ? s.k0 + (q1 - q) : steps;
            q += s.k1 - s.k0;
        } else if (tile < total) {
            s.tile = tile;
            s.k0 = 0;
            s.k1 = steps;
            tile += stride;
        } else {
            return false;
        }
        if (p.items) {
            const int4 it = p.items[s.tile];
            s.z = it.x;
            s.row0 = it.y;
            s.tok0 = it.z;
            const int most = p.wide ? kWideBN : kBN;
            s.tok_end = it.w < it.z + most ? it.w : it.z + most;
            return true;
        }
        s.z = 0;
        const int per_group = kTokGroup * row_tiles;
        const int group = s.tile / per_group, in_group = s.tile - group * per_group;
        const int group_toks = (tok_tiles - group * kTokGroup) < kTokGroup ? (tok_tiles - group * kTokGroup) : kTokGroup;
        s.row0 = (in_group / group_toks) * rows_per_tile;
        s.tok0 = (group * kTokGroup + in_group % group_toks) * p.bn;
        s.tok_end = s.tok0 + p.bn < p.m ? s.tok0 + p.bn : p.m;
        return true;
    }
};
// Accumulator columns of a tile, in chunks: its tokens rounded up to 32 (16 per SM).
__device__ __forceinline__ int tile_chunks(const GemmSeg &s) {
    const int n = (s.tok_end - s.tok0 + kChunk - 1) / kChunk;
    return n < 1 ? 1 : n;
}
// Tiles take the low and the high end of the 512 accumulator columns in turn.  Two that do not fit beside each other (both wide)
// overlap in the middle, where the epilogue begins: it gives a tile's chunks back from the middle outwards, and the MMAs of
// the next tile start as soon as those they share with it are free.
__device__ __forceinline__ int tile_column(int iter, int chunks) { return (iter & 1) ? (kChunks - chunks) * kChunk : 0; }
// Chunks of the first of a tile's two pieces (of its only one).
__device__ __forceinline__ int first_piece(int chunks) { return chunks > kBN / kChunk ? (chunks + 1) / 2 : chunks; }

// A cut tile whose shares have all arrived.
struct GemmCut {
    int row0, tok0, n_tok, c_first, c_last;
};

// Adds the shares of an SM's half of a cut tile in pair order and stores it: all warps together, once their roles are over.  Reading
// the shares is a matter of bytes in flight (several times 128 KB per SM at some 1000 cycles of latency): a thread takes four rows of
// several tokens at a time.  The four epilogue warps alone, 16 columns of one share at a time, took most of the launch where
// every tile is cut: 17408 -> 5120 in Q4_K, 48 / 256 / 512 tokens 40 / 88 / 89 us, now 32 / 47 / 75.
template <bool GATED, int THREADS> __device__ __forceinline__ void add_up_cut(const GemmParams &p, const GemmCut &t, uint32_t rank) {
    constexpr int OUT = GATED ? kBM / 2 : kBM, QUADS = OUT / 4, PARTS = GATED ? 2 : 1, LANES = THREADS / QUADS;  // LANES: columns that the CTA takes side by side
    constexpr int COLS = 4 / PARTS;
    const int quad = (int)threadIdx.x % QUADS, lane_col = (int)threadIdx.x / QUADS, row = t.row0 + (int)rank * OUT + 4 * quad;
    const int at0 = GATED ? gated_row(4 * quad) : 4 * quad;  // operand row; gated: of gate, up lies 16 rows on
    const int rows = p.n_out - row < 4 ? p.n_out - row : 4, esz = (int)dtype_size(p.y_dtype);
    if (rows <= 0 || lane_col >= LANES) return;
    for (int c0 = lane_col; c0 < t.n_tok; c0 += LANES * COLS) {
        float4 sum[PARTS][COLS];
        for (int c = t.c_first; c <= t.c_last; ++c) {
            const float *share = p.partials + ((size_t)(2 * c + (c == t.c_first ? 1 : 0)) * 2 + rank) * ((size_t)p.bn * kBM) + at0;
            float4 v[PARTS][COLS];
#pragma unroll
            for (int part = 0; part < PARTS; ++part)
#pragma unroll
                for (int k = 0; k < COLS; ++k) {
                    const int col = c0 + k * LANES;
                    v[part][k] = col < t.n_tok ? __ldcg(reinterpret_cast<const float4 *>(share + col * kBM + part * 16)) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
            for (int part = 0; part < PARTS; ++part)
#pragma unroll
                for (int k = 0; k < COLS; ++k) {
                    const float4 n = v[part][k];
                    float4 &s = sum[part][k];
                    s = c == t.c_first ? n : make_float4(s.x + n.x, s.y + n.y, s.z + n.z, s.w + n.w);
                }
        }
#pragma unroll
        for (int k = 0; k < COLS; ++k) {
            const int col = c0 + k * LANES;
            if (col >= t.n_tok) break;
            const size_t at = (size_t)(t.tok0 + col) * p.n_out + row;
            float o[4] = {sum[0][k].x, sum[0][k].y, sum[0][k].z, sum[0][k].w};
            if (GATED) {
                const float u[4] = {sum[PARTS - 1][k].x, sum[PARTS - 1][k].y, sum[PARTS - 1][k].z, sum[PARTS - 1][k].w};
#pragma unroll
                for (int j = 0; j < 4; ++j) o[j] = (o[j] / (1.0f + expf(-o[j]))) * u[j];
            }
            if (p.residual) {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (j < rows) o[j] += load_as_f32(p.residual, p.y_dtype, at + j);
            }
            if ((p.n_out & 3) == 0) {  // four whole rows, and y (16-byte aligned) is aligned to them
                uint8_t *const yb = reinterpret_cast<uint8_t *>(p.y) + at * esz;
                if (p.y_dtype == ZQ_F32) {
                    *reinterpret_cast<float4 *>(yb) = make_float4(o[0], o[1], o[2], o[3]);
                } else if (p.y_dtype == ZQ_F16) {
                    *reinterpret_cast<uint2 *>(yb) = make_uint2(h2_as_u32(__floats2half2_rn(o[0], o[1])), h2_as_u32(__floats2half2_rn(o[2], o[3])));
                } else {
                    const __nv_bfloat162 lo = __floats2bfloat162_rn(o[0], o[1]), hi = __floats2bfloat162_rn(o[2], o[3]);
                    *reinterpret_cast<uint2 *>(yb) = make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
                }
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (j < rows) store_from_f32(p.y, p.y_dtype, at + j, o[j]);
            }
        }
    }
}

// WIDE: tiles of up to 320 tokens.  What they are for: a tile of a packed type costs its dequantisation whatever its tokens, and an expert that
// got 257 to 320 tokens was two tiles (256 experts of 7168 x 2048 in Q4_K, 8192 tokens, 256 +- 16 to an expert: MoE layer 8.2 ms, now 7.1).
// A form of its own because the second piece costs the issuing warp instructions in every k-block: with one form for both, 48
// tokens of 5120 x 17408 up and down took 61.2 us instead of 56.7 (before SHORT, which takes 46.5).
template <uint32_t SRC, bool GATED, int FORM, int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GemmSmem<SRC, FORM, EPI>::threads, 1)
    gemm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_w2, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_x2, const GemmParams p) {
    using S = GemmSmem<SRC, FORM, EPI>;
    constexpr bool WIDE = S::WIDE, SHORT = S::SHORT;
    constexpr int STAGES = S::stages, PST = S::pstages > 0 ? S::pstages : 1;
    constexpr int kRows = GATED ? kPairM / 2 : kPairM;  // output rows of a tile
    constexpr int kPackedWarp = 2 + EPI;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + S::off_bar);  // first SM: a stage's operands, both SMs' bytes and dequantiser warps
    uint64_t *empty = full + STAGES;                                   // each SM: the stage's MMAs are done
    uint64_t *p_full = empty + STAGES;                                 // each SM: packed boxes
    uint64_t *p_empty = p_full + PST;
    uint64_t *acc_full = p_empty + PST;                                // each SM
    uint64_t *acc_empty = acc_full + 2;                                // first SM: both SMs' epilogue warps
    uint64_t *a_full = acc_empty + 2, *a_empty = a_full + 2;           // SHORT: a unit of weights in tensor memory: first SM, both SMs' dequantiser warps; each SM, its MMAs are done
    uint64_t *step_free = acc_empty + 2;                               // WIDE, first SM: both SMs' epilogue warps are through with the k-th chunk of a tile; once per tile each
    __shared__ uint32_t s_tmem;
    __shared__ uint32_t s_state;
    __shared__ GemmCut s_cut[2];  // cut tiles that this SM adds up: a pair's shares touch two at most
    __shared__ int s_cuts;

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;  // the shuffle tells the compiler that it is uniform
    const uint32_t rank = pair_rank();
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    // Packed rows end on whole units (zero blocks): their padding is multiplied like the rest, against columns the TMA unit fills
    // with zeros, so that every dequantiser warp has its turn in every unit.  A warp that skipped turns could meet a stage
    // barrier two phases behind, which its parity cannot tell from one phase ahead.
    const int k_blocks = SRC ? 4 * ((p.k + kStepK - 1) / kStepK) : (p.k + kBK - 1) / kBK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], SRC && !SHORT ? 9 : 1);  // the TMA issuer, and four dequantiser warps of each SM
            mbar_init(&empty[s], 1);
        }
        for (int s = 0; s < PST; ++s) {
            mbar_init(&p_full[s], 1);
            mbar_init(&p_empty[s], kDqWarps);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 2 * EPI);
        }
        for (int b = 0; SHORT && b < 2; ++b) {
            mbar_init(&a_full[b], 2 * kDqWarps);
            mbar_init(&a_empty[b], 1);
        }
        for (int c = 0; WIDE && c < 2 * kChunks; ++c) mbar_init(&step_free[c], 2 * EPI);
        fence_mbar_init();
        s_state = kStateAhead;
        s_cuts = 0;
        tma_prefetch_desc(&map_w);
        tma_prefetch_desc(&map_x);
        if (GATED) tma_prefetch_desc(&map_w2);
    }
    pdl_launch_dependents();  // what follows may be set up under this kernel; it waits for its end before it touches memory
    if (warp == 1) {
        tmem_alloc2(&s_tmem, 512);
        tmem_relinquish2();
    }
    tc_fence_before();
    __syncthreads();
    pair_sync();  // both SMs' barriers and tensor memory exist
    tc_fence_after();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t *>(&s_tmem);
    const uint32_t state_addr = smem_u32(&s_state);
    // Programmatic dependent launch: everything up to here, and for packed dense weights (constants) also their first boxes and
    // their dequantisation, runs under the previous kernel's end; activations, f16 operands, work lists, results and partials
    // belong to earlier kernels until they complete.  5120 x 17408 up and down in Q4_K: 48 tokens 76 -> 65 us, 512 tokens 192 -> 188 us.
    // The warps that run ahead (packed boxes, dequantisers) wait for stages that only the MMAs set free, but these waits count from the end of the
    // previous kernel (kStateAhead), which may itself wait for another rank for longer than any bound here.
    if (SRC == 0 || p.items || warp < kPackedWarp) pdl_wait_prior_grid();
    if (threadIdx.x == 0) *reinterpret_cast<volatile uint32_t *>(&s_state) = kStateRun;  // nobody gives up before this
    __syncwarp();
    GemmWalk walk(p, pair, pairs, kRows);
    GemmSeg sg;

    if (warp == 0) {
        // ------------------------------------------------ TMA: tokens (half a tile each), and the f16 weight operand
        int s = 0;
        uint32_t ph = 0;
        bool ok = true, fresh = true;  // fresh: first turn of the ring
        while (ok && walk.next(p, sg)) {
            const int columns = tile_chunks(sg) * kChunk, first = first_piece(columns / kChunk) * kChunk;
            const bool two = WIDE && columns > first;
            const int tok = sg.tok0 + (int)rank * (first / 2), tok2 = sg.tok0 + first + (int)rank * ((columns - first) / 2);
            const uint32_t bytes = 2u * (uint32_t)((SRC ? 0 : S::a_bytes) + (two ? kWideBN / 2 : p.box_tok) * kBK * 2);
            const int row = sg.row0 + (int)rank * (GATED ? 64 : kBM);
            const int kb1 = sg.k1 * 4 < k_blocks ? sg.k1 * 4 : k_blocks;
            if constexpr (SHORT) {  // a stage is a unit: four k-blocks side by side
                const uint32_t sub = (uint32_t)p.box_tok * kBK * 2;
                const int stages = short_stages<S>(sub);
                for (int u = sg.k0; u < sg.k1; ++u) {
                    if (!fresh && !wait_warp<true>(&empty[s], ph ^ 1u, state_addr, p.status, kStatusMmaTimeout)) {
                        ok = false;
                        break;
                    }
                    if (elect_one()) {
                        uint8_t *st = smem + (size_t)s * 4 * sub;
                        const uint32_t bar = pair_first(smem_u32(&full[s]));
                        if (rank == 0) mbar_expect_tx(&full[s], 8 * sub);
#pragma unroll
                        for (int i = 0; i < 4; ++i) tma_load_2d_pair(st + i * sub, &map_x, bar, u * kStepK + i * kBK, tok);
                    }
                    __syncwarp();
                    if (++s == stages) {
                        s = 0;
                        ph ^= 1u;
                        fresh = false;
                    }
                }
                continue;
            }
            for (int kb = sg.k0 * 4; kb < kb1; ++kb) {
                if (!fresh && !wait_flag(&empty[s], ph ^ 1u, state_addr, p.status, kStatusMmaTimeout)) {
                    ok = false;
                    break;
                }
                if (elect_one()) {
                    uint8_t *st = smem + (size_t)s * S::stage_bytes;
                    const uint32_t bar = pair_first(smem_u32(&full[s]));
                    if (rank == 0) mbar_expect_tx(&full[s], bytes);
                    if constexpr (SRC == 0) {
                        const int at = GATED ? 2 * row : row;  // gated: 16 rows of gate, 16 of up, and so on in memory already
                        if (p.items) tma_load_3d_pair(st, &map_w, bar, kb * kBK, at, sg.z);
                        else tma_load_2d_pair(st, &map_w, bar, kb * kBK, at);
                    }
                    tma_load_2d_pair(st + S::a_bytes, two ? &map_x2 : &map_x, bar, kb * kBK, tok);
                    if (two) tma_load_2d_pair(st + S::a_bytes + kWideBN / 4 * kBK * 2, &map_x2, bar, kb * kBK, tok2);
                }
                __syncwarp();
                if (++s == STAGES) {
                    s = 0;
                    ph ^= 1u;
                    fresh = false;
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------ MMA issue
        if (rank == 0) {
            int s = 0, iter = 0;
            uint32_t ph = 0;
            bool ok = true;
            const uint64_t desc0 = make_sw128_desc(smem_u32(smem));
            uint32_t ah = 0, aph = 0;  // SHORT: which unit of weights in tensor memory, and its phase
            int before = 0;  // chunks of the tile before
            for (; ok && walk.next(p, sg); ++iter) {
                // f32 accumulator, f16 A and B, both K-major, M = 256, N = the piece's tokens
                const int chunks = tile_chunks(sg), first = first_piece(chunks), second = chunks - first, shared = before + chunks - kChunks;
                before = chunks;
                const uint32_t idesc0 = (1u << 4) | ((uint32_t)(kPairM >> 4) << 24), idesc = idesc0 | ((uint32_t)(first * (kChunk >> 3)) << 17), idesc2 = idesc0 | ((uint32_t)(second * (kChunk >> 3)) << 17);
                const int b = iter & 1;
                // WIDE: every chunk of the tile before last is waited for, a lane each, and then the one shared with the last tile.  A barrier of one of
                // the two sets is thus never more than one phase ahead of or behind the one asked for, whatever the order in which arrivals at
                // different barriers are seen.
                if (iter >= 2) {
                    if constexpr (WIDE) ok = __all_sync(0xffffffffu, wait_flag(&step_free[b * kChunks + (lane & (kChunks - 1))], (uint32_t)((iter >> 1) - 1) & 1, state_addr, p.status, kStatusMmaTimeout));
                    else ok = wait_warp<SHORT>(&acc_empty[b], (uint32_t)((iter >> 1) - 1) & 1, state_addr, p.status, kStatusMmaTimeout);
                }
                if (WIDE && ok && shared > 0) ok = wait_flag(&step_free[(b ^ 1) * kChunks + shared - 1], (uint32_t)((iter - 1) >> 1) & 1, state_addr, p.status, kStatusMmaTimeout);
                if (!ok) break;
                tc_fence_after();
                const uint32_t acc = tmem_base + (uint32_t)(WIDE ? tile_column(iter, chunks) : b * (SHORT ? kShortBN : kBN)), acc2 = acc + (uint32_t)(first * kChunk);
                const int kb0 = sg.k0 * 4, kb1 = sg.k1 * 4 < k_blocks ? sg.k1 * 4 : k_blocks;
                if constexpr (SHORT) {
                    const uint32_t sub = (uint32_t)p.box_tok * kBK * 2;  // as the TMA warp has them
                    const int stages = short_stages<S>(sub);
                    for (int u = sg.k0; u < sg.k1; ++u) {
                        ok = __all_sync(0xffffffffu, wait_flag(&full[s], ph, state_addr, p.status, kStatusTmaTimeout) && wait_flag(&a_full[ah], aph, state_addr, p.status, kStatusTmaTimeout));
                        if (!ok) break;
                        tc_fence_after();
                        if (elect_one()) {
                            uint64_t db = desc0 + (uint32_t)s * (4 * sub / 16);
                            const uint32_t a = tmem_base + (uint32_t)(kShortA + ah * (kStepK / 2));
#pragma unroll
                            for (int i = 0; i < kStepK / 16; ++i) {
                                umma2_f16_ts(acc, a + 8 * i, db + 2 * (i & 3), idesc, (i > 0 || u > sg.k0) ? 1u : 0u);
                                if ((i & 3) == 3) db += sub / 16;
                            }
                            tc_commit2(&a_empty[ah]);
                            tc_commit2(&empty[s]);
                            if (u + 1 == sg.k1) tc_commit2(&acc_full[b]);
                        }
                        __syncwarp();
                        if (++s == stages) {
                            s = 0;
                            ph ^= 1u;
                        }
                        aph ^= ah;
                        ah ^= 1u;
                    }
                    continue;
                }
                for (int kb = kb0; kb < kb1; ++kb) {
                    ok = wait_flag(&full[s], ph, state_addr, p.status, kStatusTmaTimeout);
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const uint64_t da = desc0 + (uint32_t)(s * (S::stage_bytes / 16)), db = da + S::a_bytes / 16;
#pragma unroll
                        for (int k = 0; k < kBK / 16; ++k)  // 16 K elements = 32 bytes = 2 descriptor units along the swizzled row
                            umma2_f16_ss(acc, da + 2 * k, db + 2 * k, idesc, (kb > kb0 || k > 0) ? 1u : 0u);
                        if (WIDE && second) {
                            const uint64_t db2 = db + kWideBN / 4 * kBK * 2 / 16;
#pragma unroll
                            for (int k = 0; k < kBK / 16; ++k) umma2_f16_ss(acc2, da + 2 * k, db2 + 2 * k, idesc2, (kb > kb0 || k > 0) ? 1u : 0u);
                        }
                        tc_commit2(&empty[s]);
                        if (kb + 1 == kb1) tc_commit2(&acc_full[b]);
                    }
                    __syncwarp();
                    if (++s == STAGES) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
            }
        }
    } else if (warp < kPackedWarp) {
        // ------------------------------------------------ epilogue: a warp owns TMEM lanes 32 q .. 32 q + 31 = those operand rows of the SM, and
        // every second group of 16 columns
        const int q = warp & 3, part = (warp - 2) >> 2;
        int iter = 0;
        const int et = (warp - 2) * 32 + lane;
        for (; walk.next(p, sg); ++iter) {
            const int b = iter & 1;
            const int n_tok = sg.tok_end - sg.tok0, chunks = tile_chunks(sg);
            if (!GATED && p.residual) {
                // bring the tile's residual rows into L2 while its MMAs run: a warp can only have a few KB of loads in flight below
                const size_t esz = dtype_size(p.y_dtype), r0 = (size_t)sg.row0 + rank * kBM;
                const size_t bytes = (size_t)p.n_out * esz;
                for (int i = et; i < n_tok * (int)esz; i += 32 * EPI) {  // 128 rows = esz lines of 128 bytes per token
                    const size_t at = r0 * esz + (size_t)(i % (int)esz) * 128;
                    if (at < bytes) asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const uint8_t *>(p.residual) + (size_t)(sg.tok0 + i / (int)esz) * bytes + at));
                }
            }
            const bool ok = wait_warp<SHORT>(&acc_full[b], (uint32_t)(iter >> 1) & 1, state_addr, p.status, kStatusMmaTimeout, SRC ? 200 : 0);
            tc_fence_after();
            const uint32_t acc = tmem_base + (uint32_t)(WIDE ? tile_column(iter, chunks) : b * (SHORT ? kShortBN : kBN)) + ((uint32_t)(q * 32) << 16);
            auto free_step = [&](int k) {  // this warp is through with the k-th chunk
                tc_fence_before();
                __syncwarp();
                if (lane == 0) pair_arrive(pair_first(smem_u32(&step_free[b * kChunks + k])));
            };
            const bool whole = sg.k0 == 0 && sg.k1 == walk.steps;
            // output row of this lane; gated: lanes 0..15 hold gate rows, lanes 16..31 the up rows of the same outputs
            const int row = GATED ? sg.row0 + (int)rank * 64 + q * 16 + (lane & 15) : sg.row0 + (int)rank * kBM + q * 32 + lane;
            // 16 columns of finished sums (f32 bits) -> y.  With the output type known at compile time and one wide multiply-add per address
            // an element takes about 4 instructions.
            auto store16 = [&](auto dt, int c0, uint32_t (&v)[16]) {
                constexpr int DT = decltype(dt)::value;
                const size_t at = ((size_t)(sg.tok0 + c0) * p.n_out + row) * dtype_size(DT);
                uint8_t *const yb = reinterpret_cast<uint8_t *>(p.y) + at;
                auto token = [&](int j) { return (uint64_t)(uint32_t)p.n_out * (uint32_t)(j * (int)dtype_size(DT)); };  // bytes from one token's row to the j-th after it
                if (GATED) {
                    // the two lanes of an output trade: the gate lane finishes columns 0..7 of the group, the up lane 8..15
                    const bool is_up = lane >= 16;
                    float g[8], u[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const uint32_t mine = is_up ? v[8 + j] : v[j], other = __shfl_xor_sync(0xffffffffu, is_up ? v[j] : v[8 + j], 16);
                        g[j] = __uint_as_float(is_up ? other : mine);
                        u[j] = __uint_as_float(is_up ? mine : other);
                    }
                    if (row >= p.n_out) return;
                    const int cb = is_up ? 8 : 0, left = n_tok - c0 - cb;
                    uint8_t *const yc = yb + token(cb);
#pragma unroll
                    for (int j = 0; j < 8; ++j) v[j] = __float_as_uint((g[j] / (1.0f + expf(-g[j]))) * u[j]);  // src/kernel/cpu/ggml_quant.rs:352
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (j < left) store_as<DT>(yc + token(j), v[j]);
                    return;
                }
                if (row >= p.n_out) return;
                const int left = n_tok - c0;
                if (p.residual) {  // all loads of the chunk, unconverted, before anything uses one (and before the first store: y may be the residual's own buffer)
                    const uint8_t *const rb = reinterpret_cast<const uint8_t *>(p.residual) + at;
                    uint32_t r[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) r[j] = j < left ? load_raw<DT>(rb + token(j)) : 0u;
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + raw_as_f32<DT>(r[j]));
                }
                if (left >= 16) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) store_as<DT>(yb + token(j), v[j]);
                } else {
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (j < left) store_as<DT>(yb + token(j), v[j]);
                }
            };
            auto store_tile = [&](auto dt) {
                if constexpr (WIDE) {
                    for (int k = 0; k < chunks; ++k) {  // warp-uniform; from the middle of the columns outwards
                        const int c0 = ((iter & 1) ? k : chunks - 1 - k) * kChunk + 16 * part;
                        uint32_t v[16];
                        if (c0 < n_tok) tmem_ld16(acc + c0, v);
                        free_step(k);
                        if (c0 < n_tok) store16(dt, c0, v);
                    }
                } else {
                    for (int c0 = 16 * part; c0 < n_tok; c0 += 4 * EPI) {  // walked as above, 48 tokens of 5120 x 17408 up and down take 63.8 us instead of 57.7
                        uint32_t v[16];
                        tmem_ld16(acc + c0, v);
                        store16(dt, c0, v);
                    }
                }
            };
            if (ok && whole) {
                if (p.y_dtype == ZQ_F32) store_tile(DtypeTag<ZQ_F32>());
                else if (p.y_dtype == ZQ_F16) store_tile(DtypeTag<ZQ_F16>());
                else store_tile(DtypeTag<ZQ_BF16>());
            }
            if (!whole) {
                // A share of a cut tile goes to its slot; the SM that comes last takes the tile down for the end of the kernel.
                const long long Q = (long long)p.cut_tiles * walk.steps, G = p.cut_pairs, ts = (long long)sg.tile * walk.steps;
                const int c_first = (int)(((ts + 1) * G - 1) / Q), c_last = (int)(((ts + walk.steps) * G - 1) / Q);  // pairs that own the tile's first and last step
                float *slot = p.partials + ((size_t)(2 * pair + (sg.k0 == 0 ? 1 : 0)) * 2 + rank) * ((size_t)p.bn * kBM) + q * 32 + lane;
                if (ok) {
                    for (int c0 = 16 * part; c0 < n_tok; c0 += 4 * EPI) {
                        uint32_t v[16];
                        tmem_ld16(acc + c0, v);
#pragma unroll
                        for (int j = 0; j < 16; ++j) __stcg(slot + (size_t)(c0 + j) * kBM, __uint_as_float(v[j]));
                    }
                }
                __threadfence();
                asm volatile("bar.sync 3, %0;" ::"n"(32 * EPI) : "memory");
                if (et == 0 && ok && atomicAdd(p.counters + 2 * c_first + rank, 1u) == (uint32_t)(c_last - c_first)) s_cut[s_cuts++] = {sg.row0, sg.tok0, n_tok, c_first, c_last};
            }
            if (WIDE)
                for (int k = whole && ok ? chunks : 0; k < kChunks; ++k) free_step(k);
            tc_fence_before();
            __syncwarp();
            if (!WIDE && lane == 0) pair_arrive(pair_first(smem_u32(&acc_empty[b])));  // this warp's part of the accumulator may be overwritten
        }
    } else if constexpr (SRC != 0) {
        if (warp == kPackedWarp) {
            // ------------------------------------------------ TMA: packed boxes (one unit of every row) on a ring of their own
            int ps = 0;
            uint32_t pph = 0;
            bool ok = true, fresh = true;
            while (ok && walk.next(p, sg)) {
                const CUtensorMap *mw = p.items ? &p.w_maps[sg.z] : &map_w;
                const CUtensorMap *mw2 = p.items ? (GATED ? &p.w2_maps[sg.z] : mw) : &map_w2;
                const int row = sg.row0 + (int)rank * (GATED ? 64 : kBM);
                for (int u = sg.k0; u < sg.k1; ++u) {
                    if (!fresh && !wait_warp<SHORT>(&p_empty[ps], pph ^ 1u, state_addr, p.status, kStatusMmaTimeout, 50)) {
                        ok = false;
                        break;
                    }
                    if (elect_one()) {
                        uint8_t *pst = smem + S::off_p + (size_t)ps * S::p_bytes;
                        mbar_expect_tx(&p_full[ps], S::p_bytes);
                        tma_load_2d(pst, mw, &p_full[ps], u * (S::unit_bytes / 4), row);
                        if (GATED) tma_load_2d(pst + S::p_bytes / 2, mw2, &p_full[ps], u * (S::unit_bytes / 4), row);
                    }
                    __syncwarp();
                    if (++ps == PST) {
                        ps = 0;
                        pph ^= 1u;
                        fresh = false;
                    }
                }
            }
        } else {
            // ------------------------------------------------ dequantisers: thread = (row, k-block of the unit)
            const int t = threadIdx.x - (kPackedWarp + 1) * 32, mine = t >> 7;  // mine: k-block of the unit, warp-uniform
            if constexpr (SHORT) {
                // Operand in tensor memory: a warp reaches the 32 lanes of its own quarter (warp number modulo four) only.
                const int a_row = (warp & 3) * 32 + lane, row = GATED ? box_row(a_row) : a_row;
                const uint32_t box0 = smem_u32(smem) + (uint32_t)(S::off_p + row * S::unit_bytes);
                const uint32_t a0 = tmem_base + (uint32_t)(kShortA + mine * (kBK / 2)) + ((uint32_t)((warp & 3) * 32) << 16);
                const uint32_t full0 = pair_first(smem_u32(&a_full[0]));
                int ps = 0;
                uint32_t pph = 0, ah = 0, aph = 0;
                bool ok = true;
                DqBlock<SRC> dq;
                // tcgen05.st and its wait want every lane, so none leaves the loops: one whose wait has failed waits for nothing any more and walks on.  Costs
                // nothing; a vote and a way out 1.5 % at 48 tokens of Q4_K, a __syncwarp here 4 % at 128.
                while (walk.next(p, sg)) {
                    for (int u = sg.k0; u < sg.k1; ++u) {
                        ok = ok && wait_flag(&p_full[ps], pph, state_addr, p.status, kStatusTmaTimeout, 20);
                        dq.load(box0 + (uint32_t)(ps * S::p_bytes), mine);
                        ok = ok && wait_flag(&a_empty[ah], aph ^ 1u, state_addr, p.status, kStatusMmaTimeout, 20);
                        tc_fence_after();  // behind the MMAs that read this half before
                        dq.emit(DqTensorRow{a0 + ah * (kStepK / 2)});
                        tmem_st_wait();
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) {
                            pair_arrive(full0 + ah * (uint32_t)sizeof(uint64_t));
                            mbar_arrive(&p_empty[ps]);  // all that was read of the box has been stored by now
                        }
                        aph ^= ah;
                        ah ^= 1u;
                        if (++ps == PST) {
                            ps = 0;
                            pph ^= 1u;
                        }
                    }
                }
            } else {
                const int row = t & (kBM - 1);  // row of the box
                const int a_row = GATED ? gated_row(row) : row, sw = a_row & 7;
                const uint32_t row0 = smem_u32(smem) + (uint32_t)((a_row >> 3) * 1024 + sw * 128), box0 = smem_u32(smem) + (uint32_t)(S::off_p + row * S::unit_bytes);
                int s = 0, ps = 0;  // ring positions: s walks the k-blocks of all warps, this warp serves one in four
                uint32_t ph = 0, pph = 0;
                bool ok = true, fresh = true;
                DqBlock<SRC> dq;
                auto advance = [&](int n) {
                    s += n;
                    if (s >= STAGES) {
                        s -= STAGES;
                        ph ^= 1u;
                        fresh = false;
                    }
                };
                while (ok && walk.next(p, sg)) {
                    for (int u = sg.k0; u < sg.k1; ++u) {
                        ok = wait_flag(&p_full[ps], pph, state_addr, p.status, kStatusTmaTimeout, 20);
                        if (!ok) break;
                        dq.load(box0 + (uint32_t)(ps * S::p_bytes), mine);
                        // Everything the warp needs of the box is in registers once this vote has read them.  Without it the arrival
                        // overtakes shared-memory loads still queued behind other warps' stores, and the next box lands under them.
                        if (__any_sync(0xffffffffu, dq.mix() == 0x9E3779B9u)) __nanosleep(0);  // a no-op that keeps the vote
                        if (lane == 0) mbar_arrive(&p_empty[ps]);
                        if (++ps == PST) {
                            ps = 0;
                            pph ^= 1u;
                        }
                        advance(mine);
                        if (!fresh) ok = wait_flag(&empty[s], ph ^ 1u, state_addr, p.status, kStatusMmaTimeout, 20);
                        if (!ok) break;
                        dq.emit(DqSharedRow{row0 + (uint32_t)(s * S::stage_bytes), sw});
                        fence_proxy_async();  // generic-proxy stores -> visible to the tensor cores of the pair
                        __syncwarp();
                        if (lane == 0) pair_arrive(pair_first(smem_u32(&full[s])));
                        advance(4 - mine);
                    }
                }
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    pair_sync();  // nobody leaves while the other SM may still signal here or read operands
    if (warp == 1) tmem_dealloc2(tmem_base, 512);
    if (s_cuts) __threadfence();  // behind the arrivals that this SM has seen
    for (int i = 0; i < s_cuts; ++i) add_up_cut<GATED, S::threads>(p, s_cut[i], rank);
}

// activations of any supported dtype -> f16; eight values per thread and step (one 16- or 32-byte load, one 16-byte store);
// `zero`: arrival counters of the GEMM behind it
__global__ void __launch_bounds__(256) to_f16_kernel(const void *__restrict__ x, int x_dtype, __half *__restrict__ out, size_t n8, uint32_t *__restrict__ zero, int n_zero) {
    pdl_launch_dependents();
    pdl_wait_prior_grid();
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i < n_zero; i += 256) zero[i] = 0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += (size_t)gridDim.x * blockDim.x) {
        uint32_t h[4];
        if (x_dtype == ZQ_F32) {
            const float4 a = __ldcs(reinterpret_cast<const float4 *>(x) + 2 * i), b = __ldcs(reinterpret_cast<const float4 *>(x) + 2 * i + 1);
            h[0] = h2_as_u32(__floats2half2_rn(a.x, a.y)); h[1] = h2_as_u32(__floats2half2_rn(a.z, a.w));
            h[2] = h2_as_u32(__floats2half2_rn(b.x, b.y)); h[3] = h2_as_u32(__floats2half2_rn(b.z, b.w));
        } else {
            const uint4 r = __ldcs(reinterpret_cast<const uint4 *>(x) + i);
            const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) h[j] = x_dtype == ZQ_F16 ? w[j] : h2_as_u32(__floats2half2_rn(__uint_as_float(w[j] << 16), __uint_as_float(w[j] & 0xFFFF0000u)));
        }
        reinterpret_cast<uint4 *>(out)[i] = make_uint4(h[0], h[1], h[2], h[3]);
    }
}

static int make_f16_map(const void *base, size_t rows, size_t cols, int box_rows, CUtensorMap *out, zq_error *err) {
    EncodeTiledFn encode = get_encode_tiled(err);
    if (!encode) return ZQ_ERR_CUDA;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
    cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = encode(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return set_error(err, ZQ_ERR_CUDA, "cuTensorMapEncodeTiled (f16 operand %zux%zu) failed with code %d", rows, cols, (int)r);
    return ZQ_OK;
}

static int make_f16_map3(const void *base, size_t mats, size_t rows, size_t cols, int box_rows, CUtensorMap *out, zq_error *err) {
    EncodeTiledFn encode = get_encode_tiled(err);
    if (!encode) return ZQ_ERR_CUDA;
    cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)mats};
    cuuint64_t strides[2] = {(cuuint64_t)cols * 2, (cuuint64_t)rows * cols * 2};
    cuuint32_t box[3] = {(cuuint32_t)kBK, (cuuint32_t)box_rows, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = encode(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return set_error(err, ZQ_ERR_CUDA, "cuTensorMapEncodeTiled (f16 operand %zux%zux%zu) failed with code %d", mats, rows, cols, (int)r);
    return ZQ_OK;
}

// n = 0: only the counters
int launch_to_f16(zq_ctx *ctx, const void *x, int x_dtype, __half *out, size_t n, zq_error *err, uint32_t *zero, int n_zero) {
    const size_t n8 = n / 8;  // rows are multiples of 8 columns wherever this runs
    size_t blocks = (n8 + 255) / 256;
    if (blocks > (size_t)ctx->sm_count * 16) blocks = (size_t)ctx->sm_count * 16;
    if (blocks == 0) blocks = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(256);
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ctx->disable_pdl ? 0 : 1;
    ZQ_CUDA_CHECK(cudaLaunchKernelEx(&cfg, to_f16_kernel, x, x_dtype, out, n8, zero, n_zero), err);
    ctx->launches++;
    return ZQ_OK;
}

template <uint32_t SRC, bool GATED, int FORM, int EPI>
static int launch_one(zq_ctx *ctx, const CUtensorMap &mw, const CUtensorMap &mw2, const CUtensorMap &mx, const CUtensorMap &mx2, const GemmParams &p, int pairs, zq_error *err) {
    using S = GemmSmem<SRC, FORM, EPI>;
    static bool configured[64] = {};
    if (!configured[ctx->device & 63]) {
        ZQ_CUDA_CHECK(cudaFuncSetAttribute(gemm_kernel<SRC, GATED, FORM, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::total), err);
        configured[ctx->device & 63] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(2 * pairs));
    cfg.blockDim = dim3(S::threads);
    cfg.dynamicSmemBytes = S::total;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ctx->disable_pdl ? 0 : 1;
    ZQ_CUDA_CHECK(cudaLaunchKernelEx(&cfg, gemm_kernel<SRC, GATED, FORM, EPI>, mw, mw2, mx, mx2, p), err);
    ctx->launches++;
    return ZQ_OK;
}
template <uint32_t SRC> static int launch_form(zq_ctx *ctx, bool gated, const CUtensorMap &mw, const CUtensorMap &mw2, const CUtensorMap &mx, const CUtensorMap &mx2, const GemmParams &p, int pairs, zq_error *err) {
    constexpr int W = SRC ? kFormWide : kFormPlain, H = SRC ? kFormShort : kFormPlain;  // operands in memory have no other form
    constexpr int Q6 = SRC == ZQ_Q6_K ? 4 : 8;  // see the roles
    if (W && p.wide) return gated ? launch_one<SRC, true, W, 8>(ctx, mw, mw2, mx, mx2, p, pairs, err) : launch_one<SRC, false, W, 8>(ctx, mw, mw2, mx, mx2, p, pairs, err);
    if (H && p.a_tmem) {
        if (gated && (Q6 == 8 || p.bn > 64)) return launch_one<SRC, true, H, 8>(ctx, mw, mw2, mx, mx2, p, pairs, err);
        return gated ? launch_one<SRC, true, H, Q6>(ctx, mw, mw2, mx, mx2, p, pairs, err) : launch_one<SRC, false, H, Q6>(ctx, mw, mw2, mx, mx2, p, pairs, err);
    }
    return gated ? launch_one<SRC, true, kFormPlain, 8>(ctx, mw, mw2, mx, mx2, p, pairs, err) : launch_one<SRC, false, kFormPlain, Q6>(ctx, mw, mw2, mx, mx2, p, pairs, err);
}
static int launch_src(zq_ctx *ctx, uint32_t src, bool gated, const CUtensorMap &mw, const CUtensorMap &mw2, const CUtensorMap &mx, const CUtensorMap &mx2, const GemmParams &p, int pairs, zq_error *err) {
#define ZQ_GEMM_CASE(T) case T: return launch_form<T>(ctx, gated, mw, mw2, mx, mx2, p, pairs, err)
    switch (src) {
        ZQ_GEMM_CASE(0);
        ZQ_GEMM_CASE(ZQ_Q4_K);
        ZQ_GEMM_CASE(ZQ_Q5_K);
        ZQ_GEMM_CASE(ZQ_Q6_K);
        ZQ_GEMM_CASE(ZQ_Q4_0);
        ZQ_GEMM_CASE(ZQ_IQ4_NL);
        ZQ_GEMM_CASE(ZQ_Q8_0);
    default: return set_error(err, ZQ_ERR_UNSUPPORTED, "prefill GEMM: no kernel for GGUF type %u", src);
    }
#undef ZQ_GEMM_CASE
}

static void clear_params(zq_ctx *ctx, GemmParams &p) {
    memset(&p, 0, sizeof(p));
    p.status = ctx->status_dev;
}

// Token tiles of a dense GEMM: as few as tiles of `cap` tokens allow, of equal size (300 tokens in tiles of up to 256 are two of
// 160, not 256 + 44).
static void plan_tokens(size_t m, size_t cap, GemmParams &p) {
    const size_t tiles = (m + cap - 1) / cap;
    p.m = (int)m;
    p.bn = (int)(((m + tiles - 1) / tiles + 31) & ~size_t(31));
    p.wide = p.bn > kBN;
    p.box_tok = p.wide ? kBN / 2 : p.bn / 2;
}
// Boxes of half a tile's tokens, and (wide tiles) of half a piece's.
static int make_token_maps(const __half *x, size_t rows, size_t k, const GemmParams &p, CUtensorMap *map_x, CUtensorMap *map_x2, zq_error *err) {
    int rc = make_f16_map(x, rows, k, p.box_tok, map_x, err);
    if (!rc && p.wide) rc = make_f16_map(x, rows, k, kWideBN / 4, map_x2, err);
    if (!p.wide) *map_x2 = *map_x;
    return rc;
}

// How many tiles are cut along K.  Whole tiles over P pairs take ceil(T / P) rounds; cut, the tiles beyond the full rounds and one
// round more (all of them when there are fewer than two rounds) take equal shares of at least two steps, at most eight of a tile.
// Cutting saves the steps that the busiest pair is ahead of the average one, at 0.85 us (a dequantised step of up to 152 tokens; of a SHORT
// tile 0.5 us for Q4_K, Q4_0 and Q8_0, gated 0.7, and 0.9 for the others) or 5.6 ns per token each.  It costs the shares' way out and in and their addition, 3 us and 50 ns per token of the tile (gated: 30, where the addition
// takes the place of an epilogue), and 8 ns per token for every round more, in which pairs no longer meet at the same depth of K.  From
// operands in memory that costs most: 160 ns per token, and past L2 140 where the cut part is little more than a round, 400 where it is more and
// nothing is shared for long.  Without the rounds' share the rule cut 343 of 960 shapes (64 to 8192 tokens, 2048 to 17408 columns, three types,
// plain and gated) and was 0.3 % behind the better choice for plain ones on average and 1.7 % for gated ones, up to 12 %; with it 0.2 and
// 0.3 %.  800 shapes of 17 to 128 tokens, six types: 0.3 % behind, 14 of them more than 5 % (the worst 23); with one step time for all 43.  Whole and cut, us:
//   Q4_K 15360 -> 3840, 64 tokens 47 / 22;  11008 -> 4096, 64 tokens 35 / 20;  Q6_K 15360 -> 3840, 300 tokens 91 / 52;  2560 -> 1434 gated, 115 tokens 18.2 / 16.1
//   not: Q8_0 3328 -> 7537, 32 tokens 10.8 / 14.3;  Q4_0 2816 -> 7104, 30 tokens 9.9 / 14.3
//   not: Q4_K gated 4096 -> 11008, 512 tokens 74 / 83;  3840 -> 15360, 3001 tokens 553 / 587;  5120 -> 17408, 800 tokens 241 / 263
//   operands in memory past L2: 15360 -> 3840, 2500 tokens 383 / 305, 3600 tokens 460 / 390;  not 2048 tokens 252 / 339, 3001 tokens 372 / 429
static int plan_cut(const zq_ctx *ctx, int tiles, int steps, uint32_t src, bool gated, size_t operand_bytes, GemmParams &p) {
    const bool fused = src != 0;
    const int pairs = ctx->sm_count / 2 > 0 ? ctx->sm_count / 2 : 1;
    const int rounds = (tiles + pairs - 1) / pairs, whole = tiles < pairs ? tiles : pairs;
    p.cut_tiles = p.cut_pairs = 0;
    if (ctx->cut_tiles < 0 || steps < 2 || tiles % pairs == 0) return whole;
    const int full = tiles / pairs, cut = full >= 2 ? tiles - (full - 1) * pairs : tiles;
    long long shares = (long long)cut * steps / 2;
    if (shares > 8LL * cut) shares = 8LL * cut;
    const int cut_pairs = shares < pairs && cut == tiles ? (int)shares : pairs;
    const long long saved = (long long)(rounds - (tiles - cut) / pairs) * steps - ((long long)cut * steps + cut_pairs - 1) / cut_pairs;
    const bool light = p.a_tmem && (src == ZQ_Q4_K || src == ZQ_Q4_0 || src == ZQ_Q8_0);
    const long long step_ns = std::max(!fused || (light && !gated) ? 500LL : light ? 700LL : p.a_tmem ? 900LL : 850LL, 56LL * p.bn / 10);
    const long long token_ns = fused ? (gated ? 30 : 50) + 8 * (rounds - 1) : operand_bytes <= (size_t(128) << 20) ? 160 : 3 * cut <= 4 * pairs ? 140 : 400;
    const long long cost_ns = 3000 + token_ns * p.bn;
    if (!ctx->cut_tiles && saved * step_ns <= cost_ns) return whole;
    p.cut_tiles = cut;
    p.cut_pairs = cut_pairs;
    return cut_pairs;
}
// Shares and their counters are scratch of the launch and not context memory: the short prefill of f16 rows needs no other, so that
// it may be captured first, replayed after any later call and run on two streams at once, and no call needs a larger workspace
// than a longer one before it.  A launch that gave up on a wait leaves no counter behind for the next.  Taking it from the pool costs
// nothing that can be measured (two builds in turn that differed in this alone, 48 tokens of 5120 x 17408 up and down: 66.8 us from the
// pool, 66.8 to 67.0 from the context's workspace).
static int take_shares(zq_ctx *ctx, GemmParams &p, LaunchScratch &scratch, zq_error *err) {
    if (!p.cut_tiles) return ZQ_OK;
    const size_t head = ((size_t)2 * p.cut_pairs * sizeof(uint32_t) + 1023) & ~size_t(1023);
    const int rc = scratch.take(ctx, head + (size_t)p.cut_pairs * 2 * 2 * p.bn * kBM * sizeof(float), err);
    if (rc) return rc;
    p.counters = reinterpret_cast<uint32_t *>(scratch.p);
    p.partials = reinterpret_cast<float *>(reinterpret_cast<uint8_t *>(scratch.p) + head);
    return ZQ_OK;
}

// y[m, n] = x[m, k] W^T (+ residual), or silu(x gate^T) * (x up^T) when w_up is given.
int launch_gemm(zq_ctx *ctx, const zq_weight *w, const zq_weight *w_up, const void *x, int x_dtype, size_t m, void *y, int y_dtype, const void *residual, zq_error *err) {
    const bool gated = w_up != nullptr;
    const size_t n = w->rows, k = w->cols;
    if (k % 8) return set_error(err, ZQ_ERR_SHAPE, "prefill GEMM needs columns aligned to 8, got %zu", k);
    // Dequantising inside the kernel saves the operand pass (one read of the packed weight, one write and one read of its f16
    // form); against it stands that every token tile dequantises the weight again, which its MMAs hide unless there are few columns per
    // output (a short tile's epilogue competes with the dequantisers for issue) or the type takes many instructions (Q6_K, then Q5_K, then
    // IQ4_NL) and the rows are so many that the power cap, not the idle tensor cores, pays for them.  The operands are the same bits, and so
    // are results where the tiles are cut alike.  Measured in turn, inside / pass, us:
    //   rows                 1100       1500       2048       3001       4096       8192       16384
    //   Q4_K   1024 -> 4096  16/21      17/23      18/23      23/27      33/33
    //   Q4_K   2048 -> 8192  34/47      41/55      57/73      79/95      100/117    193/212    403/411
    //   Q4_K   5120 -> 17408 146/214    203/277    276/356    427/522    523/625    1092/1173  2227/2315
    //   IQ4_NL 5120 -> 17408 159/218    221/288    271/334    423/508    595/663    1159/1230  2314/2368
    //   Q5_K   2048 -> 8192  35/48      44/54      62/72      90/98      108/111    224/214    437/396
    //   Q5_K   4096 -> 11008 89/114     131/173    149/181    222/251    312/338    596/596    1234/1187
    //   Q6_K   4096 -> 11008 99/105     115/137    166/165    271/249    372/323    701/575    1442/1119
    //   gated:
    //   Q4_K   2048 -> 8192  67/86      86/105     108/123    171/179    223/219    477/416    961/792
    //   Q4_K   4096 -> 11008 156/227    189/264    292/366    375/465    540/637    1107/1195  2269/2367
    //   Q8_0   4096 -> 11008 169/213    190/255    291/348    405/471    531/603    1141/1192  2333/2401
    //   IQ4_NL 5120 -> 17408 341/455    406/546    517/645    831/969    1049/1148  2283/2392  5309/5012
    //   Q5_K   4096 -> 11008 200/256    204/264    305/355    458/499    602/625    1301/1240  2615/2369
    //   Q6_K   4096 -> 11008 181/200    243/257    341/329    493/446    750/623    1472/1145  3050/2250
    const size_t most = w->type == ZQ_Q5_K ? (gated ? 6000 : k >= 3072 ? 12000 : 4096) : w->type == ZQ_IQ4_NL && (gated || k < 3072) ? 12000 : SIZE_MAX;
    const bool inside = w->type == ZQ_Q6_K ? m <= 1536 : m <= 2048 || (k >= (gated ? 3072 : 2048) && m <= most);
    const bool fused = !ctx->disable_fused_gemm && (ctx->force_fused_gemm || inside) && has_i8_decode(w->type) && (!gated || w_up->type == w->type);
    GemmParams p;
    clear_params(ctx, p);
    const int row_tiles = (int)((n + (gated ? kPairM / 2 : kPairM) - 1) / (gated ? kPairM / 2 : kPairM));
    plan_tokens(m, kBN, p);
    // Wide tiles where the rounds of whole tiles come out shorter: a step is the dequantisation of one, 1.5 us beside the wide form's MMAs, or 5.6 ns
    // per token, and a wide tile costs up to 40 ns per token more at its end, where its accumulator is given back in chunks (gated: 20 more; 20 less
    // for types that are costly to dequantise, whose pace hides it).  Over 863 shapes of four types it is 0.4 % behind the better choice on
    // average; with 0.85 us and nothing for the end it was 1.7 %.  us, tiles of up to 256 and of up to 320:
    //   taken: Q4_K 5120 -> 17408 320 tokens 52 / 46; Q5_K 3840 -> 15360 560 tokens 71 / 60; Q6_K 3840 -> 15360 900 tokens 118 / 97, gated 5120 -> 17408 560 tokens 232 / 181
    //   not: gated Q4_K 2048 -> 8192 640 tokens 43 / 51, 3840 -> 15360 6000 tokens 1028 / 1247, gated Q8_0 4096 -> 4096 5000 tokens 240 / 284
    if (fused && m > kBN) {
        const int pairs = ctx->sm_count / 2 > 0 ? ctx->sm_count / 2 : 1, steps = (int)((k + kStepK - 1) / kStepK);
        const int end_ns = (gated ? 40 : 20) - (w->type == ZQ_Q5_K || w->type == ZQ_Q6_K ? 20 : 0);
        const auto time = [&](const GemmParams &g) {
            return (((long long)row_tiles * ((g.m + g.bn - 1) / g.bn) + pairs - 1) / pairs) * ((long long)steps * std::max(1500, 56 * g.bn / 10) + (g.wide ? end_ns * g.bn : 0));
        };
        GemmParams wide = p;
        plan_tokens(m, kWideBN, wide);
        if (wide.wide && (ctx->wide_tiles > 0 || (!ctx->wide_tiles && time(wide) <= time(p)))) p = wide;
    }
    p.a_tmem = fused && p.bn <= kShortBN;
    p.y = y;
    p.residual = residual;
    p.y_dtype = y_dtype;
    p.n_out = (int)n;
    p.k = (int)k;
    const int rows_per_tile = gated ? kPairM / 2 : kPairM;
    const size_t tiles = ((n + rows_per_tile - 1) / rows_per_tile) * ((m + p.bn - 1) / p.bn);
    if (tiles > (size_t)INT32_MAX / 4) return set_error(err, ZQ_ERR_SHAPE, "prefill GEMM: %zu rows x %zu tokens are too many for one call", n, m);
    const int pairs = plan_cut(ctx, (int)tiles, (int)((k + kStepK - 1) / kStepK), fused ? w->type : 0, gated, ((gated ? 2 : 1) * n + m) * k * 2, p);
    const size_t w_rows = gated ? 2 * ((n + 15) & ~size_t(15)) : n;  // rows of the operand in memory
    const size_t w_bytes = fused ? 0 : (w_rows * k * 2 + 1023) & ~size_t(1023);
    const size_t x_bytes = x_dtype == ZQ_F16 ? 0 : (m * k * 2 + 1023) & ~size_t(1023);
    int rc = ensure_workspace(ctx, w_bytes + x_bytes, err);
    if (rc) return rc;
    LaunchScratch scratch;
    rc = take_shares(ctx, p, scratch, err);
    if (rc) return rc;
    uint8_t *ws = reinterpret_cast<uint8_t *>(ctx->workspace);
    const __half *xin = reinterpret_cast<const __half *>(x);
    if (x_dtype != ZQ_F16) {
        __half *x16 = reinterpret_cast<__half *>(ws + w_bytes);
        rc = launch_to_f16(ctx, x, x_dtype, x16, m * k, err, p.counters, p.counters ? 2 * p.cut_pairs : 0);
        xin = x16;
    } else if (p.counters) {
        rc = launch_to_f16(ctx, nullptr, ZQ_F16, nullptr, 0, err, p.counters, 2 * p.cut_pairs);
    }
    if (rc) return rc;
    CUtensorMap map_x, map_x2;
    rc = make_token_maps(xin, m, k, p, &map_x, &map_x2, err);
    if (rc) return rc;
    if (fused) return launch_src(ctx, w->type, gated, gated ? w->unit_map_half : w->qmv_map, gated ? w_up->unit_map_half : w->qmv_map, map_x, map_x2, p, pairs, err);
    __half *w16 = reinterpret_cast<__half *>(ws);
    rc = launch_dequantize_f16(ctx, w, w16, err, gated);
    if (!rc && gated) rc = launch_dequantize_f16(ctx, w_up, w16 + 16 * k, err, true);
    if (rc) return rc;
    CUtensorMap map_w;
    rc = make_f16_map(w16, w_rows, k, kBM, &map_w, err);
    if (rc) return rc;
    return launch_src(ctx, 0, gated, map_w, map_w, map_x, map_x2, p, pairs, err);
}

static int grouped_params(zq_ctx *ctx, size_t rows, size_t k, size_t x_rows, const int4 *items, int n_items, const int *n_items_dev, bool wide, void *y, int y_dtype, GemmParams &p) {
    clear_params(ctx, p);
    p.wide = wide;
    p.y = y;
    p.y_dtype = y_dtype;
    p.m = (int)x_rows;
    p.bn = kBN;
    p.box_tok = kBN / 2;
    p.n_out = (int)rows;
    p.k = (int)k;
    p.items = items;
    p.n_items = n_items;
    p.n_items_dev = n_items_dev;
    const int pairs = ctx->sm_count / 2 > 0 ? ctx->sm_count / 2 : 1;
    return n_items < pairs ? n_items : pairs;
}

// Grouped GEMM (MoE prefill): `mats` f16 weight matrices [rows, k] stacked in one buffer (gated: gate and up of each as one matrix of twice
// the rows, 16 and 16 in turn; rows a multiple of 16), one f16 activation operand [x_rows, k] whose row ranges belong to the matrices, a device work list of
// {matrix, first row, first token row, end token row}.  y[token row, rows] in y_dtype; gated: silu(gate x) * (up x).
int launch_gemm_grouped(zq_ctx *ctx, const __half *w, bool gated, size_t mats, size_t rows, size_t k, const __half *x, size_t x_rows, const int4 *items, int n_items, void *y, int y_dtype, zq_error *err) {
    if (n_items <= 0) return ZQ_OK;
    if (k % 8) return set_error(err, ZQ_ERR_SHAPE, "grouped GEMM needs columns aligned to 8, got %zu", k);
    if (gated && rows % 16) return set_error(err, ZQ_ERR_SHAPE, "gated grouped GEMM needs rows aligned to 16, got %zu", rows);
    CUtensorMap map_w, map_x;
    int rc = make_f16_map3(w, mats, gated ? 2 * rows : rows, k, kBM, &map_w, err);
    if (!rc) rc = make_f16_map(x, x_rows, k, kBN / 2, &map_x, err);
    if (rc) return rc;
    GemmParams p;
    const int pairs = grouped_params(ctx, rows, k, x_rows, items, n_items, nullptr, false, y, y_dtype, p);
    return launch_src(ctx, 0, gated, map_w, map_w, map_x, map_x, p, pairs, err);
}

// Plain f16 x f16 GEMM on raw operands: y[m, rows] = x[m, k] w[rows, k]^T, f32 accumulation (router logits).  Whole tiles only:
// it uses no workspace, which its caller may hold.
int launch_gemm_f16(zq_ctx *ctx, const __half *w, size_t rows, size_t k, const __half *x, size_t m, void *y, int y_dtype, zq_error *err) {
    if (k % 8) return set_error(err, ZQ_ERR_SHAPE, "f16 GEMM needs columns aligned to 8, got %zu", k);
    GemmParams p;
    clear_params(ctx, p);
    plan_tokens(m, kBN, p);
    CUtensorMap map_w, map_x;
    int rc = make_f16_map(w, rows, k, kBM, &map_w, err);
    if (!rc) rc = make_f16_map(x, m, k, p.box_tok, &map_x, err);
    if (rc) return rc;
    p.y = y;
    p.y_dtype = y_dtype;
    p.n_out = (int)rows;
    p.k = (int)k;
    const size_t tiles = ((rows + kPairM - 1) / kPairM) * ((m + p.bn - 1) / p.bn);
    const int pairs = ctx->sm_count / 2 > 0 ? ctx->sm_count / 2 : 1;
    return launch_src(ctx, 0, false, map_w, map_w, map_x, map_x, p, tiles < (size_t)pairs ? (int)tiles : pairs, err);
}

// Grouped form for packed experts (MoE prefill): no f16 copy of the weights at all.  `w_maps` / `w2_maps`: device tables of the
// experts' packed-weight tensor maps (one unit x 128 rows boxes, gated: 64 rows), indexed by the work items' z.
int launch_gemm_fused_grouped(zq_ctx *ctx, uint32_t type, const CUtensorMap *w_maps, const CUtensorMap *w2_maps, size_t rows, size_t k, const __half *x, size_t x_rows, const int4 *items, int n_items, const int *n_items_dev,
                              bool wide, void *y, int y_dtype, zq_error *err) {
    if (n_items <= 0) return ZQ_OK;
    if (k % 8) return set_error(err, ZQ_ERR_SHAPE, "grouped GEMM needs columns aligned to 8, got %zu", k);
    GemmParams p;
    const int pairs = grouped_params(ctx, rows, k, x_rows, items, n_items, n_items_dev, wide, y, y_dtype, p);
    CUtensorMap map_x, map_x2;
    int rc = make_token_maps(x, x_rows, k, p, &map_x, &map_x2, err);
    if (rc) return rc;
    p.w_maps = w_maps;
    p.w2_maps = w2_maps;
    return launch_src(ctx, type, w2_maps != nullptr, map_x, map_x, map_x, map_x2, p, pairs, err);
}

}  // namespace zq
