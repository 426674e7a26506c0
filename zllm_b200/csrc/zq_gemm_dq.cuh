// Packed weights -> f16 tensor-core operand, inside the prefill GEMM (zq_gemm.cu).
//
// A dequantiser thread owns one row of a packed box (one 256-weight unit per row) and one 64-column k-block of it.
// DqBlock<TYPE>::load brings what it needs of the unit into registers (at the row pitches of these formats the eight rows of
// a quarter-warp's 16-byte loads fall into eight different bank groups, Q6_K excepted), emit() turns it into eight 16-byte
// chunks and gives them to its sink: the 128-byte-swizzle positions of a row in shared memory (chunk c of row r at c ^ (r & 7)), or a lane of tensor memory.  mix() reads every loaded
// register: an instruction that uses it has waited for the loads, so the box may be given back to the TMA unit behind it.  Shared memory is addressed
// by 32-bit shared addresses: as generic accesses the stores cost the fence behind them several times as much.
//
// Arithmetic: every operand is the codec's f32 value rounded once to f16.
//   Q4_K, Q5_K   the codec's d sc q - dmin m: sc q is at most 31 * 63, an integer f16 holds exactly, so one f16 multiply-add on the code
//                (biased by 1024 to sit in the mantissa, sc (1024 + q) - 1024 sc, for two weights) gives it without rounding, and one
//                mixed-precision multiply-add (f16 d times f16 sc q plus the f32 minimum term, rounded once to f32) does the rest: d sc has 17
//                significant bits, so the codec's products are exact too.
//                What bounds it is the ALU pipe, which takes a byte permute, a logic operation or a conversion in two cycles: 1.1 such
//                operations per weight of about 2.6 instructions.  With codes permuted under an f32 exponent (fma(s, 128 + q - 128, -m)) it were
//                1.9 of 2.9: 48 tokens of 5120 x 17408 up and down 63.1 us, now 58.0.  (A bias that stays in the product would save an
//                instruction there, but rounds the minimum away where it is small beside the scale.)
//   Q6_K         fma(s, 128 + q + 32, -160 s) = s q: 160 s is exact, there is no other offset.  Two multiply-adds per instruction
//                (fma.rn.f32x2).
//   Q4_0, IQ4_NL, Q8_0 d q with d an f16 and q an integer of at most 8 bits: an f16 multiply rounds the exact product once,
//                      which is what multiplying in f32 (exact) and rounding does.
#pragma once
#include "zq_common.cuh"

namespace zq {

__device__ __forceinline__ uint32_t dq_prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}
__device__ __forceinline__ uint64_t dq_pair(float v) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
    return r;
}
// f32 sums f16 * f16 + f32, rounded once: the mixed-precision multiply-add of this architecture takes either half of a register
// pair, at the rate of an f32 one.
__device__ __forceinline__ void dq_fma_halves(uint32_t t2, unsigned short d, float c, float &lo, float &hi) {
    asm("{\n\t.reg .b16 l, h;\n\t"
        "mov.b32 {l, h}, %2;\n\t"
        "fma.rn.f32.f16 %0, l, %3, %4;\n\t"
        "fma.rn.f32.f16 %1, h, %3, %4;\n\t}"
        : "=f"(lo), "=f"(hi)
        : "r"(t2), "h"(d), "f"(c));
}
__device__ __forceinline__ float dq_fma_half(unsigned short a, unsigned short b, float c) {
    float r;
    asm("fma.rn.f32.f16 %0, %1, %2, %3;" : "=f"(r) : "h"(a), "h"(b), "f"(c));
    return r;
}
__device__ __forceinline__ uint32_t dq_pack(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ uint32_t dq_hfma2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}
// (a & b) | c
__device__ __forceinline__ uint32_t dq_and_or(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}
// codes in bytes J, J + 1 of `codes` -> f16x2 of s * (128 + q) + c
template <int J> __device__ __forceinline__ uint32_t dq_fma2(uint32_t codes, uint64_t s2, uint64_t c2) {
    const uint32_t a = dq_prmt(codes, 0x43000000u, 0x7044u + (J << 8)), b = dq_prmt(codes, 0x43000000u, 0x7044u + ((J + 1) << 8));
    uint64_t v;
    uint32_t lo, hi, r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(a), "r"(b));
    asm("fma.rn.f32x2 %0, %0, %1, %2;" : "+l"(v) : "l"(s2), "l"(c2));
    asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v));
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(__uint_as_float(hi)), "f"(__uint_as_float(lo)));
    return r;
}
__device__ __forceinline__ uint4 dq_chunk_fma(uint32_t w0, uint32_t w1, uint64_t s2, uint64_t c2) { return make_uint4(dq_fma2<0>(w0, s2, c2), dq_fma2<2>(w0, s2, c2), dq_fma2<0>(w1, s2, c2), dq_fma2<2>(w1, s2, c2)); }
// unsigned bytes -> f16 (byte - bias) * d; bias2 = f16x2 of 1024 + bias, d2 = f16x2 of d
__device__ __forceinline__ uint4 dq_chunk_mul(uint32_t w0, uint32_t w1, uint32_t bias2, uint32_t d2) {
    uint4 r;
    r.x = hmul2_u32(hsub2_u32(dq_prmt(w0, 0x64646464u, 0x4140u), bias2), d2);
    r.y = hmul2_u32(hsub2_u32(dq_prmt(w0, 0x64646464u, 0x4342u), bias2), d2);
    r.z = hmul2_u32(hsub2_u32(dq_prmt(w1, 0x64646464u, 0x4140u), bias2), d2);
    r.w = hmul2_u32(hsub2_u32(dq_prmt(w1, 0x64646464u, 0x4342u), bias2), d2);
    return r;
}
// The 16-byte chunk c (0..7) of a 128-byte swizzled row.
__device__ __forceinline__ void dq_store(uint32_t row_base, int sw, int c, uint4 v) {
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(row_base + ((c ^ sw) << 4)), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ uint4 dq_lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint2 dq_lds64(uint32_t addr) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t dq_lds32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}

// Where emit() puts chunk c (columns 8 c .. 8 c + 7 of the k-block): the swizzled row of the operand tile in shared memory, or the
// thread's lane of the operand in tensor memory (two columns of K per 32-bit column; the whole warp stores together).
struct DqSharedRow {
    uint32_t row_base;
    int sw;
    __device__ __forceinline__ void put(int c, uint4 v) const { dq_store(row_base, sw, c, v); }
};
struct DqTensorRow {
    uint32_t at;
    __device__ __forceinline__ void put(int c, uint4 v) const {
        asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(at + 4u * (uint32_t)c), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
    }
};

template <uint32_t TYPE> struct DqBlock;

template <bool Q5> struct DqBlockK {
    uint4 q[2];          // the k-block's 32 quant bytes
    uint4 hb[Q5 ? 2 : 1];  // Q5_K: the high-bit bytes
    uint32_t sc;         // f16x2: 6-bit scales of groups 2 kb and 2 kb + 1
    unsigned short d;    // f16
    float c[2];          // -dmin m of the two groups
    int g;
    __device__ __forceinline__ void load(uint32_t unit, int kb) {  // kb is warp-uniform
        const uint4 hdr = dq_lds128(unit);
        const uint32_t qs = unit + (Q5 ? 48 : 16) + 32 * kb;
        q[0] = dq_lds128(qs);
        q[1] = dq_lds128(qs + 16);
        if constexpr (Q5) {
            hb[0] = dq_lds128(unit + 16);
            hb[1] = dq_lds128(unit + 32);
        }
        g = 2 * kb;
        uint32_t scw, mnw;  // the four groups of this half as bytes
        if (kb < 2) {
            scw = hdr.y & 0x3F3F3F3Fu;
            mnw = hdr.z & 0x3F3F3F3Fu;
        } else {
            scw = (hdr.w & 0x0F0F0F0Fu) | ((hdr.y >> 2) & 0x30303030u);
            mnw = ((hdr.w >> 4) & 0x0F0F0F0Fu) | ((hdr.z >> 2) & 0x30303030u);
        }
        const uint32_t pick = (kb & 1) ? 0x4342u : 0x4140u;  // bytes -> f16 1024 + byte
        sc = hsub2_u32(dq_prmt(scw, 0x64646464u, pick), 0x64006400u);
        const uint32_t mn = hsub2_u32(dq_prmt(mnw, 0x64646464u, pick), 0x64006400u);
        d = (unsigned short)(hdr.x & 0xFFFFu);
        const unsigned short minus_dmin = (unsigned short)((hdr.x >> 16) ^ 0x8000u);
        c[0] = dq_fma_half(minus_dmin, (unsigned short)(mn & 0xFFFFu), -0.0f);
        c[1] = dq_fma_half(minus_dmin, (unsigned short)(mn >> 16), -0.0f);
    }
    __device__ __forceinline__ uint32_t mix() const {
        uint32_t m = q[0].x ^ q[0].y ^ q[0].z ^ q[0].w ^ q[1].x ^ q[1].y ^ q[1].z ^ q[1].w ^ __float_as_uint(c[0]);
        if constexpr (Q5) m ^= hb[0].x ^ hb[0].y ^ hb[0].z ^ hb[0].w ^ hb[1].x ^ hb[1].y ^ hb[1].z ^ hb[1].w;
        return m;
    }
    // f16x2 operands of columns (0, 1) and (2, 3) from the f16x2 codes of columns (0, 2) and (1, 3), biased by 1024
    __device__ __forceinline__ uint2 four(uint32_t even, uint32_t odd, uint32_t s2, uint32_t k2, float cn) const {
        float v0, v1, v2, v3;
        dq_fma_halves(dq_hfma2(even, s2, k2), d, cn, v0, v2);
        dq_fma_halves(dq_hfma2(odd, s2, k2), d, cn, v1, v3);
        return make_uint2(dq_pack(v0, v1), dq_pack(v2, v3));
    }
    template <class Sink> __device__ __forceinline__ void emit(const Sink &sink) const {
        const uint32_t w[8] = {q[0].x, q[0].y, q[0].z, q[0].w, q[1].x, q[1].y, q[1].z, q[1].w};
#pragma unroll
        for (int n = 0; n < 2; ++n) {  // low nibbles: group 2 kb, high nibbles: group 2 kb + 1
            uint32_t s2 = dq_prmt(sc, 0u, n ? 0x3232u : 0x1010u);
            if (n && !Q5) s2 = hmul2_u32(s2, 0x2C002C00u);  // high nibbles stay in place, as 16 q
            const uint32_t k2 = hmul2_u32(s2, 0xE400E400u);   // takes the bias 1024 off again
#pragma unroll
            for (int c8 = 0; c8 < 4; ++c8) {
                uint2 r[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const uint32_t x = w[2 * c8 + i];
                    uint32_t even, odd;
                    if constexpr (Q5) {  // bit g + n of every high-bits byte -> bit 4 of the code
                        const uint4 &h4 = hb[c8 >> 1];
                        const uint32_t hw = (c8 & 1) ? (i ? h4.w : h4.z) : (i ? h4.y : h4.x);
                        const uint32_t code = ((n ? (x >> 4) : x) & 0x0F0F0F0Fu) | (((hw >> (g + n)) << 4) & 0x10101010u);
                        even = dq_prmt(code, 0x64646464u, 0x4240u);
                        odd = dq_prmt(code, 0x64646464u, 0x4341u);
                    } else {
                        const uint32_t mask = n ? 0x00F000F0u : 0x000F000Fu;
                        even = dq_and_or(x, mask, 0x64006400u);
                        odd = dq_and_or(x >> 8, mask, 0x64006400u);
                    }
                    r[i] = four(even, odd, s2, k2, c[n]);
                }
                sink.put(4 * n + c8, make_uint4(r[0].x, r[0].y, r[1].x, r[1].y));
            }
        }
    }
};
template <> struct DqBlock<ZQ_Q4_K> : DqBlockK<false> {};
template <> struct DqBlock<ZQ_Q5_K> : DqBlockK<true> {};

template <> struct DqBlock<ZQ_Q6_K> {
    uint2 lo[4];     // per t: low-nibble words of blocks G = 2 kb, 2 kb + 1
    uint32_t hi[4];  // per t: high-bit word of the k-block
    uint32_t sc;     // its four i8 group scales
    float d;
    __device__ __forceinline__ void load(uint32_t unit, int kb) {
        d = __half2float(__ushort_as_half((unsigned short)(dq_lds32(unit) & 0xFFFFu)));
        sc = dq_lds32(unit + kQ6kScales + 4 * kb);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            lo[t] = dq_lds64(unit + kQ6kLow + 32 * t + 8 * kb);
            hi[t] = dq_lds32(unit + kQ6kHigh + 16 * t + 4 * kb);
        }
    }
    __device__ __forceinline__ uint32_t mix() const {
        return lo[0].x ^ lo[0].y ^ lo[1].x ^ lo[1].y ^ lo[2].x ^ lo[2].y ^ lo[3].x ^ lo[3].y ^ hi[0] ^ hi[1] ^ hi[2] ^ hi[3] ^ sc ^ __float_as_uint(d);
    }
    template <class Sink> __device__ __forceinline__ void emit(const Sink &sink) const {
#pragma unroll
        for (int i = 0; i < 8; ++i) {  // eight columns: block G = 2 kb + c8 / 4, scale group h = (c8 / 2) & 1, t = 2 (c8 & 1) and t + 1
            const int c8 = 2 * (i & 3) + (i >> 2);  // all that t = 0, 1 serve first: fewer registers are live (no spills in 72)
            const int gb = c8 >> 2, hh = (c8 >> 1) & 1, x2 = 2 * (2 * gb + hh);
            const float s = __fmul_rn(d, (float)(int8_t)(sc >> (8 * (2 * gb + hh))));
            const uint64_t s2 = dq_pair(s), c2 = dq_pair(-160.0f * s);  // the byte below is q = c + 32 (0..63): 128 + q - 160 = q - 32
            uint32_t m[2];
#pragma unroll
            for (int w = 0; w < 2; ++w) {
                const int t = 2 * (c8 & 1) + w;
                const uint32_t lw = gb ? lo[t].y : lo[t].x, hw = hi[t];
                const uint32_t l = (hh ? (lw >> 4) : lw) & 0x0F0F0F0Fu, u = (x2 >= 4 ? (hw >> (x2 - 4)) : (hw << (4 - x2))) & 0x30303030u;
                m[w] = (l | u) ^ 0x20202020u;
            }
            sink.put(c8, dq_chunk_fma(m[0], m[1], s2, c2));
        }
    }
};

// Q4_0 and IQ4_NL: piece t of a unit half holds word t of the half's four blocks; a k-block is two of them
template <bool NL> struct DqBlock4 {
    uint2 p[4];
    uint32_t d;
    __device__ __forceinline__ void load(uint32_t unit, int kb) {
        d = dq_lds32(unit + 4 * kb);
#pragma unroll
        for (int t = 0; t < 4; ++t) p[t] = dq_lds64(unit + 16 + 16 * (t + 4 * (kb >> 1)) + 8 * (kb & 1));
    }
    __device__ __forceinline__ uint32_t mix() const { return p[0].x ^ p[0].y ^ p[1].x ^ p[1].y ^ p[2].x ^ p[2].y ^ p[3].x ^ p[3].y ^ d; }
    template <class Sink> __device__ __forceinline__ void emit(const Sink &sink) const {
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const uint32_t d2 = dq_prmt(d, 0u, b ? 0x3232u : 0x1010u);
            uint32_t lo[4], hi[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const uint32_t w = b ? p[t].y : p[t].x;
                if constexpr (NL) {
                    // codebook values + 128 as bytes, looked up with PRMT (see iq4nl_lookup in zq_i8.cuh)
                    constexpr uint32_t T0 = 0x3F2D1801u, T1 = 0x766A5D4Fu, T2 = 0xA6998D81u, T3 = 0xF1D9C5B5u;
                    const uint32_t ws = w & 0x77777777u, w4 = w << 4, ws2 = ws >> 16;
                    const uint32_t mx = dq_prmt(w4, w, 0xD9C8u), my = dq_prmt(w4, w, 0xFBEAu);
                    const uint32_t x0 = dq_prmt(T0, T1, ws), x1 = dq_prmt(T2, T3, ws), y0 = dq_prmt(T0, T1, ws2), y1 = dq_prmt(T2, T3, ws2);
                    const uint32_t x = (mx & x1) | (~mx & x0), y = (my & y1) | (~my & y0);
                    lo[t] = dq_prmt(x, y, 0x6420u);
                    hi[t] = dq_prmt(x, y, 0x7531u);
                } else {
                    lo[t] = w & 0x0F0F0F0Fu;
                    hi[t] = (w >> 4) & 0x0F0F0F0Fu;
                }
            }
            constexpr uint32_t bias2 = NL ? 0x64806480u : 0x64086408u;  // 1024 + 128, 1024 + 8
            sink.put(4 * b + 0, dq_chunk_mul(lo[0], lo[1], bias2, d2));
            sink.put(4 * b + 1, dq_chunk_mul(lo[2], lo[3], bias2, d2));
            sink.put(4 * b + 2, dq_chunk_mul(hi[0], hi[1], bias2, d2));
            sink.put(4 * b + 3, dq_chunk_mul(hi[2], hi[3], bias2, d2));
        }
    }
};
template <> struct DqBlock<ZQ_Q4_0> : DqBlock4<false> {};
template <> struct DqBlock<ZQ_IQ4_NL> : DqBlock4<true> {};

template <> struct DqBlock<ZQ_Q8_0> {  // piece t of a k-block: words t (columns 4t..) and 4 + t (columns 16 + 4t..) of its two blocks
    uint4 p[4];
    uint32_t d;
    __device__ __forceinline__ void load(uint32_t unit, int kb) {
        d = dq_lds32(unit + 4 * kb);
#pragma unroll
        for (int t = 0; t < 4; ++t) p[t] = dq_lds128(unit + 16 + 64 * kb + 16 * t);
    }
    __device__ __forceinline__ uint32_t mix() const {
        uint32_t m = d;
#pragma unroll
        for (int t = 0; t < 4; ++t) m ^= p[t].x ^ p[t].y ^ p[t].z ^ p[t].w;
        return m;
    }
    template <class Sink> __device__ __forceinline__ void emit(const Sink &sink) const {
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const uint32_t d2 = dq_prmt(d, 0u, b ? 0x3232u : 0x1010u);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const uint4 &a0 = p[2 * (c & 1)], &a1 = p[2 * (c & 1) + 1];
                const uint32_t w0 = b ? ((c >> 1) ? a0.w : a0.z) : ((c >> 1) ? a0.y : a0.x), w1 = b ? ((c >> 1) ? a1.w : a1.z) : ((c >> 1) ? a1.y : a1.x);
                sink.put(4 * b + c, dq_chunk_mul(w0 ^ 0x80808080u, w1 ^ 0x80808080u, 0x64806480u, d2));
            }
        }
    }
};

}  // namespace zq
