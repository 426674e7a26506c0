// Codec kernels: GGUF -> resident re-layout, bit-exact dequantisation (all rows or gathered rows), and the
// device-side encoders.
//
// Reference behaviour restated here:
//   decode formulas         src/weight/codec/ggml.rs:102-109 (Q4_0), 229-234 (Q8_0), 237-244 (IQ4_NL), 408-423 (Q4_K)
//   dequantize              src/weight/codec/ggml.rs:146-160
//   gathered rows to f16    src/kernel/cuda/linear.rs:1420-1437 (gguf_rows_f16)
//   encode_q4_k             src/weight/codec/ggml.rs:188-227
#include <type_traits>

#include "zq_common.cuh"

namespace zq {

// One thread per resident byte: find the GGUF byte it comes from.  Padding blocks (beyond the row's last
// GGUF block) are zero.
__global__ void repack_kernel(uint32_t type, const uint8_t *__restrict__ gguf, uint8_t *__restrict__ resident, size_t rows, size_t blocks_per_row, size_t units_per_row, int unit_bytes, int block_bytes) {
    size_t row_pitch = units_per_row * (size_t)unit_bytes;
    size_t total = rows * row_pitch;
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
        size_t row = idx / row_pitch;
        size_t in_row = idx % row_pitch;
        size_t unit = in_row / unit_bytes;
        int o = (int)(in_row % unit_bytes);
        int block, src;
        if (o < 16) {
            block = o >> 1;
            src = o & 1;
        } else {
            int u = (o - 16) >> 4, w = ((o - 16) & 15) >> 2, by = o & 3;
            int t = u & 3, h = u >> 2;
            if (type == ZQ_Q8_0) {
                block = 2 * h + (w >> 1);
                src = 2 + 4 * (4 * (w & 1) + t) + by;
            } else {
                block = 4 * h + w;
                src = 2 + 4 * t + by;
            }
        }
        size_t gblock = unit * 8 + block;
        uint8_t v = 0;
        if (gblock < blocks_per_row) v = gguf[(row * blocks_per_row + gblock) * block_bytes + src];
        resident[idx] = v;
    }
}

// The 6-bit code (0..63) of column `i` of a GGUF Q6_K super-block (src/weight/codec/ggml.rs:446-469: 128 low-nibble
// bytes, 64 high-bit bytes, 16 i8 scales, d).
__device__ __forceinline__ int q6k_gguf_code(const uint8_t *block, int i) {
    const int half = i >> 7, quarter = (i >> 5) & 3, index = i & 31;
    const uint8_t lo = block[half * 64 + index + ((quarter & 1) ? 32 : 0)];
    const uint8_t hv = block[128 + half * 32 + index];
    return (int)(((quarter & 2) ? (lo >> 4) : (lo & 0x0f)) | (((hv >> (2 * quarter)) & 3) << 4));
}

// One thread per resident byte of the Q6_K units (layout: kQ6k* in zq_common.cuh).
__global__ void repack_q6k_kernel(const uint8_t *__restrict__ gguf, uint8_t *__restrict__ resident, size_t rows, size_t units_per_row) {
    const size_t total = rows * units_per_row * 224;
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
        const size_t unit = idx / 224;
        const int o = (int)(idx - unit * 224);
        const uint8_t *block = gguf + unit * 210;  // rows are whole super-blocks: unit u of the tensor is block u of the file
        uint8_t v = 0;
        if (o < 2) {
            v = block[208 + o];
        } else if (o >= kQ6kScales && o < kQ6kLow) {
            v = block[192 + (o - kQ6kScales)];
        } else if (o >= kQ6kLow && o < kQ6kHigh) {
            const int r = o - kQ6kLow, t = r >> 5, G = (r >> 2) & 7, i = r & 3;
            const int c0 = (q6k_gguf_code(block, 32 * G + 4 * t + i) - 32) & 63, c1 = (q6k_gguf_code(block, 32 * G + 16 + 4 * t + i) - 32) & 63;
            v = (uint8_t)((c0 & 15) | ((c1 & 15) << 4));
        } else if (o >= kQ6kHigh) {
            const int r = o - kQ6kHigh, t = r >> 4, vv = (r >> 2) & 3, i = r & 3;
            for (int x = 0; x < 4; ++x) {
                const int G = 2 * vv + (x >> 1), h = x & 1;
                const int c = (q6k_gguf_code(block, 32 * G + 16 * h + 4 * t + i) - 32) & 63;
                v |= (uint8_t)((c >> 4) << (2 * x));
            }
        }
        resident[idx] = v;
    }
}

int launch_repack(zq_ctx *ctx, uint32_t type, const uint8_t *gguf, uint8_t *resident, size_t rows, size_t cols, zq_error *err) {
    if (type == ZQ_Q6_K) {
        const size_t units = cols / kUnitWeights, total_q6 = rows * units * 224;
        if (total_q6 == 0) return ZQ_OK;
        size_t nb = (total_q6 + 255) / 256;
        if (nb > 65535u * 16u) nb = 65535u * 16u;
        repack_q6k_kernel<<<(unsigned)nb, 256, 0, ctx->stream>>>(gguf, resident, rows, units);
        ctx->launches++;
        ZQ_CUDA_CHECK(cudaGetLastError(), err);
        return ZQ_OK;
    }
    FormatInfo f = format_info(type);
    size_t blocks_per_row = cols / f.block_elems;
    size_t units_per_row = (cols + kUnitWeights - 1) / kUnitWeights;
    size_t total = rows * units_per_row * f.unit_bytes;
    if (total == 0) return ZQ_OK;
    int threads = 256;
    size_t blocks = (total + threads - 1) / threads;
    if (blocks > 65535u * 16u) blocks = 65535u * 16u;
    repack_kernel<<<(unsigned)blocks, threads, 0, ctx->stream>>>(type, gguf, resident, rows, blocks_per_row, units_per_row, f.unit_bytes, f.block_bytes);
    ctx->launches++;
    ZQ_CUDA_CHECK(cudaGetLastError(), err);
    return ZQ_OK;
}

// Decode element `i` (0..255) of a resident unit.  Every product below is exactly representable in f32, so the
// only rounding is the reference's final subtraction; __fmul_rn/__fsub_rn keep the compiler from contracting.
__device__ __forceinline__ float decode_unit_element(uint32_t type, const uint8_t *unit, int i) {
    if (type == ZQ_Q5_K) {  // src/weight/codec/ggml.rs:425-444: d, dmin, 12 scale bytes, 32 high-bit bytes, 128 low-nibble bytes
        const __half *hd = reinterpret_cast<const __half *>(unit);
        const float d = __half2float(hd[0]), dmin = __half2float(hd[1]);
        const uint8_t *scales = unit + 4;
        const int g = i >> 5, j = i & 31;
        int sc, mn;
        if (g < 4) {
            sc = scales[g] & 0x3f;
            mn = scales[g + 4] & 0x3f;
        } else {
            sc = (scales[g + 4] & 0x0f) | ((scales[g - 4] >> 6) << 4);
            mn = (scales[g + 4] >> 4) | ((scales[g] >> 6) << 4);
        }
        const uint8_t packed = unit[48 + (g >> 1) * 32 + j];
        const int quant = ((g & 1) ? (packed >> 4) : (packed & 0x0f)) + (((unit[16 + j] >> g) & 1) << 4);
        return __fsub_rn(__fmul_rn(__fmul_rn(d, (float)sc), (float)quant), __fmul_rn(dmin, (float)mn));
    }
    if (type == ZQ_Q6_K) {  // src/weight/codec/ggml.rs:446-469 on the re-laid unit (kQ6k* in zq_common.cuh): (d * scale) * (q - 32)
        const float d = __half2float(*reinterpret_cast<const __half *>(unit));
        const int G = i >> 5, h = (i >> 4) & 1, t = (i >> 2) & 3, ii = i & 3;
        const int lo = (unit[kQ6kLow + 32 * t + 4 * G + ii] >> (4 * h)) & 15;
        const int hi = (unit[kQ6kHigh + 16 * t + 4 * (G >> 1) + ii] >> (2 * (2 * (G & 1) + h))) & 3;
        const int c = lo | (hi << 4);
        const int q = c >= 32 ? c - 64 : c;  // the stored code is (q - 32) mod 64
        const int8_t scale = (int8_t)unit[kQ6kScales + (i >> 4)];
        return __fmul_rn(__fmul_rn(d, (float)scale), (float)q);
    }
    if (type == ZQ_Q5_0 || type == ZQ_Q5_1) {  // src/weight/codec/ggml.rs:111-130; the unit is 8 GGUF blocks in file order
        const int e = i & 31;
        const uint8_t *block = unit + (i >> 5) * (type == ZQ_Q5_0 ? 22 : 24);
        const float d = __half2float(*reinterpret_cast<const __half *>(block));
        const int hoff = type == ZQ_Q5_0 ? 2 : 4;
        const uint32_t high = (uint32_t)block[hoff] | ((uint32_t)block[hoff + 1] << 8) | ((uint32_t)block[hoff + 2] << 16) | ((uint32_t)block[hoff + 3] << 24);
        const uint8_t packed = block[hoff + 4 + (e & 15)];
        const int q5 = (int)((e < 16 ? (packed & 15) : (packed >> 4)) | (((high >> e) & 1u) << 4));
        if (type == ZQ_Q5_0) return __fmul_rn(d, (float)(q5 - 16));
        return __fadd_rn(__fmul_rn(d, (float)q5), __half2float(*reinterpret_cast<const __half *>(block + 2)));
    }
    if (type == ZQ_IQ4_XS) {  // src/weight/codec/ggml.rs:246-261
        const float d = __half2float(*reinterpret_cast<const __half *>(unit));
        const uint32_t scales_h = (uint32_t)unit[2] | ((uint32_t)unit[3] << 8);
        const int ib = i >> 5, j = i & 31;
        const int ls = (int)(((unit[4 + ib / 2] >> (4 * (ib & 1))) & 0x0f) | (((scales_h >> (2 * ib)) & 3u) << 4));
        const float dl = __fmul_rn(d, __fsub_rn((float)ls, 32.0f));
        const uint8_t qb = unit[8 + ib * 16 + (j & 15)];
        return __fmul_rn(dl, (float)kIq4nlValues[j < 16 ? (qb & 0x0f) : (qb >> 4)]);
    }
    if (type == ZQ_Q3_K) {  // src/weight/codec/ggml.rs:384-406
        const uint8_t *hmask = unit, *quants = unit + 32, *scales = unit + 96;
        const float d = __half2float(*reinterpret_cast<const __half *>(unit + 108));
        const int group = i >> 4, index = i & 15;
        const int low = group < 8 ? (scales[group] & 0x0f) : (scales[group - 8] >> 4);
        const int high = (scales[8 + (group & 3)] >> (2 * (group >> 2))) & 3;
        const int scale = (low | (high << 4)) - 32;
        const int half = group >> 3, pair = group & 7;
        const int low_bits = (quants[half * 32 + (pair & 1) * 16 + index] >> (2 * (pair >> 1))) & 3;
        const int quant = low_bits - ((hmask[(pair & 1) * 16 + index] & (1u << (group >> 1))) ? 0 : 4);
        return __fmul_rn(__fmul_rn(d, (float)scale), (float)quant);
    }
    uint8_t q = unit[unit_quant_offset(type, i)];
    if (type == ZQ_Q4_K) {
        const __half *hd = reinterpret_cast<const __half *>(unit);
        float d = __half2float(hd[0]), dmin = __half2float(hd[1]);
        const uint8_t *scales = unit + 4;
        int g = i >> 5;
        int sc, mn;
        if (g < 4) {
            sc = scales[g] & 0x3f;
            mn = scales[g + 4] & 0x3f;
        } else {
            sc = (scales[g + 4] & 0x0f) | ((scales[g - 4] >> 6) << 4);
            mn = (scales[g + 4] >> 4) | ((scales[g] >> 6) << 4);
        }
        int quant = (g & 1) ? (q >> 4) : (q & 0x0f);
        return __fsub_rn(__fmul_rn(__fmul_rn(d, (float)sc), (float)quant), __fmul_rn(dmin, (float)mn));
    }
    int blk = i >> 5, e = i & 31;
    float d = __half2float(reinterpret_cast<const __half *>(unit)[blk]);
    if (type == ZQ_Q8_0) return __fmul_rn(d, (float)(int8_t)q);
    int nib = (e >> 4) ? (q >> 4) : (q & 0x0f);
    if (type == ZQ_Q4_0) return __fmul_rn((float)(nib - 8), d);
    return __fmul_rn(d, (float)kIq4nlValues[nib]);
}

// N = 8 or 4 consecutive elements from i0 (a multiple of N) of a resident unit, the same bits as decode_unit_element: the
// scale and the packed words are read once for all (an element-wise decode reads and unpacks them eight times, which
// at 8 bytes of output per packed byte, not HBM, bounded the passes built on it).  The elements lie in one 32-element
// group of every format and, in the re-laid formats, in one word (of neighbouring pieces) per four.
__device__ __forceinline__ void bytes_to_f32(uint32_t w, float *v) {  // four unsigned bytes
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = (float)((w >> (8 * j)) & 0xFFu);
}
__device__ __forceinline__ void sbytes_to_f32(uint32_t w, float *v) {  // four signed bytes
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = (float)(int8_t)(w >> (8 * j));
}
// f16 under an 8-bit-aligned K-quant header: (d * sc, dmin * m) of group g from the 12 scale bytes (src/weight/codec/ggml.rs:471-473)
__device__ __forceinline__ void kquant_group(const uint4 &hdr, int g, float &dsc, float &dm) {
    const __half2 dd = u32_as_h2(hdr.x);
    const int j = 8 * (g & 3);
    uint32_t sc, mn;
    if (g < 4) {
        sc = (hdr.y >> j) & 63u;
        mn = (hdr.z >> j) & 63u;
    } else {
        sc = ((hdr.w >> j) & 15u) | (((hdr.y >> (j + 6)) & 3u) << 4);
        mn = ((hdr.w >> (j + 4)) & 15u) | (((hdr.z >> (j + 6)) & 3u) << 4);
    }
    dsc = __fmul_rn(__low2float(dd), (float)sc);
    dm = __fmul_rn(__high2float(dd), (float)mn);
}
__device__ __forceinline__ uint32_t iq4nl_bytes(uint32_t nibs) {  // four codebook values (s8) of the low nibbles of four bytes
    constexpr uint32_t T0 = 0xBFAD9881u, T1 = 0xF6EADDCFu, T2 = 0x26190D01u, T3 = 0x71594535u;  // -127 .. 113
    const uint32_t sel = (nibs & 7u) | ((nibs >> 4) & 0x70u) | ((nibs >> 8) & 0x700u) | ((nibs >> 12) & 0x7000u);
    uint32_t lo, hi, mask = ((nibs >> 3) & 0x01010101u) * 0xFFu;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(lo) : "r"(T0), "r"(T1), "r"(sel));
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(hi) : "r"(T2), "r"(T3), "r"(sel));
    return (hi & mask) | (lo & ~mask);
}
template <uint32_t TYPE, int N> __device__ __forceinline__ void decode_run(const uint8_t *unit, int i0, float (&v)[N]) {
    static_assert(N == 4 || N == 8, "runs of 4 or 8 elements");
    constexpr int W = N / 4;  // packed words
    if constexpr (TYPE == ZQ_Q4_K || TYPE == ZQ_Q5_K) {
        const uint4 hdr = *reinterpret_cast<const uint4 *>(unit);
        const int g = i0 >> 5, j0 = i0 & 31;
        float dsc, dm;
        kquant_group(hdr, g, dsc, dm);
        auto words = [](const uint8_t *at, uint32_t (&w)[W]) {
            if constexpr (W == 2) {
                const uint2 x = *reinterpret_cast<const uint2 *>(at);
                w[0] = x.x;
                w[W - 1] = x.y;
            } else {
                w[0] = *reinterpret_cast<const uint32_t *>(at);
            }
        };
        const int shift = (g & 1) * 4;
        uint32_t q[W], hb[W];
        words(unit + (TYPE == ZQ_Q5_K ? 48 : 16) + (g >> 1) * 32 + j0, q);
        if constexpr (TYPE == ZQ_Q5_K) words(unit + 16 + j0, hb);
#pragma unroll
        for (int w = 0; w < W; ++w) {
            uint32_t a = (q[w] >> shift) & 0x0F0F0F0Fu;
            if constexpr (TYPE == ZQ_Q5_K) a |= ((hb[w] >> g) & 0x01010101u) << 4;
            bytes_to_f32(a, v + 4 * w);
        }
#pragma unroll
        for (int j = 0; j < N; ++j) v[j] = __fsub_rn(__fmul_rn(dsc, v[j]), dm);
    } else if constexpr (TYPE == ZQ_Q6_K) {  // columns 32 G + 16 h + 4 t + i: eight are (t, 0..3) and (t + 1, 0..3) of one scale group
        const int G = i0 >> 5, h = (i0 >> 4) & 1, t = (i0 >> 2) & 3, x2 = 2 * (2 * (G & 1) + h);
        const float ds = __fmul_rn(__half2float(*reinterpret_cast<const __half *>(unit)), (float)(int8_t)unit[kQ6kScales + (i0 >> 4)]);
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const uint32_t lo = (*reinterpret_cast<const uint32_t *>(unit + kQ6kLow + 32 * (t + w) + 4 * G) >> (4 * h)) & 0x0F0F0F0Fu;
            const uint32_t hi = (*reinterpret_cast<const uint32_t *>(unit + kQ6kHigh + 16 * (t + w) + 4 * (G >> 1)) >> x2) & 0x03030303u;
            sbytes_to_f32((lo << 2) | (hi << 6), v + 4 * w);  // 4 (q - 32) as s8
        }
#pragma unroll
        for (int j = 0; j < N; ++j) v[j] = __fmul_rn(ds, v[j] * 0.25f);
    } else if constexpr (TYPE == ZQ_Q8_0 || TYPE == ZQ_Q4_0 || TYPE == ZQ_IQ4_NL) {
        const int blk = i0 >> 5, e = i0 & 31;
        const float d = __half2float(reinterpret_cast<const __half *>(unit)[blk]);
        const uint32_t *src = reinterpret_cast<const uint32_t *>(unit + (unit_quant_offset(TYPE, i0) & ~3));  // the second word is one piece (16 bytes) on
#pragma unroll
        for (int w = 0; w < W; ++w) {
            uint32_t a = src[4 * w];
            if constexpr (TYPE != ZQ_Q8_0) a = (a >> ((e >> 4) * 4)) & 0x0F0F0F0Fu;
            if constexpr (TYPE == ZQ_IQ4_NL) a = iq4nl_bytes(a);
            if constexpr (TYPE == ZQ_Q4_0) bytes_to_f32(a, v + 4 * w);
            else sbytes_to_f32(a, v + 4 * w);
        }
#pragma unroll
        for (int j = 0; j < N; ++j) v[j] = TYPE == ZQ_Q4_0 ? __fmul_rn(v[j] - 8.0f, d) : __fmul_rn(d, v[j]);
    } else {
#pragma unroll
        for (int j = 0; j < N; ++j) v[j] = decode_unit_element(TYPE, unit, i0 + j);
    }
}

// Calls `fn` with the tensor type as a compile-time constant.
template <class Fn> static int with_type(uint32_t type, zq_error *err, Fn fn) {
    switch (type) {
    case ZQ_Q4_K: return fn(std::integral_constant<uint32_t, ZQ_Q4_K>());
    case ZQ_Q5_K: return fn(std::integral_constant<uint32_t, ZQ_Q5_K>());
    case ZQ_Q6_K: return fn(std::integral_constant<uint32_t, ZQ_Q6_K>());
    case ZQ_Q8_0: return fn(std::integral_constant<uint32_t, ZQ_Q8_0>());
    case ZQ_Q4_0: return fn(std::integral_constant<uint32_t, ZQ_Q4_0>());
    case ZQ_IQ4_NL: return fn(std::integral_constant<uint32_t, ZQ_IQ4_NL>());
    case ZQ_Q5_0: return fn(std::integral_constant<uint32_t, ZQ_Q5_0>());
    case ZQ_Q5_1: return fn(std::integral_constant<uint32_t, ZQ_Q5_1>());
    case ZQ_Q3_K: return fn(std::integral_constant<uint32_t, ZQ_Q3_K>());
    case ZQ_IQ4_XS: return fn(std::integral_constant<uint32_t, ZQ_IQ4_XS>());
    default: return set_error(err, ZQ_ERR_UNSUPPORTED, "codec: unsupported GGUF type %u", type);
    }
}

// One warp per 256-weight unit: the packed bytes are read with coalesced loads, the index division is one per warp.  A lane
// holds 8 consecutive elements of a 16-bit output, and of an f32 output columns 4 lane .. + 3 of each half of the unit, so that
// every store of the warp is 512 contiguous bytes: with 8 f32 per lane each of its two stores wrote every other 16 bytes, and
// the half-written sectors, not HBM, set the pace (Q8_0 17408 x 5120 to f32: 93 -> 68 us, 6.6 TB/s).
template <uint32_t TYPE>
__global__ void __launch_bounds__(256) dequantize_kernel(const uint8_t *__restrict__ resident, size_t row_pitch, int unit_bytes, size_t total_rows, size_t cols, int units_per_row, const uint32_t *__restrict__ row_ids, size_t n_rows,
                                                         void *__restrict__ out, int out_dtype, uint32_t *status) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t total = n_rows * (size_t)units_per_row;
    for (size_t u = (size_t)blockIdx.x * 8 + warp; u < total; u += (size_t)gridDim.x * 8) {
        const size_t orow = u / (size_t)units_per_row;
        const int ur = (int)(u - orow * units_per_row);
        const size_t srow = row_ids ? row_ids[orow] : orow;
        if (srow >= total_rows) {  // bad row id: record and skip, never read out of bounds
            if (lane == 0) atomicMax(status, (uint32_t)kStatusBadIndex);
            continue;
        }
        const uint8_t *unit = resident + srow * row_pitch + (size_t)ur * unit_bytes;
        const size_t u0 = (size_t)ur * kUnitWeights, o0 = orow * cols + u0;
        if (out_dtype == ZQ_F32) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i0 = 128 * h + 4 * lane;
                if (u0 + i0 >= cols) break;  // columns are a multiple of 32: all four elements or none
                float v[4];
                decode_run<TYPE>(unit, i0, v);
                *reinterpret_cast<float4 *>(reinterpret_cast<float *>(out) + o0 + i0) = make_float4(v[0], v[1], v[2], v[3]);
            }
        } else {
            if (u0 + 8 * lane >= cols) continue;  // all eight elements or none
            float v[8];
            decode_run<TYPE>(unit, 8 * lane, v);
            const size_t o = o0 + 8 * lane;
            uint32_t h[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (out_dtype == ZQ_F16) {
                    h[j] = h2_as_u32(__floats2half2_rn(v[2 * j], v[2 * j + 1]));
                } else {
                    const __nv_bfloat162 p = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
                    h[j] = *reinterpret_cast<const uint32_t *>(&p);
                }
            }
            uint16_t *dst = reinterpret_cast<uint16_t *>(out) + o;
            if ((reinterpret_cast<uintptr_t>(out) & 15) == 0) {
                *reinterpret_cast<uint4 *>(dst) = make_uint4(h[0], h[1], h[2], h[3]);
            } else {  // a caller's odd buffer: rows are whole 64-byte multiples, so only the base can be off
#pragma unroll
                for (int j = 0; j < 8; ++j) dst[j] = (uint16_t)(h[j >> 1] >> (16 * (j & 1)));
            }
        }
    }
}

// Packed rows -> f16 [rows, cols]: the operand pass of the prefill GEMM.  Each value is the codec's f32 value rounded
// once (zq_gemm_dq.cuh forms the same bits).  Up to kDequantBatch matrices of one type and shape
// per launch (MoE prefill dequantises the experts of a chunk together).  One warp per 256-weight unit, 8 consecutive elements per lane: the
// unit's packed bytes are read once with coalesced loads, the 512 output bytes are one coalesced store, and the only
// index division is one per warp.  `paired`: the rows alternate with those of another matrix, 16 by 16.
constexpr int kDequantBatch = 96;
struct DequantBatch {
    const uint8_t *src[kDequantBatch];
    __half *dst[kDequantBatch];
};

template <uint32_t TYPE>
__global__ void __launch_bounds__(256) dequantize_f16_batch_kernel(const __grid_constant__ DequantBatch batch, size_t row_pitch, int unit_bytes, int rows, int cols, int units_per_row, bool paired) {
    const uint8_t *resident = batch.src[blockIdx.y];
    __half *out = batch.dst[blockIdx.y];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int total_units = rows * units_per_row;
    for (int u = blockIdx.x * 8 + warp; u < total_units; u += gridDim.x * 8) {
        const int row = u / units_per_row, ur = u - row * units_per_row;
        const int k0 = ur * kUnitWeights + 8 * lane;
        if (k0 >= cols) continue;  // padded tail of the last unit (cols is a multiple of 32, so all 8 or none)
        float v[8];
        decode_run<TYPE>(resident + (size_t)row * row_pitch + (size_t)ur * unit_bytes, 8 * lane, v);
        uint4 packed;
        packed.x = h2_as_u32(__floats2half2_rn(v[0], v[1]));
        packed.y = h2_as_u32(__floats2half2_rn(v[2], v[3]));
        packed.z = h2_as_u32(__floats2half2_rn(v[4], v[5]));
        packed.w = h2_as_u32(__floats2half2_rn(v[6], v[7]));
        *reinterpret_cast<uint4 *>(out + (size_t)(paired ? row + (row & ~15) : row) * cols + k0) = packed;
    }
}

// weights[i] -> outs[i], all of one type and shape.
int launch_dequantize_f16_batch(zq_ctx *ctx, const zq_weight *const *weights, __half *const *outs, size_t count, zq_error *err, bool paired) {
    for (size_t first = 0; first < count; first += kDequantBatch) {
        const size_t n = count - first < (size_t)kDequantBatch ? count - first : (size_t)kDequantBatch;
        const zq_weight *w0 = weights[first];
        if (w0->cols % 8) return set_error(err, ZQ_ERR_SHAPE, "f16 operand pass needs columns aligned to 8, got %zu", w0->cols);
        DequantBatch batch;
        for (size_t i = 0; i < n; ++i) {
            const zq_weight *w = weights[first + i];
            if (w->type != w0->type || w->rows != w0->rows || w->cols != w0->cols) return set_error(err, ZQ_ERR_SHAPE, "batched dequantisation needs matrices of one type and shape");
            batch.src[i] = w->data;
            batch.dst[i] = outs[first + i];
        }
        const FormatInfo f = format_info(w0->type);
        const size_t units = w0->rows * w0->units_per_row;
        size_t bx = (units + 7) / 8;
        const size_t cap = ((size_t)ctx->sm_count * 64 + n - 1) / n;  // enough blocks in total to fill the machine a few times over
        if (bx > cap) bx = cap;
        if (bx == 0) bx = 1;
        const int rc = with_type(w0->type, err, [&](auto t) {
            dequantize_f16_batch_kernel<decltype(t)::value><<<dim3((unsigned)bx, (unsigned)n), 256, 0, ctx->stream>>>(batch, w0->row_pitch, f.unit_bytes, (int)w0->rows, (int)w0->cols, (int)w0->units_per_row, paired);
            return ZQ_OK;
        });
        if (rc) return rc;
        ctx->launches++;
        ZQ_CUDA_CHECK(cudaGetLastError(), err);
    }
    return ZQ_OK;
}

int launch_dequantize_f16(zq_ctx *ctx, const zq_weight *w, __half *out, zq_error *err, bool paired) {
    if (w->rows == 0 || w->cols == 0) return ZQ_OK;
    return launch_dequantize_f16_batch(ctx, &w, &out, 1, err, paired);
}

int launch_dequantize(zq_ctx *ctx, const zq_weight *w, const uint32_t *row_ids, size_t n_rows, void *out, int out_dtype, zq_error *err) {
    const size_t total = n_rows * w->units_per_row;
    if (total == 0) return ZQ_OK;
    size_t blocks = (total + 7) / 8;
    if (blocks > (size_t)ctx->sm_count * 64) blocks = (size_t)ctx->sm_count * 64;
    const FormatInfo f = format_info(w->type);
    const int rc = with_type(w->type, err, [&](auto t) {
        dequantize_kernel<decltype(t)::value><<<(unsigned)blocks, 256, 0, ctx->stream>>>(w->data, w->row_pitch, f.unit_bytes, w->rows, w->cols, (int)w->units_per_row, row_ids, n_rows, out, out_dtype, ctx->status_dev);
        return ZQ_OK;
    });
    if (rc) return rc;
    ctx->launches++;
    ZQ_CUDA_CHECK(cudaGetLastError(), err);
    return ZQ_OK;
}

// ---------------------------------------------------------------------------------------------------------------
// Encoders (GGUF layout out).
// ---------------------------------------------------------------------------------------------------------------

__device__ __forceinline__ float f16_round(float v) { return __half2float(__float2half_rn(v)); }
__device__ __forceinline__ float clampf(float v, float lo, float hi) { return v < lo ? lo : (v > hi ? hi : v); }

// Codes of 32 values under one scale: clamp(round half away from zero((v + shift) / scale), 0, 15), four codes per word.
// The IEEE division is only needed where the quotient is within its own error of a rounding boundary.  t = shifted * inv with
// inv = 1 / scale within 2 ulp is off by less than 4e-6 up to the largest code, the division by less than 1e-6, so a t further
// than 2e-5 from a half-integer rounds the same; a larger t clamps the same.  t is rounded by adding 1.5 * 2^23 (the code is
// then the low bits of the sum) and the distance to the rounded value is collected over the 32 values (max.NaN keeps a NaN or an
// infinite quotient), so the fast path takes 8 instructions a value and one test a group; about 1 group in 800 is done again.
__device__ __forceinline__ float max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void q4k_codes(const float (&v)[32], float scale, float shift, uint32_t (&q)[8]) {
    constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23
    const float inv = __fdividef(1.0f, scale);
    float off = 0.0f;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        uint32_t u[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float shifted = __fadd_rn(v[4 * w + j], shift);
            const float up = __fmaf_rn(shifted, inv, kMagic);
            off = max_nan(off, fabsf(__fmaf_rn(shifted, inv, -__fsub_rn(up, kMagic))));
            u[j] = __float_as_uint(fminf(fmaxf(up, kMagic), kMagic + 15.0f));
        }
        q[w] = __byte_perm(__byte_perm(u[0], u[1], 0x0040), __byte_perm(u[2], u[3], 0x0040), 0x5410);
    }
    if (!(off < 0.5f - 2e-5f)) {
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            q[w] = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) q[w] |= (uint32_t)clampf(roundf(__fdiv_rn(__fadd_rn(v[4 * w + j], shift), scale)), 0.0f, 15.0f) << (8 * j);
        }
    }
}

// encode_q4_k: a lane holds one group of 32 values, eight lanes a super-block, a warp four super-blocks; same operations in f32
// as the reference per value and per group (f16 rounding of d and dmin, round-half-away-from-zero codes), so the bytes are the
// reference's.  Bound by HBM (4 bytes in, 0.56 out per value).  Why a group per lane: with eight values per lane the work per
// group and per super-block was repeated by 4 and 32 lanes and the kernel was bound by issue (124 us for 17408 x 5120; this
// form 78 us, 5.2 TB/s).  Values arrive coalesced by cp.async, two tiles of 4 KB per warp in flight, at the chunk position
// c ^ (group & 7), which keeps both the arriving 16-byte chunks and a lane's reads of its own 128 bytes free of bank conflicts.
// VEC: values and blocks are 16-byte aligned (a block is 144 bytes, so every block then is).
// Super-blocks are taken from the last to the first: what wrote the values (a dequantisation, usually) wrote the last of them last, and
// some of those need not come back from HBM.  It is worth no more than runs differ by: 17408 x 5120 (356 MB of values) behind a dequantisation,
// four comparisons, 150.9 -> 148.2, 151.8 -> 151.1, 150.0 -> 148.0 and 150.7 -> 151.5 us for both.
constexpr int kEncWarps = 8, kEncTile = 4 * 1024;  // warps per CTA; bytes of a warp's tile (four super-blocks of f32)
constexpr int kEncSmem = kEncWarps * 2 * kEncTile;
template <bool VEC>
__global__ void __launch_bounds__(kEncWarps * 32) quantize_q4_k_kernel(const float *__restrict__ values, uint8_t *__restrict__ out, size_t blocks) {
    extern __shared__ __align__(128) uint8_t enc_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane & 7;
    const uint32_t tiles = smem_u32(enc_smem) + (uint32_t)(warp * 2 * kEncTile);
    const size_t step = (size_t)gridDim.x * kEncWarps * 4, end = (blocks + 3) & ~size_t(3);
    auto fetch = [&](size_t b0, uint32_t tile) {  // super-blocks b0 .. b0 + 3 of this warp
#pragma unroll
        for (int i = 0; i < 8; ++i) {  // 16-byte chunk i * 32 + lane: chunk lane & 7 of group 4 i + lane / 8
            const int group = 4 * i + (lane >> 3);
            const uint32_t dst = tile + (uint32_t)(group * 128 + ((sub ^ (group & 7)) * 16));
            if (b0 + (i >> 1) < blocks) {
                const float *src = values + b0 * 256 + (size_t)(i * 32 + lane) * 4;
                if (VEC) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
                else asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "f"(src[0]), "f"(src[1]), "f"(src[2]), "f"(src[3]) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    size_t turn = ((size_t)blockIdx.x * kEncWarps + warp) * 4;
    if (turn < end) fetch(end - 4 - turn, tiles);
    for (int buf = 0; turn < end; turn += step, buf ^= 1) {  // warp-uniform
        const size_t b0 = end - 4 - turn;
        if (turn + step < end) fetch(b0 - step, tiles + (uint32_t)((buf ^ 1) * kEncTile));
        else asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        const uint32_t row = tiles + (uint32_t)(buf * kEncTile + lane * 128);
        const bool live = b0 + (lane >> 3) < blocks;
        float v[32];
#pragma unroll
        for (int c = 0; c < 8; ++c)
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[4 * c]), "=f"(v[4 * c + 1]), "=f"(v[4 * c + 2]), "=f"(v[4 * c + 3]) : "r"(row + (uint32_t)((c ^ sub) * 16)) : "memory");
        __syncwarp();  // every lane has its values: the tile may be filled again
        float minimum = INFINITY, maximum = -INFINITY;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            minimum = fminf(minimum, v[j]);
            maximum = fmaxf(maximum, v[j]);
        }
        const float group_min = fmaxf(-minimum, 0.0f);
        const float group_scale = __fdiv_rn(fmaxf(__fadd_rn(maximum, group_min), 0.0f), 15.0f);
        float max_scale = fmaxf(group_scale, 0.0f), max_min = fmaxf(group_min, 0.0f);
#pragma unroll
        for (int s = 1; s <= 4; s <<= 1) {
            max_scale = fmaxf(max_scale, __shfl_xor_sync(0xffffffffu, max_scale, s));
            max_min = fmaxf(max_min, __shfl_xor_sync(0xffffffffu, max_min, s));
        }
        const __half dh = __float2half_rn(__fdiv_rn(max_scale, 63.0f)), dmh = __float2half_rn(__fdiv_rn(max_min, 63.0f));
        const float d = __half2float(dh), dmin = __half2float(dmh);
        const uint32_t sc = d == 0.0f ? 0 : (uint8_t)clampf(roundf(__fdiv_rn(group_scale, d)), 0.0f, 63.0f);
        const uint32_t mc = dmin == 0.0f ? 0 : (uint8_t)clampf(roundf(__fdiv_rn(group_min, dmin)), 0.0f, 63.0f);
        // header: byte g of the three scale words comes from groups g and g + 4 (lanes g and g + 4 of the eight)
        const uint32_t sc4 = __shfl_down_sync(0xffffffffu, sc, 4), mc4 = __shfl_down_sync(0xffffffffu, mc, 4);
        const int sh = 8 * (lane & 3);
        uint32_t w1 = ((sc & 0x3fu) | ((sc4 >> 4) << 6)) << sh, w2 = ((mc & 0x3fu) | ((mc4 >> 4) << 6)) << sh, w3 = ((sc4 & 0x0fu) | ((mc4 & 0x0fu) << 4)) << sh;
#pragma unroll
        for (int s = 1; s <= 2; s <<= 1) {
            w1 |= __shfl_xor_sync(0xffffffffu, w1, s);
            w2 |= __shfl_xor_sync(0xffffffffu, w2, s);
            w3 |= __shfl_xor_sync(0xffffffffu, w3, s);
        }
        const uint32_t w0 = (uint32_t)__half_as_ushort(dh) | ((uint32_t)__half_as_ushort(dmh) << 16);
        const float scale = __fmul_rn(d, (float)sc), shift = __fmul_rn(dmin, (float)mc);
        uint32_t q[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if (scale != 0.0f) q4k_codes(v, scale, shift, q);
        // the codes of an odd group are the high nibbles of the even group's bytes: the even lane stores bytes 0..15 of the pair's
        // 32, the odd lane bytes 16..31
        const bool odd = lane & 1;
        uint32_t o[4];
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? q[w] : q[4 + w], 1);
            o[w] = odd ? (got | (q[4 + w] << 4)) : (q[w] | (got << 4));
        }
        if (!live) continue;  // no shuffle below
        uint8_t *block = out + (b0 + (lane >> 3)) * 144, *dst = block + 16 + 16 * sub;
        if (VEC) {
            if (sub == 0) *reinterpret_cast<uint4 *>(block) = make_uint4(w0, w1, w2, w3);
            *reinterpret_cast<uint4 *>(dst) = make_uint4(o[0], o[1], o[2], o[3]);
        } else {
            const uint32_t hw[4] = {w0, w1, w2, w3};
            for (int j = 0; j < 16; ++j) {
                if (sub == 0) block[j] = (uint8_t)(hw[j >> 2] >> (8 * (j & 3)));
                dst[j] = (uint8_t)(o[j >> 2] >> (8 * (j & 3)));
            }
        }
    }
}

// Round-to-nearest encoders for the 32-weight block types (synthetic-input generators; the reference has none).
//   Q8_0:   d = f16(max|v| / 127), q = rint(v / d)
//   Q4_0:   d = f16(v_at_max_abs / -8), code = nearest of -8..7 to v / d
//   IQ4_NL: d = f16(v_at_max_abs / -127), code = nearest codebook entry to v / d
__global__ void quantize_block32_kernel(uint32_t type, const float *__restrict__ values, uint8_t *__restrict__ out, size_t blocks) {
    size_t b = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= blocks) return;
    const float *v = values + b * 32;
    float amax = 0.0f, smax = 0.0f;
    for (int i = 0; i < 32; ++i) {
        float a = fabsf(v[i]);
        if (a > amax) { amax = a; smax = v[i]; }
    }
    if (type == ZQ_Q8_0) {
        uint8_t *block = out + b * 34;
        float d = f16_round(__fdiv_rn(amax, 127.0f));
        float inv = d > 0.0f ? __fdiv_rn(1.0f, d) : 0.0f;
        __half dh = __float2half_rn(d);
        reinterpret_cast<uint16_t *>(block)[0] = __half_as_ushort(dh);
        for (int i = 0; i < 32; ++i) block[2 + i] = (uint8_t)(int8_t)clampf(rintf(__fmul_rn(v[i], inv)), -127.0f, 127.0f);
        return;
    }
    uint8_t *block = out + b * 18;
    float d = f16_round(__fdiv_rn(smax, type == ZQ_Q4_0 ? -8.0f : -127.0f));
    float inv = d != 0.0f ? __fdiv_rn(1.0f, d) : 0.0f;
    __half dh = __float2half_rn(d);
    reinterpret_cast<uint16_t *>(block)[0] = __half_as_ushort(dh);
    uint8_t codes[32];
    for (int i = 0; i < 32; ++i) {
        float s = __fmul_rn(v[i], inv);
        int best = 0;
        float best_err = INFINITY;
        for (int c = 0; c < 16; ++c) {
            float target = type == ZQ_Q4_0 ? (float)(c - 8) : (float)kIq4nlValues[c];
            float e = fabsf(__fsub_rn(s, target));
            if (e < best_err) { best_err = e; best = c; }
        }
        codes[i] = (uint8_t)best;
    }
    for (int i = 0; i < 16; ++i) block[2 + i] = (uint8_t)(codes[i] | (codes[i + 16] << 4));
}

int launch_quantize(zq_ctx *ctx, uint32_t type, const float *values, size_t rows, size_t cols, void *out, zq_error *err) {
    FormatInfo f = format_info(type);
    size_t blocks = rows * cols / f.block_elems;
    if (blocks == 0) return ZQ_OK;
    int threads = 128;
    unsigned grid = (unsigned)((blocks + threads - 1) / threads);
    if (type == ZQ_Q4_K) {
        size_t ctas = (blocks + 4 * kEncWarps - 1) / (4 * kEncWarps);
        if (ctas > (size_t)ctx->sm_count * 3) ctas = (size_t)ctx->sm_count * 3;  // three CTAs of 64 KB fit an SM; they walk the tensor
        const bool vec = ((reinterpret_cast<uintptr_t>(values) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
        auto kernel = vec ? quantize_q4_k_kernel<true> : quantize_q4_k_kernel<false>;
        ZQ_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kEncSmem), err);
        kernel<<<(unsigned)ctas, kEncWarps * 32, kEncSmem, ctx->stream>>>(values, reinterpret_cast<uint8_t *>(out), blocks);
    } else quantize_block32_kernel<<<grid, threads, 0, ctx->stream>>>(type, values, reinterpret_cast<uint8_t *>(out), blocks);
    ctx->launches++;
    ZQ_CUDA_CHECK(cudaGetLastError(), err);
    return ZQ_OK;
}

}  // namespace zq
