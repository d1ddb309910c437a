// fused_indexer_q_rope_quant: the sparse-indexer prologue that runs beside the attention prologue -
// GPT-J RoPE on the last rot_dim values of every index-q head (rounded to bf16), then either
//   FP8:   one power-of-two scale per (token, head), e4m3 values, scale folded into the head weight, or
//   MXFP4: one UE8M0 scale per 32 values, e2m1 values packed two per byte (cvt.rn.satfinite.e2m1x2.f32,
//          an sm_100 instruction), weights scaled by softmax_scale*head_scale only.
// Reference: src/flaggems_vllm/ops/fused_indexer_q_rope_quant.py:69-410 and its torch statement
// tests/test_fused_indexer_q_rope_quant.py:48-113.
// Three kernels: of the DeepSeek-V4 geometry (128 = 64 + 64) a warp walks several heads of one token, 4 lanes a head; other
// geometries with a rotary tail on a multiple of 8 values take head_dim/8 lanes per (token, head) row, 16 bytes per lane; any
// other takes one warp per row, where lane l keeps E = head_dim/32 consecutive values (E/2 rotary pairs).
#include "dsv4_common.cuh"

namespace dsv4 {
namespace {

struct IndexerQParams {
    const int64_t* positions;
    const uint8_t* q;  // bf16 [T, H, D], element strides
    int64_t q_stride0, q_stride1;
    const uint8_t* cos_sin;  // [max_pos, rot_dim] fp32 or bf16, row stride in elements
    int64_t cos_sin_stride;
    int32_t cos_sin_bf16, rot_dim;
    uint8_t* out;  // fp8: [T, H, D] bytes; fp4: [T, H, D/2] bytes (strides in bytes)
    int64_t out_stride0, out_stride1;
    uint8_t* scales;  // fp4 only: [T, H, D/32] bytes
    int64_t scale_stride0, scale_stride1;
    const uint8_t* weights;  // [T, H], row stride in elements; dtype code 0 bf16, 1 fp16, 2 fp32
    int64_t weights_stride;
    int32_t weights_dtype;
    float* weights_out;  // fp32 [T, H], row stride in elements
    int64_t weights_out_stride;
    float softmax_scale, head_scale;
    int64_t num_tokens;
    int32_t num_heads;
    uint32_t heads_mul, heads_shift;
    float minus_zero;  // -0.0f: see rotate_two()
    int32_t scales_word_aligned;  // fp4: every head's group of scale bytes starts on a 4-byte boundary
};

__device__ __forceinline__ float weight_value(uint32_t bits, int dtype) {
    if (dtype == 2) return __uint_as_float(bits);
    if (dtype == 0) return bf16_lo(bits);
    float f;
    asm("{.reg .f16 t; mov.b16 t, %1; cvt.f32.f16 %0, t;}" : "=f"(f) : "h"(static_cast<uint16_t>(bits)));
    return f;
}

__device__ __forceinline__ float load_weight(const uint8_t* base, int64_t idx, int dtype) {
    return weight_value(dtype == 2 ? reinterpret_cast<const uint32_t*>(base)[idx] : reinterpret_cast<const uint16_t*>(base)[idx], dtype);
}

// UE8M0 byte of an MXFP4 block whose absolute maximum is `amax`: ceil(log2(max(amax, 6*2^-126) / 6)) + 127 clamped to
// [0, 254], without the division: 6 = 1.5 * 4, so with the clamped maximum m * 2^(E-127), 1 <= m < 2, the quotient is
// below, at or above 2^(E-129) for m below, at or above 1.5.  Equal to the log2/ceil statement for every bf16
// maximum (a CPU test enumerates them).
__device__ __forceinline__ uint32_t mxfp4_code(float amax) {
    const uint32_t u = __float_as_uint(fmaxf(amax, 6.0f * 1.17549435e-38f));
    const uint32_t code = (u >> 23) - 2u + ((u & 0x7fffffu) > 0x400000u ? 1u : 0u);
    return code > 254u ? 254u : code;
}

// Two floats -> one byte of two e2m1 codes (lo in bits 0-3), round to nearest even, saturating at +-6.
__device__ __forceinline__ uint32_t pack_e2m1x2(float lo, float hi) {
    uint32_t r;
    asm("{.reg .b8 t; cvt.rn.satfinite.e2m1x2.f32 t, %1, %2; cvt.u32.u8 %0, t;}" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

// Four packed bf16 pairs times 2^(127 - code), the factor given as bf16 -> one word of eight e2m1 codes (element 0 in bits 0-3),
// round to nearest even, saturating at +-6.  Exact before the conversion (scaled_pair()).
__device__ __forceinline__ uint32_t pack_e2m1x8(const uint4& v, uint16_t factor) {
    const float2 x0 = scaled_pair(v.x, factor), x1 = scaled_pair(v.y, factor), x2 = scaled_pair(v.z, factor), x3 = scaled_pair(v.w, factor);
    uint32_t r;
    asm("{.reg .b8 t0, t1, t2, t3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 t0, %2, %1;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 t1, %4, %3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 t2, %6, %5;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 t3, %8, %7;\n\t"
        "mov.b32 %0, {t0, t1, t2, t3};}"
        : "=r"(r)
        : "f"(x0.x), "f"(x0.y), "f"(x1.x), "f"(x1.y), "f"(x2.x), "f"(x2.y), "f"(x3.x), "f"(x3.y));
    return r;
}

// mxfp4_code() of the two magnitudes in a bf16 pair, in 16-bit fields: a mantissa above 0x40 (1.5) is one that carries into the
// exponent when 0x3f is added.  The floor of the maximum is a bf16 value, 0x01c0 (a NaN becomes it, as in fmaxf).
__device__ __forceinline__ uint32_t mxfp4_codes(uint32_t magnitudes) {
    return ((max_bf16x2(magnitudes, 0x01c001c0u) + 0x003f003fu) >> 7 & 0x01ff01ffu) - 0x00020002u;
}

// Rotation of two pairs: separately rounded products, then the sums, two values an instruction.  A product is fma(., ., -0) with a
// -0 that comes from the launch's arguments: mul.rn.f32x2, or a -0 the assembler knows, it joins with the sum behind it, and a
// few values in 10^6 then differ.
__device__ __forceinline__ uint64_t f32x2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void rotate_two(uint32_t first, uint32_t second, uint64_t c, uint64_t s, uint64_t zero, uint32_t* to) {
    const uint64_t e = f32x2(bf16_lo(first), bf16_lo(second)), o = f32x2(bf16_hi(first), bf16_hi(second));
    uint64_t even, odd;
    asm("{.reg .b64 a, b, d, f;\n\t"
        "fma.rn.f32x2 a, %2, %4, %6;\n\t"
        "fma.rn.f32x2 b, %3, %5, %6;\n\t"
        "fma.rn.f32x2 d, %3, %4, %6;\n\t"
        "fma.rn.f32x2 f, %2, %5, %6;\n\t"
        "sub.rn.f32x2 %0, a, b;\n\t"
        "add.rn.f32x2 %1, d, f;}"
        : "=l"(even), "=l"(odd)
        : "l"(e), "l"(o), "l"(c), "l"(s), "l"(zero));
    asm("{.reg .f32 a, b, d, f;\n\t"
        "mov.b64 {a, b}, %2;\n\t"
        "mov.b64 {d, f}, %3;\n\t"
        "cvt.rn.bf16x2.f32 %0, d, a;\n\t"
        "cvt.rn.bf16x2.f32 %1, f, b;}"
        : "=r"(to[0]), "=r"(to[1])
        : "l"(even), "l"(odd));
}

template <int E>
__device__ __forceinline__ void load_row(const uint8_t* p, float (&x)[E]) {
    if (E == 2) {
        const uint32_t v = *reinterpret_cast<const uint32_t*>(p);
        x[0] = bf16_lo(v), x[1] = bf16_hi(v);
    } else if (E == 4) {
        const uint2 v = *reinterpret_cast<const uint2*>(p);
        x[0] = bf16_lo(v.x), x[1] = bf16_hi(v.x), x[2] = bf16_lo(v.y), x[3] = bf16_hi(v.y);
    } else {
        const uint4 v = *reinterpret_cast<const uint4*>(p);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) x[2 * i] = bf16_lo(w[i]), x[2 * i + 1] = bf16_hi(w[i]);
    }
}

template <int WARPS, int E, bool FP4>
__global__ void __launch_bounds__(WARPS * 32) indexer_q_rope_quant_kernel(const Launched<IndexerQParams> p) {
    begin_dependent_kernel();
    constexpr int D = 32 * E;
    const int lane = threadIdx.x & 31;
    const uint32_t row = blockIdx.x * WARPS + (threadIdx.x >> 5);
    if (row >= static_cast<uint32_t>(p.num_tokens) * static_cast<uint32_t>(p.num_heads)) return;
    const uint32_t t = fast_div(row, p.heads_mul, p.heads_shift);
    const int h = static_cast<int>(row - t * static_cast<uint32_t>(p.num_heads));
    float x[E];
    load_row<E>(p.q + (static_cast<int64_t>(t) * p.q_stride0 + h * p.q_stride1 + lane * E) * 2, x);
    const int first_rot = lane * E - (D - p.rot_dim);  // index of this lane's first value inside the rotary tail
    if (first_rot >= 0) {
        const int64_t pos = p.positions[t];
        const int half = p.rot_dim >> 1;
#pragma unroll
        for (int j = 0; j < E / 2; ++j) {
            const int pair = (first_rot >> 1) + j;
            float c, s;
            if (p.cos_sin_bf16) {
                const uint16_t* cs = reinterpret_cast<const uint16_t*>(p.cos_sin) + pos * p.cos_sin_stride;
                c = bf16_lo(cs[pair]), s = bf16_lo(cs[half + pair]);
            } else {
                const float* cs = reinterpret_cast<const float*>(p.cos_sin) + pos * p.cos_sin_stride;
                c = cs[pair], s = cs[half + pair];
            }
            const float e = x[2 * j], o = x[2 * j + 1];
            // separately rounded products, then the bf16 round trip the reference makes before quantising
            const uint32_t packed = pack_bf16x2(__fsub_rn(__fmul_rn(e, c), __fmul_rn(o, s)),
                                                __fadd_rn(__fmul_rn(o, c), __fmul_rn(e, s)));
            x[2 * j] = bf16_lo(packed), x[2 * j + 1] = bf16_hi(packed);
        }
    }
    float amax = 0.0f;
#pragma unroll
    for (int i = 0; i < E; ++i) amax = fmaxf(amax, fabsf(x[i]));
    uint8_t* out = p.out + static_cast<int64_t>(t) * p.out_stride0 + h * p.out_stride1;
    float weight_factor = 1.0f;
    if (FP4) {
        constexpr int kGroupLanes = 32 / E;  // lanes per block of 32 values
#pragma unroll
        for (int m = 1; m < kGroupLanes; m <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, m));
        const uint32_t code = mxfp4_code(amax);
        const float inv = __uint_as_float((254u - code) << 23);  // code >= 1 because of the amax floor
        uint32_t bytes = 0;
#pragma unroll
        for (int j = 0; j < E / 2; ++j) bytes |= pack_e2m1x2(__fmul_rn(x[2 * j], inv), __fmul_rn(x[2 * j + 1], inv)) << (8 * j);
        if (E == 2) out[lane] = static_cast<uint8_t>(bytes);
        else if (E == 4) *reinterpret_cast<uint16_t*>(out + 2 * lane) = static_cast<uint16_t>(bytes);
        else *reinterpret_cast<uint32_t*>(out + 4 * lane) = bytes;
        if ((lane & (kGroupLanes - 1)) == 0)
            p.scales[static_cast<int64_t>(t) * p.scale_stride0 + h * p.scale_stride1 + lane / kGroupLanes] = static_cast<uint8_t>(code);
    } else {
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, m));
        const uint32_t code = ue8m0_code(amax);  // 2^ceil(log2(max(amax, 1e-4)/448))
        const float inv = __uint_as_float((254u - code) << 23);
        weight_factor = __uint_as_float(code << 23);
        float y[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < E; ++i) y[i] = __fmul_rn(x[i], inv);
        if (E == 2) *reinterpret_cast<uint16_t*>(out + 2 * lane) = static_cast<uint16_t>(pack_e4m3x4(y[0], y[1], 0.f, 0.f));
        else if (E == 4) *reinterpret_cast<uint32_t*>(out + 4 * lane) = pack_e4m3x4(y[0], y[1], y[2], y[3]);
        else st_global8(out + 8 * lane, make_uint2(pack_e4m3x4(y[0], y[1], y[2], y[3]), pack_e4m3x4(y[4], y[5], y[6], y[7])));
    }
    if (lane == 0) {
        float w = load_weight(p.weights, static_cast<int64_t>(t) * p.weights_stride + h, p.weights_dtype);
        if (!FP4) w = __fmul_rn(w, weight_factor);
        w = __fmul_rn(__fmul_rn(w, p.softmax_scale), p.head_scale);
        p.weights_out[static_cast<int64_t>(t) * p.weights_out_stride + h] = w;
    }
}

// Rows of 16-byte pieces: a row is D/8 lanes holding 8 values (16 bytes) each, so one warp instruction moves 32/G rows;
// U passes per warp are loaded before any is used.  Needs 16-byte aligned rows and a rotary tail that starts
// on a multiple of 8 values.
template <int WARPS, int G, int U, bool FP4>
__global__ void __launch_bounds__(WARPS * 32) indexer_q_rope_quant_rows_kernel(const Launched<IndexerQParams, 8> p, const int cs_vec4) {
    begin_dependent_kernel();
    constexpr int D = 8 * G, ROWS = 32 / G;
    const int lane = threadIdx.x & 31, sub = lane % G, slot = lane / G;
    const uint32_t total = static_cast<uint32_t>(p.num_tokens) * static_cast<uint32_t>(p.num_heads);
    const uint32_t base_row = (blockIdx.x * WARPS + (threadIdx.x >> 5)) * (U * ROWS) + slot;
    uint4 raw[U];
    uint32_t tok[U];
    bool live[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const uint32_t row = base_row + u * ROWS;
        live[u] = row < total;
        tok[u] = fast_div(live[u] ? row : 0u, p.heads_mul, p.heads_shift);
        raw[u] = make_uint4(0u, 0u, 0u, 0u);
        if (live[u]) {
            const int h = static_cast<int>(row - tok[u] * static_cast<uint32_t>(p.num_heads));
            raw[u] = ld_stream16(p.q + (static_cast<int64_t>(tok[u]) * p.q_stride0 + h * p.q_stride1 + 8 * sub) * 2);
        }
    }
    const int first_rot = 8 * sub - (D - p.rot_dim);
    const int half = p.rot_dim >> 1;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const uint32_t row = base_row + u * ROWS;
        const int h = static_cast<int>(row - tok[u] * static_cast<uint32_t>(p.num_heads));
        float x[8];
        unpack8(raw[u], x);
        if (live[u] && first_rot >= 0) {
            const int64_t pos = p.positions[tok[u]];
            const int pair0 = first_rot >> 1;
            float c[4], sn[4];
            if (cs_vec4) {
                const float* cs = reinterpret_cast<const float*>(p.cos_sin) + pos * p.cos_sin_stride;
                const float4 c4 = ld_readonly_f4(cs + pair0), s4 = ld_readonly_f4(cs + half + pair0);
                c[0] = c4.x, c[1] = c4.y, c[2] = c4.z, c[3] = c4.w, sn[0] = s4.x, sn[1] = s4.y, sn[2] = s4.z, sn[3] = s4.w;
            } else if (p.cos_sin_bf16) {
                const uint16_t* cs = reinterpret_cast<const uint16_t*>(p.cos_sin) + pos * p.cos_sin_stride;
#pragma unroll
                for (int j = 0; j < 4; ++j) c[j] = bf16_lo(cs[pair0 + j]), sn[j] = bf16_lo(cs[half + pair0 + j]);
            } else {
                const float* cs = reinterpret_cast<const float*>(p.cos_sin) + pos * p.cos_sin_stride;
#pragma unroll
                for (int j = 0; j < 4; ++j) c[j] = cs[pair0 + j], sn[j] = cs[half + pair0 + j];
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float e = x[2 * j], o = x[2 * j + 1];
                const uint32_t packed = pack_bf16x2(__fsub_rn(__fmul_rn(e, c[j]), __fmul_rn(o, sn[j])),
                                                    __fadd_rn(__fmul_rn(o, c[j]), __fmul_rn(e, sn[j])));
                x[2 * j] = bf16_lo(packed), x[2 * j + 1] = bf16_hi(packed);
            }
        }
        float amax = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(x[i]));
        uint8_t* out = p.out + static_cast<int64_t>(tok[u]) * p.out_stride0 + h * p.out_stride1;
        float weight_factor = 1.0f;
        if (FP4) {
#pragma unroll
            for (int m = 1; m < 4; m <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, m));
            const uint32_t code = mxfp4_code(amax);
            const float inv = __uint_as_float((254u - code) << 23);
            uint32_t bytes = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) bytes |= pack_e2m1x2(__fmul_rn(x[2 * j], inv), __fmul_rn(x[2 * j + 1], inv)) << (8 * j);
            if (live[u]) {
                *reinterpret_cast<uint32_t*>(out + 4 * sub) = bytes;
                if ((sub & 3) == 0)
                    p.scales[static_cast<int64_t>(tok[u]) * p.scale_stride0 + h * p.scale_stride1 + (sub >> 2)] = static_cast<uint8_t>(code);
            }
        } else {
#pragma unroll
            for (int m = 1; m < G; m <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, m));
            const uint32_t code = ue8m0_code(amax);
            const float inv = __uint_as_float((254u - code) << 23);
            weight_factor = __uint_as_float(code << 23);
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] = __fmul_rn(x[i], inv);
            if (live[u]) st_global8(out + 8 * sub, make_uint2(pack_e4m3x4(x[0], x[1], x[2], x[3]), pack_e4m3x4(x[4], x[5], x[6], x[7])));
        }
        if (live[u] && sub == 0) {
            float w = load_weight(p.weights, static_cast<int64_t>(tok[u]) * p.weights_stride + h, p.weights_dtype);
            if (!FP4) w = __fmul_rn(w, weight_factor);
            p.weights_out[static_cast<int64_t>(tok[u]) * p.weights_out_stride + h] = __fmul_rn(__fmul_rn(w, p.softmax_scale), p.head_scale);
        }
    }
}

template <int G>
cudaError_t launch_rows(const IndexerQParams& p, bool fp4, int64_t rows, int cs_vec4, cudaStream_t stream) {
    constexpr int WARPS = 4, U = 2, PER_CTA = WARPS * U * (32 / G);
    const unsigned grid = static_cast<unsigned>((rows + PER_CTA - 1) / PER_CTA);
    if (fp4) launch_dependent(indexer_q_rope_quant_rows_kernel<WARPS, G, U, true>, grid, WARPS * 32, stream, p, cs_vec4);
    else launch_dependent(indexer_q_rope_quant_rows_kernel<WARPS, G, U, false>, grid, WARPS * 32, stream, p, cs_vec4);
    return cudaGetLastError();
}

// The DeepSeek-V4 geometry (head_dim 128 = 64 un-rotated + 64 rotary): a warp owns `heads_per_task` consecutive heads of one token,
// eight at a time.  A head is 4 lanes; lane s keeps the un-rotated values [16s, 16s+16) and the rotary values [64+16s, 64+16s+16)
// (eight pairs), so every lane rotates (no divergence) and its eight cosines and sines are loaded once per task.  MXFP4 blocks of
// 32 are 2 lanes.  WIDE: 32-byte loads, otherwise (rows on 16-byte boundaries only) two of half the size.  Two passes are in
// flight: the loads of the next one go out before the current one is worked on.  PREFETCH: one instruction sends the rest of the
// task's rows to L2 at its start.
// Large batches are bound by HBM, smaller ones by instruction issue: a pass of eight heads with MXFP4 is 217 warp instructions.  For
// that, bf16 values are widened and scaled by one instruction each (scaled_pair()), two pairs are rotated at a time (rotate_two()), two
// sets of registers take turns, and weights and scale words are written for 32 heads at once.  Without these (345 instructions) -> with,
// 64 heads a token, us a launch from a graph, FP8 and MXFP4:
//   at full clock: 61 tokens 1.88 -> 1.71 and 1.94 -> 1.71; 1531 tokens 9.4 -> 8.0 and 9.2 -> 6.7; 9216 tokens 38.7 -> 36.4 and 36.9 -> 33.1;
//     16384 tokens 63.9 -> 61.4 (6.7 TB/s) and 64-67 -> 57-59 (6.0 TB/s); 65536 tokens 238-246 -> 235 (7.0 TB/s) and 230-235 -> 207-212
//   sustained, at the clock the power limit leaves: 16384 tokens 69.2 -> 65.2 and 65.5 -> 58.7; 65536 tokens 262 -> 244 and 250 -> 218
template <int WARPS, bool FP4, bool WIDE, bool PREFETCH, int CTAS = 6>
__global__ void __launch_bounds__(WARPS * 32, CTAS) indexer_q_rope_quant_heads_kernel(const Launched<IndexerQParams, 4 * sizeof(int)> p, const int heads_per_task, const uint32_t tasks_per_token,
                                                                                const uint32_t tpt_mul, const uint32_t tpt_shift) {
    const int lane = threadIdx.x & 31, sub = lane & 3, which = lane >> 2;
    const uint32_t task = blockIdx.x * WARPS + (threadIdx.x >> 5);
    const int64_t t = fast_div(task, tpt_mul, tpt_shift);
    if (t >= p.num_tokens) return;
    const int head_begin = static_cast<int>(task - static_cast<uint32_t>(t) * tasks_per_token) * heads_per_task;
    const int head_end = head_begin + heads_per_task < p.num_heads ? head_begin + heads_per_task : p.num_heads;
    const int64_t head_bytes = p.q_stride1 * 2;
    const uint8_t* row = p.q + t * p.q_stride0 * 2 + (head_begin + which) * head_bytes + 32 * sub;
    if (starts_early()) {
        // the lines of the first pass, one per lane
        if (lane < 16 && head_begin + (lane >> 1) < head_end) prefetch_line_l2(p.q + t * p.q_stride0 * 2 + (head_begin + (lane >> 1)) * head_bytes + 128 * (lane & 1));
        if (lane == 31) prefetch_line_l2(p.positions + t);
    }
    begin_dependent_kernel();
    const auto load32 = [](const uint8_t* from) {
        if (WIDE) return ld_stream32(from);
        Bytes32 v;
        v.lo = ld_stream16(from), v.hi = ld_stream16(from + 16);
        return v;
    };
    // Of 32 heads (four passes) a lane writes the weight of head 8 * sub + which, and with MXFP4 the scales of that head: one load, one
    // multiplication and one store for four passes instead of as many predicated ones, in every lane, in each.
    const int own = head_begin + 8 * sub + which;
    const auto weight_of = [&](int h) -> uint32_t {  // (its bits only: a conversion would wait for them)
        const int64_t at = t * p.weights_stride + h;
        if (h >= head_end) return 0u;
        return p.weights_dtype == 2 ? __ldg(reinterpret_cast<const uint32_t*>(p.weights) + at) : __ldg(reinterpret_cast<const uint16_t*>(p.weights) + at);
    };
    struct Rows {
        Bytes32 nope, rope;
    };
    Rows a, b;
    int h = head_begin + which;
    a.nope.lo = a.nope.hi = a.rope.lo = a.rope.hi = make_uint4(0u, 0u, 0u, 0u);
    if (h < head_end) a.nope = load32(row), a.rope = load32(row + 128);
    b = a;
    uint32_t weight_bits = weight_of(own);
    if (PREFETCH && lane == 0 && head_bytes == 256 && head_end > head_begin + 16)
        prefetch_l2(p.q + t * p.q_stride0 * 2 + (head_begin + 16) * 256, static_cast<uint32_t>(head_end - head_begin - 16) * 256u);
    const int64_t pos = p.positions[t];
    uint64_t c[4], sn[4];  // of two pairs each
    const uint64_t zero = f32x2(p.minus_zero, p.minus_zero);
    if (p.cos_sin_bf16) {
        const uint16_t* cs = reinterpret_cast<const uint16_t*>(p.cos_sin) + pos * p.cos_sin_stride + 8 * sub;
#pragma unroll
        for (int j = 0; j < 4; ++j) c[j] = f32x2(bf16_lo(cs[2 * j]), bf16_lo(cs[2 * j + 1])), sn[j] = f32x2(bf16_lo(cs[32 + 2 * j]), bf16_lo(cs[33 + 2 * j]));
    } else {
        const float* cs = reinterpret_cast<const float*>(p.cos_sin) + pos * p.cos_sin_stride + 8 * sub;
#pragma unroll
        for (int j = 0; j < 4; ++j) c[j] = f32x2(__ldg(cs + 2 * j), __ldg(cs + 2 * j + 1)), sn[j] = f32x2(__ldg(cs + 32 + 2 * j), __ldg(cs + 33 + 2 * j));
    }
    uint8_t* out = p.out + t * p.out_stride0 + (head_begin + which) * p.out_stride1;
    uint32_t kept = 0u;  // of the head this lane writes weight and scales of: its scale word (MXFP4) or its scale code (FP8)
    // What is written once for four passes, those up to `pass`.
    const auto finish = [&](int pass) {
        const int head = own + 8 * (pass & ~3);
        if (head >= head_end || sub > (pass & 3)) return;
        float w = weight_value(weight_bits, p.weights_dtype);
        if (FP4) {
            uint8_t* sc = p.scales + t * p.scale_stride0 + head * p.scale_stride1;
            if (p.scales_word_aligned) {
                *reinterpret_cast<uint32_t*>(sc) = kept;
            } else {
                sc[0] = static_cast<uint8_t>(kept), sc[1] = static_cast<uint8_t>(kept >> 8);
                sc[2] = static_cast<uint8_t>(kept >> 16), sc[3] = static_cast<uint8_t>(kept >> 24);
            }
        } else {
            w = __fmul_rn(w, __uint_as_float(kept << 23));
        }
        p.weights_out[t * p.weights_out_stride + head] = __fmul_rn(__fmul_rn(w, p.softmax_scale), p.head_scale);
    };
    // Pass `pass` on the rows in `now`, while the next ones are on their way to `then`; says whether there is another.
    const auto step = [&](int pass, const Rows& now, Rows& then) {
        row += 8 * head_bytes;
        if (h + 8 < head_end) then.nope = load32(row), then.rope = load32(row + 128);
        const Bytes32 &nope = now.nope, &rope = now.rope;
        uint32_t rot[8];  // the rotated pairs, rounded to bf16 as the reference does before quantising
        rotate_two(rope.lo.x, rope.lo.y, c[0], sn[0], zero, rot), rotate_two(rope.lo.z, rope.lo.w, c[1], sn[1], zero, rot + 2);
        rotate_two(rope.hi.x, rope.hi.y, c[2], sn[2], zero, rot + 4), rotate_two(rope.hi.z, rope.hi.w, c[3], sn[3], zero, rot + 6);
        const uint4 ra = make_uint4(rot[0], rot[1], rot[2], rot[3]), rb = make_uint4(rot[4], rot[5], rot[6], rot[7]);
        // |.| maxima on the packed words: of the un-rotated values in `pn`, of the rotated ones in `pr`
        const auto max16 = [](const uint4& x, const uint4& y) {
            return max_abs_bf16x2(max_abs_bf16x2(max_abs_bf16x2(x.x, x.y), max_abs_bf16x2(x.z, x.w)),
                                  max_abs_bf16x2(max_abs_bf16x2(y.x, y.y), max_abs_bf16x2(y.z, y.w)));
        };
        const uint32_t pn = max16(nope.lo, nope.hi), pr = max16(ra, rb);
        if (FP4) {
            // the two maxima side by side in one word, reduced over the 2 lanes of a block
            uint32_t both = max_abs_bf16x2(__byte_perm(pn, pr, 0x5410), __byte_perm(pn, pr, 0x7632)) & 0x7fff7fffu;
            both = max_bf16x2(both, __shfl_xor_sync(0xffffffffu, both, 1));
            const uint32_t codes = mxfp4_codes(both), factors = (0x00fe00feu - codes) << 7;  // 2^(127 - code) as bf16
            const auto fn = static_cast<uint16_t>(factors), fr = static_cast<uint16_t>(factors >> 16);
            const uint2 bn = make_uint2(pack_e2m1x8(nope.lo, fn), pack_e2m1x8(nope.hi, fn)), br = make_uint2(pack_e2m1x8(ra, fr), pack_e2m1x8(rb, fr));
            // the head's four scale bytes in one word: blocks (un-rotated 0-31, 32-63, rotated 0-31, 32-63)
            const uint32_t other = __shfl_xor_sync(0xffffffffu, codes, 2);
            if (sub == (pass & 3)) kept = sub & 2 ? other | (codes << 8) : codes | (other << 8);
            if (h < head_end) {
                st_global8(out + 8 * sub, bn);
                st_global8(out + 32 + 8 * sub, br);
            }
        } else {
            uint32_t pk = max_abs_bf16x2(pn, pr) & 0x7fff7fffu;
            pk = max_bf16x2(pk, __shfl_xor_sync(0xffffffffu, pk, 1));
            pk = max_bf16x2(pk, __shfl_xor_sync(0xffffffffu, pk, 2));
            const uint32_t code = ue8m0_code(fmaxf(bf16_lo(pk), bf16_hi(pk)));
            if (sub == (pass & 3)) kept = code;
            const uint2 n0 = quant8_pow2(nope.lo, code), n1 = quant8_pow2(nope.hi, code), r0 = quant8_pow2(ra, code), r1 = quant8_pow2(rb, code);
            if (h < head_end) {
                st_stream16(out + 16 * sub, make_uint4(n0.x, n0.y, n1.x, n1.y));
                st_stream16(out + 64 + 16 * sub, make_uint4(r0.x, r0.y, r1.x, r1.y));
            }
        }
        out += 8 * p.out_stride1, h += 8;
        return h - which < head_end;
    };
    int pass = 0;
    while (step(pass, a, b)) {
        const bool more = step(pass + 1, b, a);
        if (!more || (pass & 2)) finish(pass + 1);
        if (!more) return;
        pass += 2;
        if (!(pass & 2)) weight_bits = weight_of(own + 8 * pass);
    }
    finish(pass);
}

template <int E>
cudaError_t launch_e(const IndexerQParams& p, bool fp4, unsigned grid, cudaStream_t stream) {
    constexpr int WARPS = 8;
    if (fp4) launch_dependent(indexer_q_rope_quant_kernel<WARPS, E, true>, grid, WARPS * 32, stream, p);
    else launch_dependent(indexer_q_rope_quant_kernel<WARPS, E, false>, grid, WARPS * 32, stream, p);
    return cudaGetLastError();
}

// Heads per warp (a task: that many heads of one token, or what is left of them): few rows, short tasks, so that there are enough of them;
// many rows, long ones, whose set-up more heads share; and where tasks of 64 or 32 heads make one wave that is nearly full, those.
// FP8 / MXFP4, us a launch of 64 heads a token, from a graph with three inputs in rotation (from 3072 tokens on they come from HBM):
//   8 | 16           200 tokens  2.4 / 2.4 | 2.5 / 2.4         256 tokens  2.7 / 2.7 | 2.5 / 2.5
//   16 | 32 | 64      832 tokens  3.7 / 3.7 | 3.9 / 3.5 | 5.1 / 4.7        1280 tokens  5.7 / 5.6 | 5.8 / 5.5 | 6.1 / 6.0
//                    1536 tokens  6.8 / 6.2 | 6.1 / 5.8 | 7.5 / 6.9        1800 tokens  8.8 / 8.4 | 8.9 / 8.1 | 9.0 / 8.7
//                    2500 tokens 10.7 / 10.3 | 11.5 / 11.1 | 10.7 / 10.5   3072 tokens 13.4 / 12.9 | 12.6 / 12.2 | 12.0 / 11.7
//                    4096 tokens 18.1 / 17.0 | 18.2 / 17.0 | 19.9 / 18.4   8192 tokens 36.2 / 33.1 | 34.5 / 31.0 | 35.4 / 31.9
//   32 | prefetch    8192 tokens 34.5 / 31.0 | 34.0 / 31.4       9216 tokens 39.0 / 34.9 | 37.4 / 34.3     32768 tokens 127 / 113 | 121 / 109
// (With 64 at 5500 to 6500 tokens, nearly two waves of them, 3 % less than with 32.)
// Other numbers of heads: a short last task costs nearly a long one's place, so it is the number of tasks that decides, and tasks of one
// length are preferred.  16 | 32 | 64:
//    96 heads: 1979 tokens 14.3 / 13.3 | 14.0 / 12.8 | 17.7 / 16.4     75 heads: 2533 tokens 14.6 / 13.7 | 16.0 / 14.7 | 17.8 / 16.5
//    80 heads: 1125 tokens  7.3 / 6.4 | 7.0 / 6.0 | 9.0 / 8.1          1625 tokens 10.7 / 10.1 | 11.4 / 10.6 | 11.1 / 10.1
//    48 heads: 1875 tokens  7.3 / 6.4 | 8.5 / 7.6 | 8.4 / 7.7          3958 tokens 14.3 / 13.3 | 15.4 / 14.2 | 15.9 / 14.7
//              3437 tokens 12.3 / 11.3 | 12.7 / 11.6 | 11.7 / 10.6     5416 tokens 18.4 / 17.0 | 19.7 / 18.1 | 18.4 / 16.7
//             16000 tokens 49.7 / 45.0 | 46.4 / 42.1 | 47.4 / 43.2    56 heads: 5000 tokens 20.4 / 18.9 | 19.2 / 17.2 | 20.0 / 18.3
//    40 heads: 5520 tokens 16.8 / 15.8 | 17.6 / 16.3 | 15.9 / 14.4    14746 tokens 41.0 / 37.9 | 37.5 / 34.7 | 37.0 / 34.1
//    24 heads: 2500 tokens  5.3 / 5.1 | 5.0 / 4.6 | 5.0 / 4.6          6875 tokens 13.4 / 12.6 | 12.0 / 10.7 | 12.0 / 10.7
constexpr int kHeadsWarps = 4;                    // per CTA
constexpr int64_t kWave = 148 * 6 * kHeadsWarps;  // warps of a B200
constexpr int64_t kPrefetchRows = 589824;         // from here on a task sends the rest of its rows to L2 at its start
constexpr int heads_of_a_task(int64_t tokens, int heads) {
    const int64_t rows = tokens * heads;
    const auto one_length = [&](int n) { return heads <= n || heads % n == 0; };
    const auto fills = [&](int n, int64_t waves) {
        const int64_t tasks = tokens * ((heads + n - 1) / n);
        return tasks <= waves * kWave && 9 * tasks >= 7 * waves * kWave;
    };
    if (one_length(64) && fills(64, 1)) return 64;
    if (rows > kWave * 64) return heads > 32 && heads <= (rows >= kPrefetchRows ? 40 : 48) ? 64 : 32;
    if (fills(32, 1) || (one_length(32) && fills(32, 2))) return 32;
    if (rows < 14336) return 8;
    for (int n = 32; n <= 64 && !one_length(16); n *= 2)
        if (one_length(n) && 9 * rows >= 7 * kWave * n) return n;
    return 16;
}
static_assert(heads_of_a_task(223, 64) == 8 && heads_of_a_task(224, 64) == 16 && heads_of_a_task(1381, 64) == 16 && heads_of_a_task(1382, 64) == 32);
static_assert(heads_of_a_task(1777, 64) == 16 && heads_of_a_task(2763, 64) == 64 && heads_of_a_task(3552, 64) == 64 && heads_of_a_task(3553, 64) == 32);
static_assert(heads_of_a_task(1979, 96) == 32 && heads_of_a_task(2533, 75) == 16 && heads_of_a_task(4600, 48) == 16 && heads_of_a_task(1875, 48) == 16);
static_assert(heads_of_a_task(3437, 48) == 64 && heads_of_a_task(5416, 48) == 64 && heads_of_a_task(12289, 48) == 32 && heads_of_a_task(2250, 40) == 16 && heads_of_a_task(6500, 40) == 64);

// Heads per warp of the form with seven CTAs per SM (72 registers, 56 to 108 bytes a thread spilled), or 0 for that with six: seven where
// the tasks make one or two waves of seven and a little more than as many of six.  FP8 / MXFP4, us as above, six | seven:
//   16 heads, 1 wave:   64 heads, 889 tokens 4.3 / 4.1 | 4.8 / 4.6     950 tokens 5.2 / 4.8 | 4.9 / 4.6     1036 tokens 5.5 / 5.2 | 5.0 / 4.8
//                       16 heads, 4000 tokens 5.6 / 5.2 | 5.1 / 4.8    32 heads, 2000 tokens 5.5 / 5.2 | 5.0 / 4.7
//   32 heads, 1 wave:   64 heads, 1777 tokens 9.3 / 8.4 | 9.5 / 8.4    1850 tokens 10.3 / 9.6 | 9.5 / 8.6     2072 tokens 11.0 / 10.4 | 10.4 / 9.6
//             2 waves:  64 heads, 3553 tokens 16.4 / 15.0 | 16.4 / 14.9    3700 tokens 18.0 / 16.6 | 17.2 / 15.6     4144 tokens 19.3 / 17.6 | 18.6 / 16.8
// Rows on 16-byte boundaries spill more and gain with 16 heads only (64 heads, 1000 tokens 6.9 / 6.8 | 6.4 / 6.1; 1850 tokens 10.4 / 10.1 | 10.4 / 9.4;
// 3700 tokens 18.5 / 17.0 | 18.6 / 16.6).  Up to 8 heads a token are one pass a task, for which the spills do not pay (8000 tokens of 8 5.8 / 5.7 | 6.0 / 5.8).
constexpr int heads_with_seven_ctas(int64_t tokens, int heads, bool wide) {
    for (int n = wide ? 32 : 16; n >= 16 && heads > 8; n /= 2) {
        if (heads > n && n == 32 && heads % n != 0) continue;
        const int64_t tasks = tokens * ((heads + n - 1) / n);
        for (int waves = 1; waves <= (wide ? 2 : 1); ++waves)
            if (33 * tasks > 34 * waves * kWave && 6 * tasks <= 7 * waves * kWave) return n;
    }
    return 0;
}
static_assert(heads_with_seven_ctas(914, 64, true) == 0 && heads_with_seven_ctas(915, 64, false) == 16 && heads_with_seven_ctas(1036, 64, true) == 16 && heads_with_seven_ctas(1037, 64, true) == 0);
static_assert(heads_with_seven_ctas(1829, 64, true) == 0 && heads_with_seven_ctas(1830, 64, true) == 32 && heads_with_seven_ctas(1830, 64, false) == 0 && heads_with_seven_ctas(2072, 64, true) == 32);
static_assert(heads_with_seven_ctas(4000, 8, true) == 0 && heads_with_seven_ctas(4000, 16, false) == 16 && heads_with_seven_ctas(3660, 64, true) == 32 && heads_with_seven_ctas(4144, 64, true) == 32 && heads_with_seven_ctas(4145, 64, true) == 0);

}  // namespace

cudaError_t launch_indexer_q_rope_quant(const int64_t* positions, const void* q, int64_t q_stride0, int64_t q_stride1,
                                        const void* cos_sin, int64_t cos_sin_stride, int cos_sin_bf16, int rot_dim, void* out,
                                        int64_t out_stride0, int64_t out_stride1, void* scales, int64_t scale_stride0,
                                        int64_t scale_stride1, const void* weights, int64_t weights_stride, int weights_dtype,
                                        float* weights_out, int64_t weights_out_stride, float softmax_scale, float head_scale,
                                        int64_t num_tokens, int num_heads, int head_dim, int fp4, cudaStream_t stream) {
    const int64_t rows = num_tokens * num_heads;
    if (rows == 0) return cudaSuccess;
    if (rows >= (1LL << 31)) return cudaErrorInvalidConfiguration;
    IndexerQParams p{};
    p.positions = positions, p.q = static_cast<const uint8_t*>(q), p.q_stride0 = q_stride0, p.q_stride1 = q_stride1;
    p.cos_sin = static_cast<const uint8_t*>(cos_sin), p.cos_sin_stride = cos_sin_stride, p.cos_sin_bf16 = cos_sin_bf16;
    p.rot_dim = rot_dim, p.out = static_cast<uint8_t*>(out), p.out_stride0 = out_stride0, p.out_stride1 = out_stride1;
    p.scales = static_cast<uint8_t*>(scales), p.scale_stride0 = scale_stride0, p.scale_stride1 = scale_stride1;
    p.weights = static_cast<const uint8_t*>(weights), p.weights_stride = weights_stride, p.weights_dtype = weights_dtype;
    p.weights_out = weights_out, p.weights_out_stride = weights_out_stride;
    p.softmax_scale = softmax_scale, p.head_scale = head_scale, p.num_tokens = num_tokens, p.num_heads = num_heads, p.minus_zero = -0.0f;
    make_fast_divisor(static_cast<uint32_t>(num_heads), &p.heads_mul, &p.heads_shift);
    const auto addr = [](const void* q_) { return reinterpret_cast<uintptr_t>(q_); };
    p.scales_word_aligned = addr(scales) % 4 == 0 && scale_stride0 % 4 == 0 && scale_stride1 % 4 == 0;
    const int nope = head_dim - rot_dim;
    const bool rows_shape = nope % 8 == 0 && rot_dim % 8 == 0 && addr(q) % 16 == 0 && q_stride0 % 8 == 0 && q_stride1 % 8 == 0 &&
                            addr(out) % 8 == 0 && out_stride0 % 8 == 0 && out_stride1 % 8 == 0;
    const bool heads_shape = head_dim == 128 && rot_dim == 64 && rows_shape &&
                             (fp4 || (addr(out) % 16 == 0 && out_stride0 % 16 == 0 && out_stride1 % 16 == 0));
    if (heads_shape) {
        constexpr int WARPS = kHeadsWarps;
        const bool prefetch = rows >= kPrefetchRows;
        const bool wide = addr(q) % 32 == 0 && q_stride0 % 16 == 0 && q_stride1 % 16 == 0;
        const int with_seven = heads_with_seven_ctas(num_tokens, num_heads, wide);
        const int heads_per_task = with_seven != 0 ? with_seven : heads_of_a_task(num_tokens, num_heads);
        const int64_t tasks_per_token = (num_heads + heads_per_task - 1) / heads_per_task;
        const dim3 grid(static_cast<unsigned>((num_tokens * tasks_per_token + WARPS - 1) / WARPS));
        uint32_t mul, shift;
        make_fast_divisor(static_cast<uint32_t>(tasks_per_token), &mul, &shift);
        const auto run = [&](auto* kernel) { launch_dependent(kernel, grid, WARPS * 32, stream, p, heads_per_task, static_cast<uint32_t>(tasks_per_token), mul, shift); };
        if (with_seven != 0 && wide) fp4 ? run(indexer_q_rope_quant_heads_kernel<WARPS, true, true, false, 7>) : run(indexer_q_rope_quant_heads_kernel<WARPS, false, true, false, 7>);
        else if (with_seven != 0) fp4 ? run(indexer_q_rope_quant_heads_kernel<WARPS, true, false, false, 7>) : run(indexer_q_rope_quant_heads_kernel<WARPS, false, false, false, 7>);
        else if (!wide) fp4 ? run(indexer_q_rope_quant_heads_kernel<WARPS, true, false, false>) : run(indexer_q_rope_quant_heads_kernel<WARPS, false, false, false>);
        else if (!prefetch) fp4 ? run(indexer_q_rope_quant_heads_kernel<WARPS, true, true, false>) : run(indexer_q_rope_quant_heads_kernel<WARPS, false, true, false>);
        else fp4 ? run(indexer_q_rope_quant_heads_kernel<WARPS, true, true, true>) : run(indexer_q_rope_quant_heads_kernel<WARPS, false, true, true>);
        count_launch();
        return cudaGetLastError();
    }
    if (rows_shape) {
        const int cs_vec4 = !cos_sin_bf16 && rot_dim > 0 && addr(cos_sin) % 16 == 0 && cos_sin_stride % 4 == 0 && (rot_dim / 2) % 4 == 0;
        cudaError_t e = head_dim == 64 ? launch_rows<8>(p, fp4 != 0, rows, cs_vec4, stream)
                        : head_dim == 128 ? launch_rows<16>(p, fp4 != 0, rows, cs_vec4, stream)
                        : head_dim == 256 ? launch_rows<32>(p, fp4 != 0, rows, cs_vec4, stream) : cudaErrorInvalidValue;
        if (e != cudaErrorInvalidValue) count_launch();
        return e;
    }
    const unsigned grid = static_cast<unsigned>((rows + 7) / 8);
    cudaError_t err;
    if (head_dim == 64) err = launch_e<2>(p, fp4 != 0, grid, stream);
    else if (head_dim == 128) err = launch_e<4>(p, fp4 != 0, grid, stream);
    else if (head_dim == 256) err = launch_e<8>(p, fp4 != 0, grid, stream);
    else return cudaErrorInvalidValue;
    count_launch();
    return err;
}

}  // namespace dsv4
