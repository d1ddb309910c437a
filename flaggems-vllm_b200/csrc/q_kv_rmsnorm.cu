// fused_q_kv_rmsnorm: the step before the prologue - weighted RMSNorm of the q low-rank
// activations [N, Q] and of the latent KV [N, KV] in one launch.
// Reference: src/flaggems_vllm/ops/deepseek_v4_attention_fused_q_kv_rmsnorm.py:24-103
//   y = (x * rsqrt(mean(x^2) + eps)) * w, fp32 arithmetic, bf16 in and out.
// The order of the sum of squares is this kernel's own (a lane adds up runs of 16 neighbouring values, then the warp its lanes),
// as the reference leaves it open; runs of 8 move 3 outputs in 10^6 by one bf16 step, and are no nearer to the 64-bit result (6.5 in
// 10^6 differ from it, 5 with runs of 16; 4097 tokens).
// One warp per row; a row of up to 2048 elements stays in registers between the reduction and
// the scaling (one read, one write per element); longer or unaligned rows take a two-pass
// scalar path.  Row 2t is the q row of token t, row 2t+1 its kv row.
#include <algorithm>

#include <cuda_fp16.h>

#include "dsv4_common.cuh"

namespace dsv4 {
namespace {

struct NormRows {
    const uint8_t* in;
    uint8_t* out;
    const uint8_t* weight;
    int64_t in_stride, out_stride;  // elements
    int32_t size;
    int32_t vec_ok;                 // vectorised path usable for this tensor
};

constexpr int kMaxChunks = 4;  // at most 4 32-byte chunks per lane are held in registers: 4 * 32 * 16 = 2048 elements

__device__ __forceinline__ float inv_rms_of(float sum, int size, float eps) {
    const float v = __fadd_rn(__fdiv_rn(sum, static_cast<float>(size)), eps);
    const float r0 = rsqrtf(v);
    return fmaf(r0, fmaf(-0.5f * v * r0, r0, 0.5f), r0);
}

// CH = 32-byte chunks per lane the launch needs (1 to 4): fewer live registers for the common 1536 / 512 rows.  WIDE: one 32-byte
// access per chunk, otherwise (rows on 16-byte boundaries only) two.  EARLY: the weights are fetched before the reduction.
constexpr int ctas_per_sm(int chunks, bool early) {  // of 128 threads
    return early ? (chunks == 1 ? 10 : chunks == 2 ? 7 : chunks == 3 ? 5 : 4) : (chunks == 1 ? 16 : chunks == 2 ? 10 : chunks == 3 ? 7 : 6);
}

template <int WARPS, int CH, bool WIDE, bool EARLY, int CTAS = ctas_per_sm(CH, EARLY)>
__global__ void __launch_bounds__(WARPS * 32, CTAS)
q_kv_rmsnorm_kernel(const Launched<NormRows, sizeof(NormRows) + 16> q, const NormRows kv, int64_t num_tokens, float eps) {
    const int lane = threadIdx.x & 31;
    const int64_t r = static_cast<int64_t>(blockIdx.x) * WARPS + (threadIdx.x >> 5);
    if (r >= 2 * num_tokens) return;
    const bool is_q = (r & 1) == 0;  // rows alternate q, kv, q, kv ... so long and short rows mix in every CTA
    const NormRows& t = is_q ? q : kv;
    const int64_t token = r >> 1;
    const uint8_t* in = t.in + token * t.in_stride * 2;
    uint8_t* out = t.out + token * t.out_stride * 2;
    const int size = t.size;
    if (t.vec_ok && lane == 0 && starts_early()) prefetch_l2(in, 2u * static_cast<uint32_t>(size));
    begin_dependent_kernel();
    if (t.vec_ok) {
        const int chunks = (size + 15) >> 4;
        const int half = WIDE ? -1 : (size & 8 ? chunks - 1 : -1);  // the chunk whose second 8 values lie outside the row
        Bytes32 x[CH], w[CH];
        const auto load_weights = [&](int j) {
            const int c = lane + 32 * j;
            const uint4* from = reinterpret_cast<const uint4*>(t.weight + 32 * c);
            w[j].lo = w[j].hi = make_uint4(0u, 0u, 0u, 0u);
            if (c < chunks) {
                w[j].lo = __ldg(from);
                if (c != half) w[j].hi = __ldg(from + 1);
            }
        };
        float acc = 0.0f;
#pragma unroll
        for (int j = 0; j < CH; ++j) {
            const int c = lane + 32 * j;
            x[j].lo = x[j].hi = make_uint4(0u, 0u, 0u, 0u);
            if (c < chunks) {
                if (WIDE) x[j] = ld_stream32(in + 32 * c);
                else x[j].lo = ld_stream16(in + 32 * c);
                if (!WIDE && c != half) x[j].hi = ld_stream16(in + 32 * c + 16);
            }
        }
        if (EARLY) {
#pragma unroll
            for (int j = 0; j < CH; ++j) load_weights(j);
        }
#pragma unroll
        for (int j = 0; j < CH; ++j) {
            float f[8], g[8];
            unpack8(x[j].lo, f), unpack8(x[j].hi, g);
#pragma unroll
            for (int i = 0; i < 8; ++i) acc = fmaf(f[i], f[i], acc);
#pragma unroll
            for (int i = 0; i < 8; ++i) acc = fmaf(g[i], g[i], acc);
        }
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
        const float rr = inv_rms_of(acc, size, eps);
        // Two values an instruction, the same products, each rounded: rows of 512 on 16-byte boundaries 16384 tokens 16.8 -> 15.1 us, others
        // up to 2 %.  Not where it spills (16-byte form, rows of up to 1024 and 2048: 16384 tokens 19.2 us scalar and 21.9 packed, 32.2 and 34.3).
        constexpr bool kPairs = WIDE || CH % 2 == 1;
        const auto product = [&](uint32_t xv, uint32_t wv) {
            float2 y;
            asm("{.reg .b64 x, r, w;\n\t"
                "mov.b64 x, {%2, %3};\n\t"
                "mov.b64 r, {%4, %4};\n\t"
                "mov.b64 w, {%5, %6};\n\t"
                "mul.rn.f32x2 x, x, r;\n\t"
                "mul.rn.f32x2 x, x, w;\n\t"
                "mov.b64 {%0, %1}, x;}"
                : "=f"(y.x), "=f"(y.y)
                : "f"(bf16_lo(xv)), "f"(bf16_hi(xv)), "f"(rr), "f"(bf16_lo(wv)), "f"(bf16_hi(wv)));
            return pack_bf16x2(y.x, y.y);
        };
        const auto apply = [&](const uint4& xv, const uint4& wv) {
            if (!kPairs) {
                float f[8], g[8];
                unpack8(xv, f), unpack8(wv, g);
#pragma unroll
                for (int i = 0; i < 8; ++i) f[i] = __fmul_rn(__fmul_rn(f[i], rr), g[i]);
                return pack8(f);
            }
            return make_uint4(product(xv.x, wv.x), product(xv.y, wv.y), product(xv.z, wv.z), product(xv.w, wv.w));
        };
#pragma unroll
        for (int j = 0; j < CH; ++j) {
            const int c = lane + 32 * j;
            if (!EARLY) load_weights(j);
            if (c < chunks) {
                const Bytes32 y{apply(x[j].lo, w[j].lo), apply(x[j].hi, w[j].hi)};
                if (WIDE) st_stream32(out + 32 * c, y);
                else st_stream16(out + 32 * c, y.lo);
                if (!WIDE && c != half) st_stream16(out + 32 * c + 16, y.hi);
            }
        }
    } else {
        const uint16_t* in16 = reinterpret_cast<const uint16_t*>(in);
        const uint16_t* w16 = reinterpret_cast<const uint16_t*>(t.weight);
        uint16_t* out16 = reinterpret_cast<uint16_t*>(out);
        float acc = 0.0f;
        for (int i = lane; i < size; i += 32) {
            const float f = bf16_lo(in16[i]);
            acc = fmaf(f, f, acc);
        }
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
        const float rr = inv_rms_of(acc, size, eps);
        for (int i = lane; i < size; i += 32) {
            const float y = __fmul_rn(__fmul_rn(bf16_lo(in16[i]), rr), bf16_lo(w16[i]));
            out16[i] = static_cast<uint16_t>(pack_bf16x2(y, 0.0f) & 0xffffu);
        }
    }
}

// Any of bf16 (0), fp16 (1), fp32 (2) for the rows and, independently, for the weights: the reference kernel is
// generic over the element types (it loads everything as fp32 and stores in the output's type).  One warp per row,
// two passes over the row, element by element.  The DeepSeek-V4 layer passes bf16 everywhere and takes the kernel above.
struct AnyRows {
    const uint8_t* in;
    uint8_t* out;
    const uint8_t* weight;
    int64_t in_stride, out_stride;  // elements
    int32_t size, dtype, weight_dtype;
};

__device__ __forceinline__ float load_any(const uint8_t* base, int64_t i, int dtype) {
    if (dtype == 2) return reinterpret_cast<const float*>(base)[i];
    const uint16_t h = reinterpret_cast<const uint16_t*>(base)[i];
    return dtype == 0 ? bf16_lo(h) : __half2float(__ushort_as_half(h));
}

__device__ __forceinline__ void store_any(uint8_t* base, int64_t i, int dtype, float v) {
    if (dtype == 2) reinterpret_cast<float*>(base)[i] = v;
    else if (dtype == 0) reinterpret_cast<uint16_t*>(base)[i] = static_cast<uint16_t>(pack_bf16x2(v, 0.0f) & 0xffffu);
    else reinterpret_cast<uint16_t*>(base)[i] = __half_as_ushort(__float2half_rn(v));
}

template <int WARPS>
__global__ void __launch_bounds__(WARPS * 32) q_kv_rmsnorm_any_kernel(const Launched<AnyRows, sizeof(AnyRows) + 16> q, const AnyRows kv, int64_t num_tokens, float eps) {
    begin_dependent_kernel();
    const int lane = threadIdx.x & 31;
    const int64_t r = static_cast<int64_t>(blockIdx.x) * WARPS + (threadIdx.x >> 5);
    if (r >= 2 * num_tokens) return;
    const AnyRows& t = (r & 1) == 0 ? q : kv;
    const int64_t token = r >> 1;
    const int esize = t.dtype == 2 ? 4 : 2;
    const uint8_t* in = t.in + token * t.in_stride * esize;
    uint8_t* out = t.out + token * t.out_stride * esize;
    float acc = 0.0f;
    for (int i = lane; i < t.size; i += 32) {
        const float f = load_any(in, i, t.dtype);
        acc = fmaf(f, f, acc);
    }
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
    const float rr = inv_rms_of(acc, t.size, eps);
    for (int i = lane; i < t.size; i += 32)
        store_any(out, i, t.dtype, __fmul_rn(__fmul_rn(load_any(in, i, t.dtype), rr), load_any(t.weight, i, t.weight_dtype)));
}

// Rows and weights on boundaries of `bytes` (16 or 32), 16 values per lane and chunk.
bool on_boundaries(uintptr_t bytes, const NormRows& t) {
    const auto off = [&](const void* p) { return reinterpret_cast<uintptr_t>(p) % bytes; };
    const int64_t elements = static_cast<int64_t>(bytes / 2);
    return off(t.in) == 0 && off(t.out) == 0 && reinterpret_cast<uintptr_t>(t.weight) % 16 == 0 && t.in_stride % elements == 0 &&
           t.out_stride % elements == 0 && t.size % elements == 0 && t.size <= kMaxChunks * 512;
}

// Whether the weights are fetched before the reduction or after it.  Before, they wait for nothing; after, fewer registers are held and
// more rows are in flight.  Before | after, us a launch from a graph, rows of 1536 and 512 (96 registers and five CTAs per SM | 72 and
// seven), out of L2 as a projection has just written them, and from HBM:
//   tokens   61         600        1100       1480       1531       2000       2300       2960       3600       4096       8192
//   L2       1.5|1.9    1.7|2.3    2.3|3.0    2.4|3.1    2.9|3.1    3.3|3.1    3.5|4.4    4.0|4.9    4.8|5.1    5.1|5.4    8.8|8.7
//   HBM      1.5|1.8    1.9|2.4    2.4|2.9    2.6|3.2    3.4|3.2    4.0|3.3    4.3|4.9    5.0|5.4    6.2|6.0    6.8|6.4   12.3|11.4
// So before up to 4096 tokens (from about 3300 on out of L2 only), except where the launch is one wave of the other form and no longer
// one of this: 1481 to 2072 tokens (1481 tokens 2.7|3.1 and 3.0|3.2).  Other widths have such a range too, but there the other form spills, or loses out of L2 what it gains
// from HBM: 512 + 512, 3200 tokens 2.6|3.7 and 3.4|3.6; 1024 + 512, 2073 tokens 2.4|3.2 and 2.9|3.2, 2600 tokens 3.1|3.2 and 3.8|3.4;
// 2048 + 512, 1185 tokens 2.8|3.5 and 3.2|3.6, 1500 tokens 3.4|3.5 and 4.1|3.5.
constexpr int64_t kEarlyWeightTokens = 4096;
// With rows of up to 1536, the early form with four CTAs per SM (102 registers) instead of five, while the launch is one wave of it and
// two such launches, one draining and one starting, no longer fit side by side with five: 741 to 1184 tokens.  Four | five: 600 tokens
// 2.0|1.7 and 2.0|1.9, 740 tokens 2.2|1.8 and 2.2|2.0, 780 tokens 2.2|2.2 and 2.3|2.3, 900 tokens 2.0|2.3 and 2.2|2.4, 1184 tokens 2.1|2.3
// and 2.3|2.4, 1185 tokens 2.5|2.3 and 2.9|2.4, 2960 tokens 4.3|4.0 and 5.8|5.0.
constexpr int kRoomyCtas = 4;
constexpr int64_t kSms = 148;

template <bool WIDE, int CH>
void launch_chunks(const NormRows& q, const NormRows& kv, int64_t num_tokens, float eps, cudaStream_t stream) {
    constexpr int WARPS = 4;
    const int64_t ctas = (2 * num_tokens + WARPS - 1) / WARPS;
    const auto run = [&](auto* kernel) { launch_dependent(kernel, static_cast<unsigned>(ctas), WARPS * 32, stream, q, kv, num_tokens, eps); };
    if constexpr (WIDE) {
        if constexpr (CH == 3) {
            if (2 * ctas > kSms * ctas_per_sm(CH, true) && ctas <= kSms * kRoomyCtas) return run(q_kv_rmsnorm_kernel<WARPS, CH, WIDE, true, kRoomyCtas>);
        }
        const bool one_wave_late = CH == 3 && ctas > kSms * ctas_per_sm(CH, true) && ctas <= kSms * ctas_per_sm(CH, false);
        if (num_tokens <= kEarlyWeightTokens && !one_wave_late) return run(q_kv_rmsnorm_kernel<WARPS, CH, WIDE, true>);
    }
    run(q_kv_rmsnorm_kernel<WARPS, CH, WIDE, false>);
}

template <bool WIDE>
void launch_rows(const NormRows& q, const NormRows& kv, int64_t num_tokens, float eps, cudaStream_t stream) {
    const int32_t longest = std::max(q.vec_ok ? q.size : 0, kv.vec_ok ? kv.size : 0);
    if (longest <= 512) launch_chunks<WIDE, 1>(q, kv, num_tokens, eps, stream);
    else if (longest <= 1024) launch_chunks<WIDE, 2>(q, kv, num_tokens, eps, stream);
    else if (longest <= 1536) launch_chunks<WIDE, 3>(q, kv, num_tokens, eps, stream);
    else launch_chunks<WIDE, 4>(q, kv, num_tokens, eps, stream);
}

}  // namespace

cudaError_t launch_q_kv_rmsnorm(const void* q, void* q_out, const void* q_weight, int64_t q_in_stride, int64_t q_out_stride,
                                int64_t q_size, const void* kv, void* kv_out, const void* kv_weight, int64_t kv_in_stride,
                                int64_t kv_out_stride, int64_t kv_size, int64_t num_tokens, float eps, cudaStream_t stream) {
    if (num_tokens == 0) return cudaSuccess;
    if ((2 * num_tokens + 3) / 4 > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    NormRows a{static_cast<const uint8_t*>(q), static_cast<uint8_t*>(q_out), static_cast<const uint8_t*>(q_weight),
               q_in_stride, q_out_stride, static_cast<int32_t>(q_size), 0};
    NormRows b{static_cast<const uint8_t*>(kv), static_cast<uint8_t*>(kv_out), static_cast<const uint8_t*>(kv_weight),
               kv_in_stride, kv_out_stride, static_cast<int32_t>(kv_size), 0};
    a.vec_ok = on_boundaries(16, a) ? 1 : 0, b.vec_ok = on_boundaries(16, b) ? 1 : 0;
    const bool wide = (!a.vec_ok || on_boundaries(32, a)) && (!b.vec_ok || on_boundaries(32, b));
    if (wide) launch_rows<true>(a, b, num_tokens, eps, stream);
    else launch_rows<false>(a, b, num_tokens, eps, stream);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_q_kv_rmsnorm_any(const void* q, void* q_out, const void* q_weight, int64_t q_in_stride, int64_t q_out_stride,
                                    int64_t q_size, int q_dtype, int q_weight_dtype, const void* kv, void* kv_out,
                                    const void* kv_weight, int64_t kv_in_stride, int64_t kv_out_stride, int64_t kv_size,
                                    int kv_dtype, int kv_weight_dtype, int64_t num_tokens, float eps, cudaStream_t stream) {
    constexpr int WARPS = 4;
    if (num_tokens == 0) return cudaSuccess;
    const AnyRows a{static_cast<const uint8_t*>(q), static_cast<uint8_t*>(q_out), static_cast<const uint8_t*>(q_weight),
                    q_in_stride, q_out_stride, static_cast<int32_t>(q_size), q_dtype, q_weight_dtype};
    const AnyRows b{static_cast<const uint8_t*>(kv), static_cast<uint8_t*>(kv_out), static_cast<const uint8_t*>(kv_weight),
                    kv_in_stride, kv_out_stride, static_cast<int32_t>(kv_size), kv_dtype, kv_weight_dtype};
    const int64_t grid = (2 * num_tokens + WARPS - 1) / WARPS;
    if (grid > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    launch_dependent(q_kv_rmsnorm_any_kernel<WARPS>, static_cast<unsigned>(grid), WARPS * 32, stream, a, b, num_tokens, eps);
    count_launch();
    return cudaGetLastError();
}

}  // namespace dsv4
