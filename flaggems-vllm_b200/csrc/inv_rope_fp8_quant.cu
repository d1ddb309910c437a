// fused_inv_rope_fp8_quant: the attention epilogue that mirrors the prologue - inverse GPT-J RoPE on
// the rotary tail of the attention output o [N, H, 512], then FP8 e4m3 quantisation in groups of 128
// with one scale per group (fp32 = amax/448, or a power of two packed as UE8M0 bytes).
// Reference: src/flaggems_vllm/ops/fused_inv_rope_fp8_quant.py:37-256 and its torch statement
// tests/test_fused_inv_rope_fp8_quant.py:150-198, which this kernel follows to the bit: the rotated
// tail is rounded to bf16 before it is quantised (the torch path does, the Triton kernel does not).
//
// HBM traffic: 1 KiB read, 512 + 16 bytes written per (token, head) row.
#include "dsv4_common.cuh"

namespace dsv4 {
namespace {

struct InvRopeParams {
    const uint8_t* o;          // bf16 [N, H, 512], element strides below
    int64_t o_stride_token, o_stride_head;
    const int64_t* positions;  // [N]
    const float* cos_sin;      // fp32 rows of 64, row stride below
    int64_t cos_sin_stride;
    uint8_t* fp8;              // [G, N, hpg*512] e4m3
    uint8_t* scale;            // fp32 or int32, element (g, t, k) at g*scale_stride_group + t + k*padded_tokens
    int64_t scale_stride_group;
    int64_t num_tokens, padded_tokens;
    int32_t num_heads, heads_per_group;
    float eps;
    uint32_t hpg_mul, hpg_shift;      // fast division of a head index by heads_per_group
};

// A warp owns `heads_per_task` consecutive heads of one token and walks them U at a time.  Of a head, lane l < 28 holds the
// un-rotated values [16l, 16l + 16) and every lane the 4-byte rotary pair 448+2l, 449+2l, so every lane rotates exactly one
// pair with a cosine and sine it loaded once for the whole task.  The quantisation groups of 128 are the lanes 0-7, 8-15,
// 16-23, and 24-27 together with all rotary pairs.
// PACKED: power-of-two scales, the 4 UE8M0 bytes of a head packed into one int32.
// FASTDIV (fp32-scale mode only): see ScaleDivider.
// WIDE: one 32-byte load and one 16-byte store per lane and head; otherwise (rows on 16-byte boundaries only) two of half the
// size.
// Two passes of U heads are in flight: the loads of the next pass go out before the current one is worked on.
// HBM-bound at full clock (8192 x 128 rows 240 us = 6.7 TB/s, fp32 scales 245).  In a run of some tenths of a second the power limit takes
// the clock to 1.58 GHz, and there instruction issue bounds it as well: 250 us, fp32 scales 273 (rows on 16-byte boundaries 278 and 298).
// So every lane loads 32 bytes, the last four the rotary values once more, and a mask keeps them out of the maximum (no lane-dependent
// branch around the loads, no zeroing), and the last group's scale is formed once, by its own lanes, and fetched by a shuffle: about 150
// warp instructions a head (tasks of 16 heads; fp32 scales 168) instead of 182, with which it took 264 and 293 us (284 and 312).
// Heads per pass and CTAs per SM, 8192 x 128 rows, sustained: 2, 7 252 us; 1, 10 258; 1, 8 269; 2, 6 258; 2, 8 254 (fp32 scales 298); 3, 6 306.
constexpr int kMainLanes = 28;
constexpr int kHeadsInFlight = 2;  // per pass
constexpr int kCtasPerSm = 7;      // 72 registers

template <int WARPS, bool PACKED, bool FASTDIV, int U, int MIN_CTAS, bool WIDE>
__global__ void __launch_bounds__(WARPS * 32, MIN_CTAS) inv_rope_fp8_quant_kernel(const Launched<InvRopeParams, 4 * sizeof(int)> p, const int heads_per_task, const uint32_t tasks_per_token,
                                                                      const uint32_t tpt_mul, const uint32_t tpt_shift) {
    begin_dependent_kernel();
    const int lane = threadIdx.x & 31;
    const uint32_t task = blockIdx.x * WARPS + (threadIdx.x >> 5);
    if (task >= static_cast<uint32_t>(p.padded_tokens) * tasks_per_token) return;
    const uint32_t token = fast_div(task, tpt_mul, tpt_shift);
    const int head_begin = static_cast<int>(task - token * tasks_per_token) * heads_per_task;
    const int head_end = head_begin + heads_per_task < p.num_heads ? head_begin + heads_per_task : p.num_heads;
    if (token >= p.num_tokens) {
        // token padding of the scale storage (a multiple of 4 tokens): zero scales
        for (int head = head_begin; head < head_end; ++head) {
            const int group = static_cast<int>(fast_div(static_cast<uint32_t>(head), p.hpg_mul, p.hpg_shift));
            const int head_in_group = head - group * p.heads_per_group;
            uint8_t* scale_row = p.scale + (group * p.scale_stride_group + token) * 4;
            if (PACKED) {
                if (lane == 0) *reinterpret_cast<uint32_t*>(scale_row + head_in_group * p.padded_tokens * 4) = 0u;
            } else if (lane < 4) {
                *reinterpret_cast<float*>(scale_row + (head_in_group * 4 + lane) * p.padded_tokens * 4) = 0.0f;
            }
        }
        return;
    }
    // A pass is U heads.  Past the last head of the task its first one is loaded once more.
    struct Pass {
        Bytes32 v[U];
        uint32_t tail[U];
    };
    const int64_t head_stride = p.o_stride_head * 2;
    const uint8_t* in = p.o + static_cast<int64_t>(token) * p.o_stride_token * 2 + head_begin * head_stride;  // of the next pass to load
    const auto load_pass = [&](int h0, Pass& to) {
        if (h0 < head_end) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint8_t* from = u == 0 || h0 + u < head_end ? in + u * head_stride : in;
                if (WIDE) to.v[u] = ld_stream32(from + 32 * lane);
                else to.v[u].lo = ld_stream16(from + 32 * lane), to.v[u].hi = ld_stream16(from + 32 * lane + 16);
                to.tail[u] = ld_stream4(from + 2 * kNopeDim + 4 * lane);
            }
        }
        in += U * head_stride;
    };
    Pass first, second;
    load_pass(head_begin, first);
    const float* cs = p.cos_sin + p.positions[token] * p.cos_sin_stride;
    const float c = cs[lane], sn = cs[32 + lane];
    // Output addresses advance by constants from one head to the next and are recomputed only where a new group of heads
    // begins: `out` = the head's 512 e4m3 bytes, `scale_at` = its scales (fp32: this lane group's of the four).
    int group = static_cast<int>(fast_div(static_cast<uint32_t>(head_begin), p.hpg_mul, p.hpg_shift));
    int head_in_group = head_begin - group * p.heads_per_group;
    const int64_t group_bytes = static_cast<int64_t>(p.heads_per_group) * (kRowBytes / 2);
    const int64_t scale_column = p.padded_tokens * 4;                       // bytes between scale columns of one token
    const int64_t scale_step = PACKED ? scale_column : 4 * scale_column;    // ... between consecutive heads
    const int64_t lane_scale = PACKED ? 0 : (lane >> 3) * scale_column;     // fp32: lanes 0 / 8 / 16 / 24 store one each
    const auto group_out = [&](int g) { return p.fp8 + (static_cast<int64_t>(g) * p.num_tokens + token) * group_bytes; };
    const auto group_scale = [&](int g) { return p.scale + (g * p.scale_stride_group + token) * 4 + lane_scale; };
    uint8_t* out = group_out(group) + static_cast<int64_t>(head_in_group) * (kRowBytes / 2);
    uint8_t* scale_at = group_scale(group) + head_in_group * scale_step;
    const uint32_t main_mask = lane < kMainLanes ? 0xffffffffu : 0u;  // lanes whose 16 values are not rotary ones
    const uint32_t rotary_mask = lane >= 24 ? 0xffff0000u : 0u;  // lanes of the last group: the pairs belong to it
    const int scale_shift = lane & 24;                           // chunk k of the head in byte k
    const auto finish_pass = [&](int h0, const Pass& pass) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (h0 + u >= head_end) break;
            // inverse rotation of the lane's pair, products rounded separately, then to bf16 as the torch path does
            const float e = bf16_lo(pass.tail[u]), o = bf16_hi(pass.tail[u]);
            const uint32_t rot = pack_bf16x2(__fadd_rn(__fmul_rn(e, c), __fmul_rn(o, sn)), __fsub_rn(__fmul_rn(o, c), __fmul_rn(e, sn)));
            // Group maxima on the packed words: |.| maxima of the even and the odd elements side by side (the sign bits of
            // the intermediate words are meaningless and cleared at the end), then the maximum of the lane's 16 values in
            // the low half and that of its pair in the high half of one word.
            const uint4 &a = pass.v[u].lo, &b = pass.v[u].hi;
            const uint32_t all = max_abs_bf16x2(max_abs_bf16x2(max_abs_bf16x2(a.x, a.y), max_abs_bf16x2(a.z, a.w)),
                                               max_abs_bf16x2(max_abs_bf16x2(b.x, b.y), max_abs_bf16x2(b.z, b.w)));
            const uint32_t pm = all & main_mask;
            uint32_t both = max_abs_bf16x2(__byte_perm(pm, rot, 0x5410), __byte_perm(pm, rot, 0x7632)) & 0x7fff7fffu;
#pragma unroll
            for (int m = 1; m <= 4; m <<= 1) both = max_bf16x2(both, __shfl_xor_sync(0xffffffffu, both, m));
            const uint32_t of_eight = both;  // low half: the group's maximum, in the last group without the pairs
#pragma unroll
            for (int m = 8; m <= 16; m <<= 1) both = max_bf16x2(both, __shfl_xor_sync(0xffffffffu, both, m));
            const float largest = fmaxf(bf16_lo(of_eight), __uint_as_float(both & rotary_mask));
            const float scale = __fmul_rn(fmaxf(largest, p.eps), 1.0f / 448.0f);
            uint2 qa, qb;
            const auto store_pair = [&](const float2& t) {
                *reinterpret_cast<uint16_t*>(out + kNopeDim + 2 * lane) = static_cast<uint16_t>(pack_e4m3x4(t.x, t.y, 0.f, 0.f));
            };
            if (PACKED) {
                const uint32_t code = pow2_ceil_code(scale), factor = pow2_reciprocal(code), factor_3 = __shfl_sync(0xffffffffu, factor, 24);
                qa = quant8_times(a, factor), qb = quant8_times(b, factor);
                store_pair(scaled_pair(rot, static_cast<uint16_t>(factor_3)));
                const uint32_t word = __reduce_or_sync(0xffffffffu, code << scale_shift);
                if (lane == 0) *reinterpret_cast<uint32_t*>(scale_at) = word;
            } else {
                // the three-instruction form of the fast division for every scale: a warp-uniform choice between it and the
                // two-instruction form was no faster
                constexpr int kDivision = FASTDIV ? kDivideFast : kDivideIeee;
                // Scale and pair are stored before the other values are divided, which then have the registers: without that the
                // 16-byte form spills 8 bytes a thread (8192 x 128 rows, sustained, 309 us instead of 298).
                if ((lane & 7) == 0) *reinterpret_cast<float*>(scale_at) = scale;
                const float divisor = FASTDIV ? finite_scale(scale) : scale;
                store_pair(quotients<kDivision, false>(rot, ScaleDivider<kDivision>(__shfl_sync(0xffffffffu, divisor, 24))));
                const ScaleDivider<kDivision> by(divisor);
                qa = quant8_by<kDivision, false>(a, by), qb = quant8_by<kDivision, false>(b, by);
            }
            if (lane < kMainLanes) {
                if (WIDE) st_stream16(out + 16 * lane, make_uint4(qa.x, qa.y, qb.x, qb.y));
                else st_global8(out + 16 * lane, qa), st_global8(out + 16 * lane + 8, qb);
            }
            // on to the next head
            out += kRowBytes / 2, scale_at += scale_step;
            if (++head_in_group == p.heads_per_group) {
                head_in_group = 0, ++group;
                out = group_out(group), scale_at = group_scale(group);
            }
        }
    };
    for (int h0 = head_begin; h0 < head_end; h0 += U) {
        load_pass(h0 + U, second);  // past the end of the task: nothing
        finish_pass(h0, first);
        first = second;
    }
}

// Any geometry the reference wrapper accepts (head_dim = nope + rope a multiple of the group size, the rotary tail
// ending the last group, even group size): one warp per (token, head), one group after the other, two passes over a
// group (maximum, then quantise; the rotation is recomputed, which is deterministic).  Same arithmetic as above: rotated
// values rounded to bf16 before quantising, fp32 scales divide (IEEE), power-of-two scales multiply by the exact
// reciprocal.  Packed scales need four groups per head: one int32 per head is the only layout in which the reference's
// kernel and its allocation agree (src/flaggems_vllm/ops/fused_inv_rope_fp8_quant.py:133-143, 206-217).
struct InvRopeGeometry {
    int32_t nope_dim, rope_dim, group, chunks;
};

template <int WARPS, bool PACKED>
__global__ void __launch_bounds__(WARPS * 32) inv_rope_fp8_quant_any_kernel(const Launched<InvRopeParams, sizeof(InvRopeGeometry)> p, const InvRopeGeometry geo) {
    begin_dependent_kernel();
    const int lane = threadIdx.x & 31;
    const int64_t row = static_cast<int64_t>(blockIdx.x) * WARPS + (threadIdx.x >> 5);
    if (row >= p.padded_tokens * p.num_heads) return;
    const int64_t token = row / p.num_heads;
    const int head = static_cast<int>(row - token * p.num_heads);
    const int group = head / p.heads_per_group, head_in_group = head - group * p.heads_per_group;
    uint8_t* scale_row = p.scale + (group * p.scale_stride_group + token) * 4;
    if (token >= p.num_tokens) {  // token padding of the scale storage: zero scales
        if (PACKED) {
            if (lane == 0) *reinterpret_cast<uint32_t*>(scale_row + static_cast<int64_t>(head_in_group) * p.padded_tokens * 4) = 0u;
        } else if (lane < geo.chunks) {
            *reinterpret_cast<float*>(scale_row + (static_cast<int64_t>(head_in_group) * geo.chunks + lane) * p.padded_tokens * 4) = 0.0f;
        }
        return;
    }
    const int head_dim = geo.nope_dim + geo.rope_dim, half_rope = geo.rope_dim / 2;
    const float* cs = p.cos_sin + p.positions[token] * p.cos_sin_stride;
    const uint16_t* in = reinterpret_cast<const uint16_t*>(p.o) + token * p.o_stride_token + static_cast<int64_t>(head) * p.o_stride_head;
    uint8_t* out = p.fp8 + (static_cast<int64_t>(group) * p.num_tokens + token) * (static_cast<int64_t>(p.heads_per_group) * head_dim) +
                   static_cast<int64_t>(head_in_group) * head_dim;
    // the pair (2j, 2j+1) of the head after the inverse rotation (if it lies in the rotary tail) and the bf16 rounding
    const auto pair_at = [&](int e0, float* a, float* b) {
        const float e = bf16_lo(in[e0]), o = bf16_lo(in[e0 + 1]);
        if (e0 >= geo.nope_dim) {
            const int j = (e0 - geo.nope_dim) >> 1;
            const float c = cs[j], sn = cs[half_rope + j];
            const uint32_t rot = pack_bf16x2(__fadd_rn(__fmul_rn(e, c), __fmul_rn(o, sn)), __fsub_rn(__fmul_rn(o, c), __fmul_rn(e, sn)));
            *a = bf16_lo(rot), *b = bf16_hi(rot);
        } else {
            *a = e, *b = o;
        }
    };
    uint32_t word = 0;
    for (int k = 0; k < geo.chunks; ++k) {
        float amax = 0.0f;
        for (int pr = lane; pr < geo.group / 2; pr += 32) {
            float a, b;
            pair_at(k * geo.group + 2 * pr, &a, &b);
            amax = fmaxf(amax, fmaxf(fabsf(a), fabsf(b)));
        }
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, m));
        float scale = __fmul_rn(fmaxf(amax, p.eps), 1.0f / 448.0f);
        float inv = 0.0f;
        if (PACKED) {
            const uint32_t code = pow2_ceil_code(scale);
            word |= code << (8 * k);
            inv = bf16_lo(pow2_reciprocal(code));
        }
        for (int pr = lane; pr < geo.group / 2; pr += 32) {
            const int e0 = k * geo.group + 2 * pr;
            float a, b;
            pair_at(e0, &a, &b);
            const float qa = PACKED ? __fmul_rn(a, inv) : __fdiv_rn(a, scale), qb = PACKED ? __fmul_rn(b, inv) : __fdiv_rn(b, scale);
            *reinterpret_cast<uint16_t*>(out + e0) = static_cast<uint16_t>(pack_e4m3x4(qa, qb, 0.f, 0.f));
        }
        if (!PACKED && lane == 0)
            *reinterpret_cast<float*>(scale_row + (static_cast<int64_t>(head_in_group) * geo.chunks + k) * p.padded_tokens * 4) = scale;
    }
    if (PACKED && lane == 0) *reinterpret_cast<uint32_t*>(scale_row + static_cast<int64_t>(head_in_group) * p.padded_tokens * 4) = word;
}

}  // namespace

cudaError_t launch_inv_rope_fp8_quant_any(const void* o, int64_t o_stride_token, int64_t o_stride_head, const int64_t* positions,
                                          const float* cos_sin, int64_t cos_sin_stride, void* fp8, void* scale,
                                          int64_t scale_stride_group, int64_t num_tokens, int64_t padded_tokens, int num_heads,
                                          int heads_per_group, int nope_dim, int rope_dim, int group_size, float eps, int packed,
                                          cudaStream_t stream) {
    constexpr int WARPS = 4;
    const int64_t rows = padded_tokens * num_heads;
    if (rows == 0) return cudaSuccess;
    const int64_t grid = (rows + WARPS - 1) / WARPS;
    if (grid > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    InvRopeParams p{};
    p.o = static_cast<const uint8_t*>(o), p.o_stride_token = o_stride_token, p.o_stride_head = o_stride_head;
    p.positions = positions, p.cos_sin = cos_sin, p.cos_sin_stride = cos_sin_stride;
    p.fp8 = static_cast<uint8_t*>(fp8), p.scale = static_cast<uint8_t*>(scale), p.scale_stride_group = scale_stride_group;
    p.num_tokens = num_tokens, p.padded_tokens = padded_tokens, p.num_heads = num_heads, p.heads_per_group = heads_per_group;
    p.eps = eps;
    const InvRopeGeometry geo{nope_dim, rope_dim, group_size, (nope_dim + rope_dim) / group_size};
    if (packed) launch_dependent(inv_rope_fp8_quant_any_kernel<WARPS, true>, static_cast<unsigned>(grid), WARPS * 32, stream, p, geo);
    else launch_dependent(inv_rope_fp8_quant_any_kernel<WARPS, false>, static_cast<unsigned>(grid), WARPS * 32, stream, p, geo);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_inv_rope_fp8_quant(const void* o, int64_t o_stride_token, int64_t o_stride_head, const int64_t* positions,
                                      const float* cos_sin, int64_t cos_sin_stride, void* fp8, void* scale,
                                      int64_t scale_stride_group, int64_t num_tokens, int64_t padded_tokens, int num_heads,
                                      int heads_per_group, float eps, int packed, cudaStream_t stream) {
    constexpr int WARPS = 4;
    const int64_t rows = padded_tokens * num_heads;
    if (rows == 0) return cudaSuccess;
    // The longest task that still leaves about 4096 of them (the GPU holds 148 x 28 warps): its set-up is shared by more heads,
    // and two passes are in flight.  61 x 128 rows: 3.7 us with 2 heads per task, 7.2 with 16; 256 x 128: 9.9 us with 8, 11.3 with
    // 2 or 16; 4096 x 128: 123 us with 16, 162 with 2.
    int heads_per_task = 2;
    while (heads_per_task < 16 && rows >= 8192LL * heads_per_task) heads_per_task *= 2;
    const int64_t tasks_per_token = (num_heads + heads_per_task - 1) / heads_per_task;
    const int64_t tasks = padded_tokens * tasks_per_token;
    const int64_t grid = (tasks + WARPS - 1) / WARPS;
    if (grid > 0x7fffffffLL || tasks >= (1LL << 31)) return cudaErrorInvalidConfiguration;
    InvRopeParams p{};
    p.o = static_cast<const uint8_t*>(o), p.o_stride_token = o_stride_token, p.o_stride_head = o_stride_head;
    p.positions = positions, p.cos_sin = cos_sin, p.cos_sin_stride = cos_sin_stride;
    p.fp8 = static_cast<uint8_t*>(fp8), p.scale = static_cast<uint8_t*>(scale), p.scale_stride_group = scale_stride_group;
    p.num_tokens = num_tokens, p.padded_tokens = padded_tokens, p.num_heads = num_heads, p.heads_per_group = heads_per_group;
    p.eps = eps;
    make_fast_divisor(static_cast<uint32_t>(heads_per_group), &p.hpg_mul, &p.hpg_shift);
    uint32_t tpt_mul, tpt_shift;
    make_fast_divisor(static_cast<uint32_t>(tasks_per_token), &tpt_mul, &tpt_shift);
    const unsigned g = static_cast<unsigned>(grid);
    const uint32_t tpt = static_cast<uint32_t>(tasks_per_token);
    const auto addr = [](const void* q) { return reinterpret_cast<uintptr_t>(q); };
    const bool wide = addr(o) % 32 == 0 && o_stride_token % 16 == 0 && o_stride_head % 16 == 0 && addr(fp8) % 16 == 0;
    const auto run = [&](auto* kernel) { launch_dependent(kernel, g, WARPS * 32, stream, p, heads_per_task, tpt, tpt_mul, tpt_shift); };
    constexpr int U = kHeadsInFlight, C = kCtasPerSm;
    if (packed) wide ? run(inv_rope_fp8_quant_kernel<WARPS, true, false, U, C, true>) : run(inv_rope_fp8_quant_kernel<WARPS, true, false, U, C, false>);
    else if (eps == 1e-10f) wide ? run(inv_rope_fp8_quant_kernel<WARPS, false, true, U, C, true>) : run(inv_rope_fp8_quant_kernel<WARPS, false, true, U, C, false>);
    else wide ? run(inv_rope_fp8_quant_kernel<WARPS, false, false, U, C, true>) : run(inv_rope_fp8_quant_kernel<WARPS, false, false, U, C, false>);
    count_launch();
    return cudaGetLastError();
}

}  // namespace dsv4
