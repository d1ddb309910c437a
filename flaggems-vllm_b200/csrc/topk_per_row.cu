// top_k_per_row_decode / top_k_per_row_prefill: the indices of the top_k largest logits of every row inside the
// row's valid range, the selection step of the sparse indexer between its logits and the index bookkeeping.
// Reference: src/flaggems_vllm/ops/top_k_per_row_decode.py:1263-1399, src/flaggems_vllm/ops/top_k_per_row_prefill.py
// (wrapper `top_k_per_row_prefill`), and their torch statements tests/test_top_k_per_row_decode.py:111-124,
// tests/test_top_k_per_row_prefill.py:80-99:
//   row i, range [start_i, end_i): k = min(top_k, end_i - start_i); indices[i, :k] = positions (relative to start_i) of
//   the k largest values, in any order, ties broken arbitrarily; indices[i, k:] = -1.
//   decode:  start_i = 0, end_i = seq_lens[i / next_n] - next_n + i % next_n + 1
//   prefill: start_i = row_starts[i], end_i = row_ends[i]
//
// Values are ranked by the order-preserving 32-bit key of their fp32 pattern.  ONE read of the row on the normal route:
//   1. a sample of the row gives a value t that k values plus four standard deviations of that count are expected to
//      reach (histogram of a coarse, monotone 11-bit code: the top bits of the fp16 rounding of the value, which spreads
//      real logits over hundreds of bins where the top bits of the fp32 pattern would hit a handful);
//   2. every value that reaches t goes with its position to a pool in shared memory, where a warp reserves room for all
//      candidates among 512 values with one atomic; no branches (these kernels are bound by instruction issue and by the
//      phases between barriers before they are bound by HBM);
//   3. the candidates (about 1.1 to 3 k of them) are ranked by a histogram of (key - key(t)), whose bins are fine where
//      the k-th largest is to be expected; the few candidates of its bin are ranked by counting.
// Three kernels:
//   topk_short_kernel       one CTA per row, the row's coarse codes in registers; short rows, of which a large part is selected, go
//                           without a sample: a coarse histogram of all values, then straight to the ranking
//   topk_registers_kernel   one CTA per row, the row in registers, its sample taken from them
//   topk_stream_kernel      longer rows: one CTA, or a thread-block cluster of 2 / 4 / 8 CTAs, streams the row past t; the
//                           first 64 bytes of every thread are on their way while the sample is evaluated.  In a
//                           cluster every CTA takes the same sample, streams its share and hands its candidates to the
//                           first CTA through distributed shared memory (two hardware cluster barriers, no spinning).
// When the sample misjudged the row (fewer than k candidates, or the pool full), or k is too large
// for the pool, a histogram route reads the row twice more; thousands of near-equal values take a radix selection over the
// row.  The result does not depend on the route; the sample only decides how fast it is reached.
// HBM traffic on the normal route: the row once (4 bytes per value); top_k * 4 bytes written.
// Bound by instruction issue and by the phases between barriers before HBM: a row of 32768 values takes 20.5 k warp instructions with
// k 2048 and 17.6 k with k 512 (27.6 k and 22.8 k before signs were shifted into a word instead of counted by comparisons, the
// sample was halved, and places in the result were reserved for four candidates per thread at a time).  Measured before -> after
// that: rows of full length, 4096 x 32768, k 2048 137 -> 121 us, k 512 111 -> 100 us (5.4 TB/s); a causal chunk of 4096 rows,
// k 2048 145 -> 121 us (its sample is now taken in whole lines, the ends of its rows are loaded early); ragged rows, 496 x 262144,
// k 512 74 -> 70 us (67 us with two batches in flight, 60 us with the longest rows first); 4096 x 65536, k 1024 147 -> 130 us; 1000 x 40000, k 512 37 -> 30 us.
#include <cooperative_groups.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <mutex>

#include "dsv4_common.cuh"

namespace dsv4 {
namespace {

namespace cg = cooperative_groups;

constexpr int kBins = 2048;
constexpr int kCountingMax = kBins / 2;  // candidates of one bin ranked by counting (they are kept where the histogram was)
constexpr int kStreamBatch = 4;          // quads (of 4 consecutive values) per thread in flight
constexpr int kSelectBatch = 4;          // candidates per thread that share one reservation of places in the result
// Quads in the sample of the streaming kernel with CTAs of that size.  A larger sample leaves fewer candidates to rank, a smaller one
// is sooner done: rows of 32768 to 65536 values with CTAs of 256 threads, 512 | 1024 quads, 4096 x 32768, k 2048 121 | 128 us,
// k 512 100 | 111 us; 4096 x 65536, k 1024 132 | 142 us.
// All that holds for values independent of their neighbours.  Where they vary smoothly along the row, the 32 values of a run count for
// less, and a row is misjudged (and read twice more) oftener, with either size alike.  Share of such rows among moving sums of L
// independent values, 32768 to 262144 wide, k 512 to 2048: none up to L 4, 0-2 % at 8, 4-8 % at 16, 10-20 % at 32, 18-31 % at 128.
// L 1 | 8 | 32 | 128, us (in brackets with 1024 quads for all CTAs, in the kernel before):
//   4096 x 32768, k 2048  117 | 152 | 193 | 210 (137 | 173 | 227 | 230)     k 512  98 | 127 | 166 | 191 (111 | 142 | 180 | 202)
//   4096 x 65536, k 1024  182 | 242 | 303 | 352 (195 | 255 | 333 | 385)     496 x 262144, k 512  92 | 203 | 239 | 257 (101 | 227 | 313 | 361)
__host__ __device__ constexpr int sample_quads(int threads) { return threads >= 512 ? 1024 : 512; }

struct TopkParams {
    const float* logits;
    int64_t stride0, stride1;
    int32_t* indices;  // [num_rows, top_k]
    int32_t num_rows, vocab, top_k;
    uint32_t capacity;  // of the candidate pool
    bool sampled;       // top_k is small enough for it
    bool ahead;         // the streaming kernel sends batches to L2 ahead of their loads
    int32_t length_shift;  // where it takes the rows in the order of their lengths: which brings the width below 64
    // decode
    const int32_t* seq_lens;
    int32_t next_n;
    // prefill
    const int32_t* row_starts;  // null: every range starts at 0
    const int32_t* row_ends;
};

// Unsigned key with the order of the float values (negative values below positive ones, -0 below +0, a NaN above +inf or, with
// its sign bit set, below -inf).
__device__ __forceinline__ uint32_t order_key(uint32_t bits) { return bits ^ (static_cast<uint32_t>(static_cast<int32_t>(bits) >> 31) | 0x80000000u); }

// Coarse monotone code: the top 11 bits of the order key of the value rounded to fp16.  The sign is the value's own: the
// conversion drops that of a NaN, and the code has to order NaNs as order_key() does (the top one or the bottom one).
__device__ __forceinline__ uint32_t coarse_bin(float x) {
    const uint32_t sign = static_cast<uint32_t>(__float_as_int(x) >> 31);  // all ones or zero
    const uint32_t h = __half_as_ushort(__float2half_rn(fabsf(x)));
    return ((h ^ sign ^ 0x8000u) & 0xffffu) >> 5;
}

// The same for two values, x in the low half of the result.
__device__ __forceinline__ uint32_t coarse_bins(float x, float y) {
    uint32_t magnitudes, signs, bins;
    asm("{.reg .f32 a, b;\n"
        "abs.f32 a, %1;\n"
        "abs.f32 b, %2;\n"
        "cvt.rn.f16x2.f32 %0, b, a;}"
        : "=r"(magnitudes)
        : "f"(x), "f"(y));
    asm("prmt.b32 %0, %1, %2, 0xffbb;" : "=r"(signs) : "r"(__float_as_uint(x)), "r"(__float_as_uint(y)));  // each sign 16 times
    bins = ((magnitudes ^ signs ^ 0x80008000u) >> 5) & 0x07ff07ffu;
    return bins;
}
constexpr uint32_t kBinOfMinusInfinity = 31;  // below it lie the NaNs with their sign bit set only

// A value whose coarse code is `bin`, the lowest one up to the rounding to fp16; -inf for the codes below it.
__device__ __forceinline__ float value_of_bin(uint32_t bin) {
    uint32_t key = bin << 5;
    key = key < 0x0400u ? 0x03ffu : key;  // -inf
    key = key > 0xfc00u ? 0xfc00u : key;  // +inf
    const uint32_t h = (key & 0x8000u) ? key & 0x7fffu : ~key & 0xffffu;
    return __half2float(__ushort_as_half(static_cast<unsigned short>(h)));
}

// State the threads of a CTA share, apart from the candidates.
struct Shared {
    __align__(16) uint32_t hist[kBins];  // later the dense list of the candidates of one bin: kBins / 2 (key, position) pairs
    uint32_t scratch[32];
    uint32_t result[4];
    uint32_t counters[4];  // 0: emitted, 1: collected, 2: ties taken / dense candidates, 3: largest key of the sample
    uint32_t pooled;  // candidates in the pool
};

struct Threshold {
    uint32_t bin;    // the bin holding the k-th largest element
    uint32_t need;   // how many elements of that bin belong to the top k
    uint32_t count;  // how many elements that bin holds
};

// The bin, counted from the top, in which the running count reaches `want` (1 <= want <= total of hist).
// All threads call it; ends with a barrier.
template <int THREADS>
__device__ __forceinline__ Threshold find_threshold(Shared& s, uint32_t want) {
    constexpr int kPerThread = kBins / THREADS;  // thread 0 owns the highest bins
    constexpr int kWarps = THREADS / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t local[kPerThread], sum = 0;
#pragma unroll
    for (int j = 0; j < kPerThread; j += 4) {
        const uint4 v = *reinterpret_cast<const uint4*>(&s.hist[kBins - 4 - (tid * kPerThread + j)]);
        local[j] = v.w, local[j + 1] = v.z, local[j + 2] = v.y, local[j + 3] = v.x;
        sum += v.x + v.y + v.z + v.w;
    }
    uint32_t incl = sum;
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) {
        const uint32_t up = __shfl_up_sync(0xffffffffu, incl, m);
        if (lane >= m) incl += up;
    }
    if (lane == 31) s.scratch[warp] = incl;
    __syncthreads();
    // every warp adds up the totals of the warps in front of it
    uint32_t before = lane < warp && lane < kWarps ? s.scratch[lane] : 0u;
    before = __reduce_add_sync(0xffffffffu, before);
    uint32_t above = before + incl - sum;  // elements in bins higher than this thread's
    if (above < want && want <= above + sum) {
#pragma unroll
        for (int j = 0; j < kPerThread; ++j) {
            if (above < want && want <= above + local[j]) {
                s.result[0] = kBins - 1 - (tid * kPerThread + j);
                s.result[1] = want - above;
                s.result[2] = local[j];
            }
            above += local[j];
        }
    }
    __syncthreads();
    Threshold t;
    t.bin = s.result[0], t.need = s.result[1], t.count = s.result[2];
    return t;
}

// The same by one warp (all its lanes call it), 32 bins at a time: from bin `start` down until the running count reaches
// `want` >= 1.  One warp's work instead of the CTA's, and short where the bin lies near the start.
__device__ __forceinline__ Threshold scan_down(const uint32_t* hist, int start, uint32_t want) {
    const int lane = threadIdx.x & 31;
    Threshold t{0u, 1u, 1u};
    uint32_t above = 0u;
    for (int top = start; top >= 0; top -= 32) {
        const uint32_t mine = top - lane >= 0 ? hist[top - lane] : 0u;
        const uint32_t total = __reduce_add_sync(0xffffffffu, mine);
        if (above + total < want) {
            above += total;
            continue;
        }
        uint32_t incl = mine;
#pragma unroll
        for (int m = 1; m < 32; m <<= 1) {
            const uint32_t up = __shfl_up_sync(0xffffffffu, incl, m);
            if (lane >= m) incl += up;
        }
        const int at = __ffs(__ballot_sync(0xffffffffu, above + incl >= want)) - 1;
        t.bin = static_cast<uint32_t>(top - at);
        t.count = __shfl_sync(0xffffffffu, mine, at);
        t.need = want - (above + __shfl_sync(0xffffffffu, incl - mine, at));
        break;
    }
    return t;
}

// The same from bin 0 up: `skip` elements are left out, the next one is the smallest of those selected.
__device__ __forceinline__ Threshold scan_up(const uint32_t* hist, uint32_t skip) {
    const int lane = threadIdx.x & 31;
    Threshold t{kBins - 1u, 1u, 1u};
    uint32_t below = 0u;
    for (int b = 0; b < kBins; b += 32) {
        const uint32_t mine = hist[b + lane];
        const uint32_t total = __reduce_add_sync(0xffffffffu, mine);
        if (below + total <= skip) {
            below += total;
            continue;
        }
        uint32_t incl = mine;
#pragma unroll
        for (int m = 1; m < 32; m <<= 1) {
            const uint32_t up = __shfl_up_sync(0xffffffffu, incl, m);
            if (lane >= m) incl += up;
        }
        const int at = __ffs(__ballot_sync(0xffffffffu, below + incl > skip)) - 1;
        t.bin = static_cast<uint32_t>(b + at);
        t.count = __shfl_sync(0xffffffffu, mine, at);
        t.need = t.count - (skip - (below + __shfl_sync(0xffffffffu, incl - mine, at)));
        break;
    }
    return t;
}

template <int THREADS>
__device__ __forceinline__ void clear_histogram(Shared& s) {
    for (int i = threadIdx.x; i < kBins / 4; i += THREADS) reinterpret_cast<uint4*>(s.hist)[i] = make_uint4(0u, 0u, 0u, 0u);
}

// Appends `value` of the lanes whose `take` is set to list[], one atomic per warp.  Whole warps call it.
__device__ __forceinline__ void append(int32_t* list, uint32_t* counter, bool take, int32_t value) {
    const uint32_t mask = __ballot_sync(0xffffffffu, take);
    if (mask == 0u) return;
    const int lane = threadIdx.x & 31;
    uint32_t base = 0u;
    if (lane == 0) base = atomicAdd(counter, __popc(mask));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (take) list[base + __popc(mask & ((1u << lane) - 1u))] = value;
}

// Histogram increment shared by the lanes of a warp that hit the same bin (degenerate inputs put a whole warp
// into one bin, which plain shared-memory atomics would serialise).
__device__ __forceinline__ void add_aggregated(uint32_t* hist, uint32_t bin, bool active) {
    const uint32_t mask = __ballot_sync(0xffffffffu, active);
    if (!active) return;
    const uint32_t peers = __match_any_sync(mask, bin);
    if ((threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&hist[bin], __popc(peers));
}

// The `want` largest of the n candidates (key, position) in shared memory; their positions are appended to out
// through counters[0], ties at the smallest selected key through counters[2] (zero on entry).  Radix selection in digits of
// up to 11 bits on key - min(key), starting at the highest bit in which the candidates differ at all (they share sign,
// exponent and leading mantissa bits, which a selection on fixed bit positions would waste passes and atomic
// conflicts on).
template <int THREADS>
__device__ __noinline__ void select_radix(Shared& s, const uint2* cand, uint32_t n, uint32_t want, int32_t* out) {
    const int tid = threadIdx.x;
    __syncthreads();
    if (want >= n) {
        for (uint32_t i = tid; i < n; i += THREADS) out[atomicAdd(&s.counters[0], 1u)] = static_cast<int32_t>(cand[i].y);
        return;
    }
    // range of the keys
    if (tid == 0) s.result[0] = 0xffffffffu, s.result[1] = 0u;
    __syncthreads();
    uint32_t lo = 0xffffffffu, hi = 0u;
    for (uint32_t i = tid; i < n; i += THREADS) {
        const uint32_t key = cand[i].x;
        lo = key < lo ? key : lo, hi = key > hi ? key : hi;
    }
    lo = __reduce_min_sync(0xffffffffu, lo), hi = __reduce_max_sync(0xffffffffu, hi);
    if ((tid & 31) == 0) atomicMin(&s.result[0], lo), atomicMax(&s.result[1], hi);
    __syncthreads();
    const uint32_t base = s.result[0], range = s.result[1] - s.result[0];
    __syncthreads();
    uint32_t need = want, prefix = 0u, prefix_mask = 0u;
    int top = 32 - __clz(range | 1u);  // bits of (key - base) that can be set
    while (top > 0) {
        const int shift = top > 11 ? top - 11 : 0;
        const uint32_t digit_mask = (1u << (top - shift)) - 1u;
        clear_histogram<THREADS>(s);
        __syncthreads();
        for (uint32_t i = tid; i < n; i += THREADS) {
            const uint32_t rel = cand[i].x - base;
            if ((rel & prefix_mask) == prefix) atomicAdd(&s.hist[(rel >> shift) & digit_mask], 1u);
        }
        __syncthreads();
        const Threshold t = find_threshold<THREADS>(s, need);
        prefix |= t.bin << shift;
        prefix_mask |= digit_mask << shift;
        need = t.need;
        top = shift;
        if (t.need == t.count) break;  // every candidate with this prefix is taken: the lower bits do not matter
    }
    // keys above the prefix (on the bits examined) are in; `need` of those equal to it are in
    for (uint32_t i = tid; i < n; i += THREADS) {
        const uint2 e = cand[i];
        const uint32_t rel_hi = (e.x - base) & prefix_mask;
        if (rel_hi > prefix || (rel_hi == prefix && atomicAdd(&s.counters[2], 1u) < need)) out[atomicAdd(&s.counters[0], 1u)] = static_cast<int32_t>(e.y);
    }
}

// The `want` largest of n candidates by counting: a candidate's rank is the number of candidates ahead of it in the
// total order (key descending, position ascending); one pass, no histogram.
template <int THREADS>
__device__ __forceinline__ void rank_by_counting(Shared& s, const uint2* dense, uint32_t n, uint32_t want, int32_t* out) {
    for (uint32_t a = threadIdx.x; a < n; a += THREADS) {
        const uint2 e = dense[a];
        uint32_t ahead = 0u;
#pragma unroll 4
        for (uint32_t b = 0; b < n; ++b) {
            const uint2 o = dense[b];  // the same address for all lanes: a broadcast
            ahead += (o.x > e.x || (o.x == e.x && o.y < e.y)) ? 1u : 0u;
        }
        if (ahead < want) out[atomicAdd(&s.counters[0], 1u)] = static_cast<int32_t>(e.y);
    }
}

__device__ __forceinline__ float4 load_quad(const float* p) {
    const uint4 q = ld_stream16(p);
    return make_float4(__uint_as_float(q.x), __uint_as_float(q.y), __uint_as_float(q.z), __uint_as_float(q.w));
}

// The valid range of a row, seen as 16-byte quads of 4 consecutive values counted from the 16-byte boundary at or below its
// first value (`lead` = values between the two).  Rows whose values are not adjacent have lead 0 and are loaded value by value.
struct Row {
    const float* x;
    int64_t stride;
    int32_t len, lead, quads;

    __device__ __forceinline__ Row(const float* first, int64_t stride1, int32_t length) : x(first), stride(stride1), len(length), lead(0) {
        if (stride1 == 1) lead = static_cast<int32_t>((reinterpret_cast<uintptr_t>(first) & 15u) >> 2);
        quads = (len + lead + 3) >> 2;
    }
    // Quads [first_whole(), end_whole()) lie inside the row and are one 16-byte load each.
    __device__ __forceinline__ int32_t first_whole() const { return stride != 1 ? quads : lead > 0 ? 1 : 0; }
    __device__ __forceinline__ int32_t end_whole() const { return stride != 1 ? quads : (len + lead) >> 2; }
    __device__ __forceinline__ float value(int32_t i) const { return __uint_as_float(ld_stream4(x + static_cast<int64_t>(i) * stride)); }
    __device__ __forceinline__ int32_t position(int32_t quad) const { return 4 * quad - lead; }  // of the quad's first value
    // Values outside the row are -inf (their positions tell them from values that are).
    __device__ __forceinline__ float4 load(int32_t quad) const {
        const int32_t p = position(quad);
        if (stride == 1 && p >= 0 && p + 4 <= len) return load_quad(x + p);
        return make_float4(edge(p), edge(p + 1), edge(p + 2), edge(p + 3));
    }
    __device__ __forceinline__ bool inside(int32_t i) const { return static_cast<uint32_t>(i) < static_cast<uint32_t>(len); }
    __device__ __forceinline__ float edge(int32_t i) const { return inside(i) ? value(i) : -INFINITY; }
};

// The candidates a CTA has found: (bits of the value, position) pairs in shared memory.  `size` counts past `capacity` when
// it does not hold all of them.
struct Pool {
    uint2* entries;
    uint32_t* size;
    uint32_t capacity;

    // Takes the values of N quads per lane that reach `floor` (> -inf); quad u holds the positions from p + u * step on, and what
    // is no part of the row is -inf.  NaNs of either sign are taken: one with its sign bit clear is among the largest values, one
    // with it set is sorted out by select().  Whole warps call it: a lane marks its candidates, the warp adds up their numbers and
    // reserves room with one atomic, the lane writes them.
    template <int N>
    __device__ __forceinline__ void take(const float4 (&v)[N], int32_t p, int32_t step, float floor) const {
        static_assert(N <= 4, "one bit per value");
        const int lane = threadIdx.x & 31;
        // Bit 4N - 1 - i: value i is below the floor, by the sign of their difference (of a NaN it is +).  Two differences an
        // instruction and one instruction a value to shift the sign in, where a comparison and a predicated addition were two.
        uint64_t minus_floor;
        asm("{.reg .f32 n; neg.f32 n, %1; mov.b64 %0, {n, n};}" : "=l"(minus_floor) : "f"(floor));
        uint32_t below = 0u;
        const auto push = [&](float a, float b) {
            uint64_t d;
            asm("{.reg .b64 t; mov.b64 t, {%1, %2}; add.rn.f32x2 %0, t, %3;}" : "=l"(d) : "f"(a), "f"(b), "l"(minus_floor));
            below = __funnelshift_l(static_cast<uint32_t>(d), below, 1);
            below = __funnelshift_l(static_cast<uint32_t>(d >> 32), below, 1);
        };
#pragma unroll
        for (int u = 0; u < N; ++u) push(v[u].x, v[u].y), push(v[u].z, v[u].w);
        const uint32_t marks = ~below & ((1u << (4 * N)) - 1u), mine = __popc(marks);
        uint32_t upto = mine;
#pragma unroll
        for (int m = 1; m < 32; m <<= 1)
            asm volatile(
                "{.reg .u32 r;\n"
                ".reg .pred t;\n"
                "shfl.sync.up.b32 r|t, %0, %1, 0, 0xffffffff;\n"
                "@t add.u32 %0, %0, r;}"
                : "+r"(upto)
                : "r"(m));
        uint32_t at = 0u;
        if (lane == 31 && upto > 0u) at = atomicAdd(size, upto);
        at += upto;  // lane 31: the end of the warp's part
        const uint32_t end = __shfl_sync(0xffffffffu, at, 31), total = __shfl_sync(0xffffffffu, upto, 31);
        if (total == 0u || end > capacity) return;
        uint32_t address = static_cast<uint32_t>(__cvta_generic_to_shared(entries + (end - total + upto - mine)));
#pragma unroll
        for (int u = 0; u < N; ++u) {
            const float e[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (marks & (1u << (4 * (N - u) - 1 - j))) {
                    asm volatile("st.shared.f32 [%0], %1; st.shared.u32 [%0+4], %2;" ::"r"(address), "f"(e[j]), "r"(p + u * step + j) : "memory");
                    address += sizeof(uint2);
                }
        }
    }
};

// Bin of a candidate in the histogram that ranks them: linear in the key from `anchor` on, the first and the last bin open.
__device__ __forceinline__ uint32_t fine_bin(uint32_t key, uint32_t anchor, int shift) {
    return min((max(key, anchor) - anchor) >> shift, kBins - 1u);
}
// 2048 bins between the key candidates start at and one near the top of the row (the largest of the sample) leave a handful
// of candidates in the bin of the k-th largest.
__device__ __forceinline__ int fine_shift(uint32_t floor_key, uint32_t top_key) {
    const int bits = 32 - __clz(top_key > floor_key ? top_key - floor_key : 1u);
    return bits > 11 ? bits - 11 : 0;
}

// What the sample says: the value to collect from, its key, and the anchor and shift of fine_bin().  The sample is in hist and its largest
// key in counters[3], a barrier ago; `size` values of it stand for `len` values of the row.  Clears hist; the caller's next
// barrier completes that.
struct Floor {
    float value;
    uint32_t key, anchor;
    int shift;
};
template <int THREADS>
__device__ __forceinline__ Floor floor_from_sample(Shared& s, int32_t k, int32_t size, int32_t len) {
    if (threadIdx.x < 32) {
        // rank inside the sample that stands for k values of the row, plus four standard deviations of that count
        const float mean = static_cast<float>(k) * static_cast<float>(size) / static_cast<float>(len);
        const uint32_t rank = static_cast<uint32_t>(mean + 4.0f * sqrtf(mean)) + 3u;
        const uint32_t limit = static_cast<uint32_t>(size);
        const uint32_t top_key = s.counters[3];
        const uint32_t bin = scan_down(s.hist, coarse_bin(__uint_as_float((top_key & 0x80000000u) ? top_key & 0x7fffffffu : ~top_key)), rank < limit ? rank : limit).bin;
        if (threadIdx.x == 0) {
            const uint32_t bits = __float_as_uint(value_of_bin(bin));
            // a row hardly longer than k: all finite values are candidates (no more of them than expected)
            s.result[0] = rank < limit ? bits : 0xff7fffffu;
            s.result[1] = order_key(bits), s.result[2] = fine_shift(order_key(bits), top_key);
        }
    }
    __syncthreads();
    Floor f;
    f.value = __uint_as_float(s.result[0]), f.key = order_key(s.result[0]), f.anchor = s.result[1], f.shift = static_cast<int>(s.result[2]);
    clear_histogram<THREADS>(s);
    return f;
}

// Histogram route: two reads of the row by one CTA, any k, any distribution.  `cand` holds `capacity` pairs.
template <int THREADS>
__device__ __noinline__ void select_from_histogram(Shared& s, uint2* cand, uint32_t capacity, const Row row, int32_t k, int32_t* out) {
    const int tid = threadIdx.x;
    __syncthreads();
    clear_histogram<THREADS>(s);
    if (tid < 4) s.counters[tid] = 0u;
    __syncthreads();
    // four quads per thread in flight; whole warps stay together for append()
    const auto for_each_quad = [&](auto&& visit) {
        for (int32_t q = tid; q - (tid & 31) < row.quads; q += kStreamBatch * THREADS) {
            float4 v[kStreamBatch];
#pragma unroll
            for (int u = 0; u < kStreamBatch; ++u)
                if (q + u * THREADS < row.quads) v[u] = row.load(q + u * THREADS);
#pragma unroll
            for (int u = 0; u < kStreamBatch; ++u) {
                const int32_t p = q + u * THREADS < row.quads ? row.position(q + u * THREADS) : -8;
                visit(v[u].x, p), visit(v[u].y, p + 1), visit(v[u].z, p + 2), visit(v[u].w, p + 3);
            }
        }
    };
    for_each_quad([&](float v, int32_t i) {
        if (row.inside(i)) atomicAdd(&s.hist[coarse_bin(v)], 1u);
    });
    __syncthreads();
    const Threshold coarse = find_threshold<THREADS>(s, static_cast<uint32_t>(k));
    const bool collect_bin = coarse.count <= capacity && coarse.need < coarse.count;
    const bool take_all = coarse.need == coarse.count;  // the whole bin belongs to the top k
    // emit everything above the bin (and the bin itself if it is taken whole); collect the bin's candidates
    for_each_quad([&](float v, int32_t i) {
        const uint32_t c = coarse_bin(v);
        append(out, &s.counters[0], row.inside(i) && (c > coarse.bin || (take_all && c == coarse.bin)), i);
        if (row.inside(i) && collect_bin && c == coarse.bin) cand[atomicAdd(&s.counters[1], 1u)] = make_uint2(order_key(__float_as_uint(v)), static_cast<uint32_t>(i));
    });
    if (take_all) return;
    if (collect_bin) {
        select_radix<THREADS>(s, cand, coarse.count, coarse.need, out);
        return;
    }
    // The bin is too crowded for shared memory.  Radix selection on the fp32 key over the row itself, restricted to the
    // elements of the bin: bits 31-21, 20-10, 9-0.
    uint32_t need = coarse.need, prefix = 0u, prefix_mask = 0u;
    const int shifts[3] = {21, 10, 0};
    const uint32_t widths[3] = {11, 11, 10};
    for (int pass = 0; pass < 3; ++pass) {
        __syncthreads();
        clear_histogram<THREADS>(s);
        __syncthreads();
        for (int32_t i = tid; i - (tid & 31) < row.len; i += THREADS) {  // whole warps stay together for the aggregated increment
            bool active = false;
            uint32_t bin = 0u;
            if (i < row.len) {
                const float v = row.value(i);
                const uint32_t key = order_key(__float_as_uint(v));
                active = coarse_bin(v) == coarse.bin && (key & prefix_mask) == prefix;
                bin = (key >> shifts[pass]) & ((1u << widths[pass]) - 1u);
            }
            add_aggregated(s.hist, bin, active);
        }
        __syncthreads();
        const Threshold t = find_threshold<THREADS>(s, need);
        prefix |= t.bin << shifts[pass];
        prefix_mask |= ((1u << widths[pass]) - 1u) << shifts[pass];
        need = t.need;
    }
    for (int32_t i = tid; i < row.len; i += THREADS) {
        const float v = row.value(i);
        if (coarse_bin(v) != coarse.bin) continue;
        const uint32_t key = order_key(__float_as_uint(v));
        if (key > prefix || (key == prefix && atomicAdd(&s.counters[2], 1u) < need)) out[atomicAdd(&s.counters[0], 1u)] = i;
    }
}

// Ranks the `size` candidates and emits the k largest; false (in every thread) when the pool does not hold them.  hist and the
// counters are zero on entry, a barrier ago or more.  A negative NaN, the smallest key, may be among the candidates: where the
// k-th largest is so near the floor that it could count, the pool does not do.
template <int THREADS>
__device__ __forceinline__ bool select(Shared& s, const uint2* pool, uint32_t size, uint32_t capacity, uint32_t k, const Floor& f, int32_t* out) {
    const int tid = threadIdx.x;
    const uint32_t floor_key = f.key;
    if (size < k || size > capacity) return false;
#pragma unroll 4
    for (uint32_t i = tid; i < size; i += THREADS) atomicAdd(&s.hist[fine_bin(order_key(pool[i].x), f.anchor, f.shift)], 1u);
    __syncthreads();
    Threshold t;
    if (f.shift > 16) {  // the bins cover many octaves: the candidates reach down to values near zero
        t = find_threshold<THREADS>(s, k);
    } else {
        if (tid < 32) {
            t = scan_up(s.hist, size - k);
            if (tid == 0) s.result[0] = t.bin, s.result[1] = t.need, s.result[2] = t.count;
        }
        __syncthreads();
        t.bin = s.result[0], t.need = s.result[1], t.count = s.result[2];
    }
    if (t.bin == 0u) {  // where keys below the floor would be, and are not told apart
        bool strays = false;
        for (uint32_t i = tid; i < size; i += THREADS) strays |= order_key(pool[i].x) < floor_key;
        if (__syncthreads_or(strays)) return false;
    }
    const bool take_all = t.need == t.count;
    if (!take_all && t.count > kCountingMax) return false;
    // The bins as ranges of keys: above `untaken` a candidate is selected, above `below` (and not above `untaken`) it is in the
    // bin of the k-th largest.  The first bin begins at the floor, the last one has no end.
    const auto last_before = [&](uint32_t bin) {
        if (bin >= kBins) return 0xffffffffu;
        const uint32_t start = f.anchor + (bin << f.shift);
        if (start < f.anchor) return 0xffffffffu;  // past the largest key there is
        return (bin == 0u || start < floor_key ? floor_key : start) - 1u;
    };
    const uint32_t untaken = last_before(take_all ? t.bin : t.bin + 1u), below = last_before(t.bin);
    uint2* dense = reinterpret_cast<uint2*>(s.hist);  // the histogram is no longer needed
    const int lane = tid & 31;
    for (uint32_t i0 = tid; i0 - lane < size; i0 += kSelectBatch * THREADS) {  // whole warps stay together
        uint32_t key[kSelectBatch], at = 0u;
        int32_t position[kSelectBatch];
#pragma unroll
        for (int u = 0; u < kSelectBatch; ++u) {
            const uint32_t i = i0 + u * THREADS;
            key[u] = 0u, position[u] = 0;
            if (i < size) {
                const uint2 e = pool[i];
                key[u] = order_key(e.x), position[u] = static_cast<int32_t>(e.y);
            }
            if (key[u] > untaken) ++at;
        }
        const uint32_t mine = at;
#pragma unroll
        for (int m = 1; m < 32; m <<= 1) {
            const uint32_t up = __shfl_up_sync(0xffffffffu, at, m);
            if (lane >= m) at += up;
        }
        uint32_t base = 0u;
        if (lane == 31 && at > 0u) base = atomicAdd(&s.counters[0], at);
        int32_t* to = out + (__shfl_sync(0xffffffffu, base, 31) + at - mine);
#pragma unroll
        for (int u = 0; u < kSelectBatch; ++u) {
            if (key[u] > untaken) *to++ = position[u];
            else if (key[u] > below) dense[atomicAdd(&s.counters[2], 1u)] = make_uint2(key[u], static_cast<uint32_t>(position[u]));
        }
    }
    if (take_all) return true;
    __syncthreads();
    rank_by_counting<THREADS>(s, dense, t.count, t.need, out);
    return true;
}

// The valid range of row `r`: its first value's index and its length.
template <bool DECODE>
__device__ __forceinline__ int32_t row_range(const TopkParams& p, int r, int64_t* first) {
    int64_t start, end;
    if (DECODE) {
        start = 0;
        const int request = p.next_n == 1 ? r : r / p.next_n;
        end = static_cast<int64_t>(p.seq_lens[request]) - p.next_n + (r - request * p.next_n) + 1;
    } else {
        start = p.row_starts ? p.row_starts[r] : 0;
        end = p.row_ends[r];
    }
    start = start < 0 ? 0 : start;
    end = end > p.vocab ? p.vocab : end;
    *first = start;
    return end > start ? static_cast<int32_t>(end - start) : 0;
}

// One CTA per row, no sample: the coarse histogram of all values gives the bin of the k-th largest, what lies above it is emitted, and
// the values of the bin are ranked by counting.  For short rows, of which a large part is selected.  Bound by instruction issue, so
// two values travel in one register from the conversion to fp16 on: their codes are compared by an addition that carries into
// bit 15 and bit 31, and the values themselves are not kept (the few that are ranked are read once more).
// 4096 x 4096, k 512: 9.4 k -> 6.2 k warp instructions a row, 45.6 -> 29.9 us; 4096 x 2048 27.1 -> 18.9 us; 1531 x 2600 14.6 -> 10.8 us;
// 61 x 4096 4.2 -> 3.8 us.  Values beside the row count as -inf, which only matters where the k-th largest is that small: such rows
// take the histogram route.  4096 x 1400, k 512, 400 finite values a row and -inf or the lowest float behind them: 73 us, where rows of
// finite values take 20 us (ranking the thousand equal values by counting took 1267 us); 61 x 1400 7.4 and 3.0 us; 4096 x 4096, where
// they are too many for the pool, 201 and 30 us.
template <bool DECODE, int THREADS, int QUADS>
__global__ void __launch_bounds__(THREADS, 1536 / THREADS) topk_short_kernel(const Launched<TopkParams> p) {
    begin_dependent_kernel();
    __shared__ Shared s;
    extern __shared__ uint2 dynamic[];
    constexpr int kPairs = 2 * QUADS;
    static_assert(kPairs <= 8, "a pair has one bit in either half of a word, from bits 15 and 31 down");
    const int tid = threadIdx.x, lane = tid & 31;
    const int r = blockIdx.x;
    int64_t first;
    const int32_t len = row_range<DECODE>(p, r, &first);
    const int32_t k = len < p.top_k ? len : p.top_k;
    int32_t* out = p.indices + static_cast<int64_t>(r) * p.top_k;
    for (int i = k + tid; i < p.top_k; i += THREADS) out[i] = -1;
    if (len <= p.top_k) {  // everything is selected
        for (int i = tid; i < len; i += THREADS) out[i] = i;
        return;
    }
    const Row row(p.logits + static_cast<int64_t>(r) * p.stride0 + first * p.stride1, p.stride1, len);
    const int32_t begin = row.first_whole(), whole = row.end_whole() - begin;
    float4 v[QUADS];
#pragma unroll
    for (int u = 0; u < QUADS; ++u) {
        const int32_t quad = tid + u * THREADS;
        if (static_cast<uint32_t>(quad - begin) < static_cast<uint32_t>(whole)) v[u] = load_quad(row.x + row.position(quad));
        else if (quad < row.quads) v[u] = row.load(quad);
        else v[u] = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
    }
    clear_histogram<THREADS>(s);
    if (tid < 4) s.counters[tid] = 0u;
    __syncthreads();
    const auto beyond = [&](int pair) { return (tid & ~31) + (pair >> 1) * THREADS >= row.quads; };  // nothing of it for the warp
    uint32_t bins[kPairs], largest = 0u;
#pragma unroll
    for (int j = 0; j < kPairs; ++j) {
        bins[j] = 0u;
        if (beyond(j)) continue;
        bins[j] = j & 1 ? coarse_bins(v[j >> 1].z, v[j >> 1].w) : coarse_bins(v[j >> 1].x, v[j >> 1].y);
        atomicAdd(&s.hist[bins[j] & 0xffffu], 1u), atomicAdd(&s.hist[bins[j] >> 16], 1u);
        asm("max.u16x2 %0, %0, %1;" : "+r"(largest) : "r"(bins[j]));
    }
    largest = __reduce_max_sync(0xffffffffu, max(largest & 0xffffu, largest >> 16));
    if (lane == 0) atomicMax(&s.counters[3], largest);
    __syncthreads();
    Threshold t;
    if (4 * k > len) {  // far from the top, perhaps behind the many bins of values near zero
        t = find_threshold<THREADS>(s, static_cast<uint32_t>(k));
    } else {
        if (tid < 32) {
            t = scan_down(s.hist, static_cast<int>(s.counters[3]), static_cast<uint32_t>(k));
            if (tid == 0) s.result[0] = t.bin, s.result[1] = t.need, s.result[2] = t.count;
        }
        __syncthreads();
        t.bin = s.result[0], t.need = s.result[1], t.count = s.result[2];
    }
    const bool take_all = t.need == t.count;
    if (t.bin <= kBinOfMinusInfinity || (!take_all && t.count > kCountingMax)) {
        select_from_histogram<THREADS>(s, dynamic, p.capacity, row, k, out);
        return;
    }
    // pair j: bit 15 - j for its first value, bit 31 - j for its second
    const auto at_least = [&](uint32_t bin) {
        const uint32_t up = (0x8000u - bin) * 0x10001u;
        uint32_t marks = 0u;
#pragma unroll
        for (int j = 0; j < kPairs; ++j) marks |= ((bins[j] + up) >> j) & (0x80008000u >> j);
        return marks;
    };
    uint2* dense = reinterpret_cast<uint2*>(s.hist);  // the histogram is no longer needed
    const uint32_t reach = at_least(t.bin), taken = take_all ? reach : at_least(t.bin + 1u);  // of the bins taken whole
    uint32_t at = __popc(taken);
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) {
        const uint32_t up = __shfl_up_sync(0xffffffffu, at, m);
        if (lane >= m) at += up;
    }
    uint32_t base = 0u;
    if (lane == 31 && at > 0u) base = atomicAdd(&s.counters[0], at);
    at += __shfl_sync(0xffffffffu, base, 31) - __popc(taken);
    const auto position = [&](int pair) { return row.position(tid + (pair >> 1) * THREADS) + 2 * (pair & 1); };
#pragma unroll
    for (int j = 0; j < kPairs; ++j) {
        if (beyond(j)) continue;
        if (taken & (0x8000u >> j)) out[at++] = position(j);
        if (taken & (0x80000000u >> j)) out[at++] = position(j) + 1;
    }
    if (take_all) return;
    for (uint32_t left = reach & ~taken; left;) {
        const int bit = 31 - __clz(left);
        left ^= 1u << bit;
        const int32_t i = position(15 - (bit & 15)) + (bit >> 4);
        dense[atomicAdd(&s.counters[2], 1u)] = make_uint2(order_key(__float_as_uint(row.value(i))), static_cast<uint32_t>(i));
    }
    __syncthreads();
    rank_by_counting<THREADS>(s, dense, t.count, t.need, out);
}

// One CTA per row, the row in registers: QUADS x 4 values per thread.  The sample is the first value of every quad.
template <bool DECODE, int THREADS, int QUADS>
__global__ void __launch_bounds__(THREADS) topk_registers_kernel(const Launched<TopkParams> p) {
    begin_dependent_kernel();
    __shared__ Shared s;
    extern __shared__ uint2 dynamic[];
    const int tid = threadIdx.x;
    const int r = blockIdx.x;
    int64_t first;
    const int32_t len = row_range<DECODE>(p, r, &first);
    const int32_t k = len < p.top_k ? len : p.top_k;
    int32_t* out = p.indices + static_cast<int64_t>(r) * p.top_k;
    for (int i = k + tid; i < p.top_k; i += THREADS) out[i] = -1;
    if (len <= p.top_k) {  // everything is selected
        for (int i = tid; i < len; i += THREADS) out[i] = i;
        return;
    }
    const Row row(p.logits + static_cast<int64_t>(r) * p.stride0 + first * p.stride1, p.stride1, len);
    float4 v[QUADS];
#pragma unroll
    for (int u = 0; u < QUADS; ++u) {
        const int32_t quad = tid + u * THREADS;
        v[u] = quad < row.quads ? row.load(quad) : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
    }
    clear_histogram<THREADS>(s);
    if (tid < 4) s.counters[tid] = 0u;
    if (tid == 4) s.pooled = 0u;
    __syncthreads();
    uint32_t largest = 0u;
#pragma unroll
    for (int u = 0; u < QUADS; ++u) {
        const int32_t quad = tid + u * THREADS;
        if (row.inside(row.position(quad))) {
            atomicAdd(&s.hist[coarse_bin(v[u].x)], 1u);
            const uint32_t key = order_key(__float_as_uint(v[u].x));
            largest = key > largest ? key : largest;
        }
    }
    largest = __reduce_max_sync(0xffffffffu, largest);
    if ((tid & 31) == 0) atomicMax(&s.counters[3], largest);
    __syncthreads();
    const int32_t size = row.quads - (row.lead > 0 ? 1 : 0);  // quads whose first value belongs to the row
    const Floor f = floor_from_sample<THREADS>(s, k, size, len);
    __syncthreads();
    bool done = false;
    if (p.sampled && f.value > -INFINITY) {
        const Pool pool{dynamic, &s.pooled, p.capacity};
        constexpr int kBatch = QUADS < kStreamBatch ? QUADS : kStreamBatch;
#pragma unroll
        for (int u = 0; u < QUADS; u += kBatch) {
            float4 batch[kBatch];
#pragma unroll
            for (int w = 0; w < kBatch; ++w) batch[w] = v[u + w];
            pool.take(batch, row.position(tid + u * THREADS), 4 * THREADS, f.value);
        }
        __syncthreads();
        done = select<THREADS>(s, dynamic, s.pooled, p.capacity, static_cast<uint32_t>(k), f, out);
    }
    if (!done) select_from_histogram<THREADS>(s, dynamic, p.capacity, row, k, out);
}

// The row at `place` in the order of lengths, the longest first: by 64 classes of length and, inside a class, by index, so that every
// CTA finds the same order.  All threads call it; at most kOrderedRows rows.
constexpr int kOrderedRows = 1024;
template <bool DECODE, int THREADS>
__device__ __forceinline__ int row_at_place(Shared& s, const TopkParams& p, uint32_t place) {
    constexpr int kPer = kOrderedRows / THREADS, kWarps = THREADS / 32;
    const int tid = threadIdx.x, lane = tid & 31;
    uint32_t* const classes = s.hist;       // rows per class
    uint32_t* const cells = s.hist + 64;    // rows of the class looked for, by 32 rows
    if (tid < 128) s.hist[tid] = 0u;
    __syncthreads();
    uint32_t mine[kPer];
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const int r = i * THREADS + tid;
        mine[i] = 64u;
        if (r < p.num_rows) {
            int64_t first;
            mine[i] = 63u - min(static_cast<uint32_t>(row_range<DECODE>(p, r, &first)) >> p.length_shift, 63u);
            atomicAdd(&classes[mine[i]], 1u);
        }
    }
    __syncthreads();
    // the class in which the count reaches the place, and the place inside it
    const auto scan = [&](uint32_t a) {
#pragma unroll
        for (int m = 1; m < 32; m <<= 1) {
            const uint32_t up = __shfl_up_sync(0xffffffffu, a, m);
            if (lane >= m) a += up;
        }
        return a;
    };
    const auto find = [&](const uint32_t* counts, uint32_t want, uint32_t* inside) {  // of 64 counts
        const uint32_t a = counts[2 * lane], b = counts[2 * lane + 1], upto = scan(a + b), before = upto - a - b;
        const int at = __ffs(__ballot_sync(0xffffffffu, upto > want)) - 1;
        const uint32_t left = want - __shfl_sync(0xffffffffu, before, at), first = __shfl_sync(0xffffffffu, a, at);
        *inside = left < first ? left : left - first;
        return static_cast<uint32_t>(2 * at) + (left < first ? 0u : 1u);
    };
    uint32_t inside;
    const uint32_t wanted = find(classes, place, &inside);
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const uint32_t votes = __ballot_sync(0xffffffffu, mine[i] == wanted);
        if (lane == 0) cells[i * kWarps + (tid >> 5)] = __popc(votes);
    }
    __syncthreads();
    uint32_t nth;
    const uint32_t cell = find(cells, inside, &nth);
    if (static_cast<int>(cell % kWarps) == (tid >> 5)) {
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            const uint32_t votes = __ballot_sync(0xffffffffu, mine[i] == wanted);
            if (i == static_cast<int>(cell / kWarps) && mine[i] == wanted && __popc(votes & ((1u << lane) - 1u)) == nth) s.result[0] = i * THREADS + tid;
        }
    }
    __syncthreads();
    const int r = static_cast<int>(s.result[0]);
    __syncthreads();
    return r;
}

// TWO: two batches in flight per thread, the next one asked for before this one is looked through: 64 registers, so two CTAs of 512
// threads per SM instead of three, but a CTA by itself runs at about twice the rate (30 x 262144 in clusters of 8: 14.3 -> 11.7 us,
// 60 x 50000, k 1024: 11.4 -> 9.1 us, 100 x 262144, k 2048: 29.5 -> 25.8 us).  LONGEST_FIRST: the CTAs (one per row) take the rows in the
// order of their lengths.  CTAs of 256 threads: five per SM with 48 registers; six with 40 were up to 3 % slower (a causal chunk of
// 4096 x 32768, k 2048 122.5 | 119 us, 1000 x 40000 30.2 | 29.6 us; the pool for k 2048 leaves room for five anyway).
template <bool DECODE, int THREADS, bool TWO, bool LONGEST_FIRST = false>
__global__ void __launch_bounds__(THREADS, THREADS == 256 ? 5 : TWO ? 2 : 3) topk_stream_kernel(const Launched<TopkParams> p) {
    constexpr int kSampleQuads = sample_quads(THREADS);
    begin_dependent_kernel();
    __shared__ Shared s;
    extern __shared__ uint2 dynamic[];  // the candidate pool
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t ctas = cluster.num_blocks(), rank = cluster.block_rank();  // the CTAs of a cluster share one row
    const int tid = threadIdx.x;
    const int r = LONGEST_FIRST ? row_at_place<DECODE, THREADS>(s, p, blockIdx.x) : static_cast<int>(blockIdx.x >> (31 - __clz(ctas)));  // a power of two
    int64_t first;
    const int32_t len = row_range<DECODE>(p, r, &first);
    const int32_t k = len < p.top_k ? len : p.top_k;
    int32_t* out = p.indices + static_cast<int64_t>(r) * p.top_k;
    // Everything up to the first cluster barrier depends on the row only, so the CTAs of a cluster leave together.
    if (rank == 0)
        for (int i = k + tid; i < p.top_k; i += THREADS) out[i] = -1;
    if (len <= p.top_k) {  // everything is selected
        if (rank == 0)
            for (int i = tid; i < len; i += THREADS) out[i] = i;
        return;
    }
    const Row row(p.logits + static_cast<int64_t>(r) * p.stride0 + first * p.stride1, p.stride1, len);
    if (!p.sampled) {
        if (rank == 0) select_from_histogram<THREADS>(s, dynamic, p.capacity, row, k, out);
        return;
    }
    // this CTA's share of the whole quads; its first batch is on its way while the sample is evaluated
    const int32_t begin = row.first_whole(), end = row.end_whole();
    const int32_t share = end > begin ? (end - begin + static_cast<int32_t>(ctas) - 1) / static_cast<int32_t>(ctas) : 0;
    const int32_t from = begin + static_cast<int32_t>(rank) * share, to = from + share < end ? from + share : end;
    const float4 none = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
    int32_t left = to - from - tid;  // quads from this thread's next one to the end of the share
    int32_t position = row.position(from + tid);
    const float* next = row.x + position;
    // every CTA of the cluster takes the same sample: runs of 8 consecutive quads (one 128-byte line each, where the row is
    // so aligned) spread evenly over the row
    const int32_t base = row.stride == 1 ? begin : 0, span = row.stride == 1 ? end - begin : row.quads;
    const auto sampled_quad = [&](int32_t j) {  // runs of 8, each on a multiple of 8
        const int32_t run = j >> 3;
        const int32_t at = span > kSampleQuads ? static_cast<int32_t>(static_cast<uint32_t>((static_cast<uint64_t>(run) * static_cast<uint32_t>(span)) / (kSampleQuads / 8)) & ~7u) : 8 * run;
        return at + (j & 7);
    };
    // The sample is asked for first: everything waits for it, and it came late behind the first batches of a full GPU.  Before -> after, k 512:
    // 496 x 262144 ragged 59.7 -> 58.6 us, full length 92.0 -> 90.7; 592 x 100000 37.2 -> 36.2; 2000 x 17003 39.1 -> 37.6; 4096 x 20001, k 2048
    // 92.8 -> 90.0; 290 x 200000 34.7 -> 34.1; 4096 x 32768, k 2048 118.1 and 118.3.  More batches to L2 at the start cost more than they gave:
    // 2 | 4 | 6 instead of one, 496 x 262144 60.2 | 61.9 | 64.7 us, 4096 x 32768, k 512 102 | 109 | 112 instead of 99.
    constexpr int kMine = kSampleQuads / THREADS;
    float4 sample[kMine];
#pragma unroll
    for (int u = 0; u < kMine; ++u) {
        const int32_t quad = sampled_quad(tid + u * THREADS);
        sample[u] = quad >= span ? none : row.stride == 1 ? load_quad(row.x + row.position(base + quad)) : row.load(base + quad);
    }
    float4 v[kStreamBatch];
#pragma unroll
    for (int u = 0; u < kStreamBatch; ++u) v[u] = u * THREADS < left ? load_quad(next + 4 * u * THREADS) : none;
    // The up to three values in front of the first whole quad and behind the last one, one per lane of the first CTA's first warp.
    float edge_value = -INFINITY;
    int32_t edge_position = -1;
    if (row.stride == 1 && rank == 0 && tid < 6) {
        edge_position = tid < 3 ? (tid < row.position(begin) ? tid : -1) : (end >= begin ? row.position(end) + tid - 3 : -1);
        if (begin == 0 && tid < 3) edge_position = -1;
        edge_value = row.edge(edge_position);
    }
    // With many rows, the batch after that one to L2, by one instruction of one thread; from then on always the batch after the next.
    constexpr int kBatch = kStreamBatch * THREADS;
    const auto send_to_l2 = [&](int32_t quads_ahead) {  // (thread 0's `left` is what remains of the share)
        const int32_t room = left - quads_ahead;
        if (tid == 0 && p.ahead && room > 0) prefetch_l2(next + 4 * quads_ahead, 16u * static_cast<uint32_t>(room < kBatch ? room : kBatch));
    };
    send_to_l2(kBatch);
    clear_histogram<THREADS>(s);
    if (tid < 4) s.counters[tid] = 0u;
    if (tid == 4) s.pooled = 0u;
    __syncthreads();
    uint32_t largest = 0u;
    float peak = -INFINITY;
#pragma unroll
    for (int u = 0; u < kMine; ++u) {
        if (sampled_quad(tid + u * THREADS) >= span) continue;
        const float value[4] = {sample[u].x, sample[u].y, sample[u].z, sample[u].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            atomicAdd(&s.hist[coarse_bin(value[e])], 1u);
            peak = fmaxf(peak, value[e]);
        }
    }
    largest = order_key(__float_as_uint(peak));
    largest = __reduce_max_sync(0xffffffffu, largest);
    if ((tid & 31) == 0) atomicMax(&s.counters[3], largest);
    __syncthreads();
    const Floor f = floor_from_sample<THREADS>(s, k, 4 * (span < kSampleQuads ? span : kSampleQuads), len);
    if (!(f.value > -INFINITY)) {
        __syncthreads();
        if (rank == 0) select_from_histogram<THREADS>(s, dynamic, p.capacity, row, k, out);
        return;
    }
    if (ctas > 1) cluster.sync();  // the first CTA's counters are zero before anybody reserves room in its pool
    else __syncthreads();
    const Pool pool{dynamic, &s.pooled, p.capacity};
    // full batches, then what is left of the share, then the quads that are not whole
    const auto load_next = [&](float4(&to)[kStreamBatch]) {
        if (left + tid >= kBatch) {
#pragma unroll
            for (int u = 0; u < kStreamBatch; ++u) to[u] = load_quad(next + 4 * u * THREADS);
        } else {
#pragma unroll
            for (int u = 0; u < kStreamBatch; ++u) to[u] = u * THREADS < left ? load_quad(next + 4 * u * THREADS) : none;
        }
    };
    // looks through the batch in `now` while the next one is on its way to `then`, and says whether there is one
    const auto step = [&](float4(&now)[kStreamBatch], float4(&then)[kStreamBatch]) {
        send_to_l2(2 * kBatch);
        left -= kBatch, next += 4 * kBatch;
        if (TWO) load_next(then);
        pool.take(now, position, 4 * THREADS, f.value);
        if (!TWO) load_next(then);
        position += 4 * kBatch;
        return left + tid > 0;
    };
    if (left + tid > 0) {
        if constexpr (TWO) {
            float4 w[kStreamBatch];
            while (step(v, w) && step(w, v)) {}
        } else {
            while (step(v, v)) {}
        }
    }
    float4 edge[1];
    if (row.stride != 1) {
        for (int32_t e = static_cast<int32_t>(rank) * THREADS + tid; e - (tid & 31) < row.quads; e += static_cast<int32_t>(ctas) * THREADS) {
            edge[0] = e < row.quads ? row.load(e) : none;
            pool.take(edge, row.position(e), 0, f.value);
        }
    } else if (rank == 0 && tid < 32) {
        edge[0] = make_float4(edge_value, -INFINITY, -INFINITY, -INFINITY);
        pool.take(edge, edge_position, 0, f.value);
    }
    __syncthreads();
    if (ctas > 1) {
        if (rank != 0) {
            // hand the candidates over to the first CTA through distributed shared memory
            const uint32_t mine = s.pooled;
            if (tid == 0) s.result[3] = atomicAdd(cluster.map_shared_rank(&s.pooled, 0), mine);
            __syncthreads();
            const uint32_t at = s.result[3];
            if (mine <= p.capacity && at + mine <= p.capacity) {
                uint2* remote = cluster.map_shared_rank(dynamic, 0);
                for (uint32_t i = tid; i < mine; i += THREADS) remote[at + i] = dynamic[i];
            }
        }
        cluster.sync();  // all candidates have arrived
        if (rank != 0) return;
    }
    if (!select<THREADS>(s, dynamic, s.pooled, p.capacity, static_cast<uint32_t>(k), f, out))
        select_from_histogram<THREADS>(s, dynamic, p.capacity, row, k, out);
}

// Candidates to expect when the sample holds `size` of `len` values (see floor_from_sample): their number, and its spread.
struct Expected {
    double count, deviation;
    Expected(double k, double size, double len) {
        const double mean = k * size / len, rank = mean + 4.0 * std::sqrt(mean) + 3.0;
        count = rank * len / size, deviation = count / std::sqrt(rank);
    }
};

// Room for them with six standard deviations on top.
uint32_t pool_capacity(const Expected& e) { return static_cast<uint32_t>(std::min(e.count + 6.0 * e.deviation + 64.0, 8192.0)); }

constexpr size_t kMaxDynamicBytes = sizeof(uint2) * 8192;

template <typename Kernel>
cudaError_t launch(Kernel kernel, const TopkParams& p, int threads, unsigned ctas, cudaStream_t stream) {
    if (p.num_rows * static_cast<int64_t>(ctas) > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    const cudaError_t err = launch_dependent_cluster(kernel, static_cast<unsigned>(p.num_rows) * ctas, static_cast<unsigned>(threads), ctas,
                                                     sizeof(uint2) * p.capacity, stream, p);
    if (err != cudaSuccess) return err;
    count_launch();
    return cudaGetLastError();
}

// Per-device set-up, once per device however many host threads make their first call at the same time.
struct DeviceSetup {
    std::once_flag once;
    cudaError_t status = cudaSuccess;
    int sms = 0;
};

template <bool DECODE>
cudaError_t set_up(DeviceSetup** result) {
    static DeviceSetup setups[64];
    int dev = 0;
    const cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    DeviceSetup& setup = setups[dev];
    std::call_once(setup.once, [&]() {
        const auto allow = [&](auto* kernel) {
            if (setup.status == cudaSuccess)
                setup.status = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kMaxDynamicBytes));
        };
        allow(topk_stream_kernel<DECODE, 512, true>), allow(topk_stream_kernel<DECODE, 512, true, true>), allow(topk_stream_kernel<DECODE, 512, false>), allow(topk_stream_kernel<DECODE, 256, false>);
        allow(topk_registers_kernel<DECODE, 512, 4>), allow(topk_registers_kernel<DECODE, 512, 8>), allow(topk_registers_kernel<DECODE, 256, 8>);
        if (setup.status == cudaSuccess) setup.status = cudaDeviceGetAttribute(&setup.sms, cudaDevAttrMultiProcessorCount, dev);
    });
    *result = &setup;
    return setup.status;
}

template <bool DECODE>
cudaError_t launch_topk(TopkParams& p, cudaStream_t stream) {
    DeviceSetup* setup = nullptr;
    const cudaError_t err = set_up<DECODE>(&setup);
    if (err != cudaSuccess) return err;
    const int sms = setup->sms;
    const bool aligned = p.stride1 == 1 && (reinterpret_cast<uintptr_t>(p.logits) & 15u) == 0 && p.stride0 % 4 == 0 && !p.row_starts;
    const int64_t quads = (static_cast<int64_t>(p.vocab) + (aligned ? 0 : 3) + 3) / 4;
    const auto registers = [&](auto* kernel, int threads) {
        p.capacity = pool_capacity(Expected(p.top_k, 1.0, 4.0));
        return launch(kernel, p, threads, 1, stream);
    };
    const auto whole = [&](auto* kernel, int threads) {
        p.capacity = kCountingMax;  // of the histogram route
        return launch(kernel, p, threads, 1, stream);
    };
    const auto stream_rows = [&](auto* kernel, int threads, unsigned ctas) {
        p.capacity = pool_capacity(Expected(p.top_k, std::min(p.vocab, 4 * sample_quads(threads)), p.vocab));
        // Pays once the GPU is full.  Without | with it, us, k 512 and rows of full length unless said otherwise: 4096 x 32768 106 | 98,
        // causal with k 2048 130 | 117; 1531 x 32768 49.4 | 45.3; 1000 x 40000 40.7 | 38.6; 890 x 32768, k 2048 40.1 | 37.5; 496 x 262144
        // 92.0 | 90.8, ragged 60.6 | 59.4; 444 x 100000 ragged 29.5 | 27.7.  Below the line small CTAs gain too (880 x 32768, k 2048
        // 40.0 | 37.5; 600 x 32768 21.3 | 20.7; 296 x 65536 25.3 | 22.7), clusters hardly (61 x 65536 10.1 | 10.3; 140 x 65536 13.4 |
        // 13.0; 290 x 40000 14.2 | 14.1).  Three wide CTAs per SM, which are past it only when all are there, gain up to 100000 values
        // (320 x 100000 30.6 | 30.0) and lose beyond (400 x 140000 42.8 | 43.7; 440 x 262144 74.3 | 78.2; 444 x 262144 75.0 | 79.2).
        p.ahead = p.num_rows * static_cast<int64_t>(ctas) * threads >= 1536LL * sms;
        return launch(kernel, p, threads, ctas, stream);
    };
    // Few rows: the time of one row counts, so it gets many threads, or a cluster.  Many rows: small CTAs, of which more are
    // resident and cover each other's barriers.  Where the lines lie was measured: 61 x 4096, k 512: 5.1 us with 512 threads, 6.0 with
    // 256, 8.4 with 128; 4096 x 2048: 57 / 29 / 23 us (both before the codes of two values shared a register: 3.8 and 19 us now).  Rows
    // of up to 4096 values need no sample (1531 x 4096, k 512: 17 us, 23 us with one), longer ones do (4096 x 8192: 49 us, 67 us without).
    const int64_t rows = p.num_rows;
    if (rows < 2 * sms) {
        if (quads <= 512 * 2) return whole(topk_short_kernel<DECODE, 512, 2>, 512);
        if (quads <= 512 * 4) return registers(topk_registers_kernel<DECODE, 512, 4>, 512);
        if (quads <= 512 * 8) return registers(topk_registers_kernel<DECODE, 512, 8>, 512);
        // Up to two CTAs per SM, and 8192 values for each.  One | two | four CTAs a row, us: 61 x 17000 7.3 | 7.6 | 7.9; 61 x 40000 9.1 |
        // 8.7 | 9.0; 100 x 20000 7.6 | 8.9 | 12.6; 140 x 20000 8.0 | 9.2 | 15.8; 140 x 40000 10.9 | 11.6 | 18.9; 148 x 65536 13.7 | 13.6 |
        // 21.6; 120 x 262144 34.3 | 28.0 | 33.8.  (61 x 65536: 10.6 us with four, 15 with one or eight, before two batches were in flight;
        // 10 us now with four.)  So from about 100 rows on a pair wants 32768 values or more for each, which the rule does not ask for.
        unsigned ctas = 1;
        while (ctas < 8 && rows * ctas * 2 <= 2 * sms && static_cast<int64_t>(p.vocab) >= 8192LL * ctas * 2) ctas *= 2;
        return stream_rows(topk_stream_kernel<DECODE, 512, true>, 512, ctas);
    }
    if (quads <= 128 * 4) return whole(topk_short_kernel<DECODE, 128, 4>, 128);
    if (quads <= 256 * 4) return whole(topk_short_kernel<DECODE, 256, 4>, 256);
    if (quads <= 256 * 8) return registers(topk_registers_kernel<DECODE, 256, 8>, 256);
    if (p.vocab <= 65536) return stream_rows(topk_stream_kernel<DECODE, 256, false>, 256, 1);
    // Longer rows: three CTAs per SM while that makes one wave, then two with two batches in flight each.  Three | two per SM, us,
    // k 512 unless said otherwise, rows of ragged and of full length:
    //   320 x 200000  43 | 43, 50 | 64        310 x 140000, k 2048  35 | 37        444 x 262144, full 79 | 86
    //   496 x 262144  73 | 67, 108 | 88       496 x 100000  35 | 33, 47 | 44       800 x 262144  98 | 97, 134 | 134
    //   320 x 262144  54 | 52, 62 | 80        400 x 262144  57 | 61, 70 | 86       444 x 262144  60 | 63, 79 | 86
    //   320 x 262144, k 2048  57 | 54         400 x 262144, k 2048  60 | 64        400 x 131072  33 | 37
    //   445 x 100000  27.6 | 31.6
    // (A pair of CTAs per row: 496 x 262144 70, 100; 320 x 200000 45, 56; 320 x 262144 53, 69; 400 x 262144 60, 77; 800 x 262144 99, 138.)
    // Up to 444 rows the longest first with two per SM (see below) would take 44, 51 and 56 us for 320, 400 and 444 ragged rows of 262144,
    // but 83, 89 and 89 us for rows of full length, and the host does not know which they are.
    if (rows <= 3LL * sms) return stream_rows(topk_stream_kernel<DECODE, 512, false>, 512, 1);
    // Up to two waves of them, the longest rows first: what runs at the end, on a GPU that is no longer full, is then short.  Finding
    // the order costs a CTA about 1 us, which pays for very long rows of different length only.  By index | longest first, us:
    //   460 x 131072  39 | 36, full length 50 | 52    460 x 200000  54 | 47, 70 | 73    592 x 200000  60 | 56, 81 | 85
    //   496 x 262144  67 | 60, full length 90 | 94    592 x 262144, k 1024  76 | 70, 102 | 105
    //   740 x 131072  54 | 56    740 x 262144  91 | 91, full length 133 | 137    496 x 100000  33 | 33, full length 44 | 46
    if (rows <= 4LL * sms && rows <= kOrderedRows && p.vocab >= 131072) {
        while ((p.vocab >> p.length_shift) >= 64) ++p.length_shift;
        return stream_rows(topk_stream_kernel<DECODE, 512, true, true>, 512, 1);
    }
    return stream_rows(topk_stream_kernel<DECODE, 512, true>, 512, 1);
}

}  // namespace

cudaError_t launch_topk_per_row(const float* logits, int64_t stride0, int64_t stride1, int32_t* indices, int64_t num_rows, int vocab,
                                int top_k, const int32_t* seq_lens, int next_n, const int32_t* row_starts, const int32_t* row_ends,
                                cudaStream_t stream) {
    if (num_rows == 0 || top_k == 0) return cudaSuccess;
    TopkParams p{};
    p.logits = logits, p.stride0 = stride0, p.stride1 = stride1, p.indices = indices;
    p.num_rows = static_cast<int32_t>(num_rows), p.vocab = vocab, p.top_k = top_k;
    p.seq_lens = seq_lens, p.next_n = next_n, p.row_starts = row_starts, p.row_ends = row_ends;
    p.sampled = 2 * static_cast<int64_t>(top_k) + 512 <= 8192;
    return seq_lens ? launch_topk<true>(p, stream) : launch_topk<false>(p, stream);
}

}  // namespace dsv4
