// Recognises the structured bool attention masks the models build, in one pass over the mask.
//
// One CTA per sample.  The mask rows of a sample are described by a valid prefix of `lead` keys, a valid suffix of `trail`
// keys and one of two forms:
//   form 1   every query row shows exactly those keys (a key mask)
//   form 2   a valid query shows the valid keys up to itself, a padded one ([lead, Lk - trail)) itself alone
//            (`causal_valid_attention_mask`)
// A description is guessed from two rows and the first column (under form 2 the last row that sees key 0 shows every valid
// key, or, without a prefix, the last row does) and then compared with every element, so a wrong guess only means
// form 0, "not recognised".  The samples are combined by the caller, who needs the suffix length on the host: the verdict
// goes to pinned host memory, so the caller pays one stream synchronisation and no copy.
//
// Bound by reading the mask once (B Lq Lk bytes).  Eight lanes share a row and compare 16 bytes at a time with the words
// the description predicts, so that a CTA has 128 rows in flight (64 masks of 256 x 256: 37 us with one row per warp, 14 us like this).
#include "tb200_common.cuh"

namespace tb200 {
void count_launch();

namespace {

constexpr int kThreads = 1024;
constexpr int kRowLanes = 8;   // lanes per row in the comparison

// bytes [lo, hi) of the word at position p, as ones
__device__ __forceinline__ uint32_t range_word(int p, int lo, int hi) {
    const int a = min(max(lo - p, 0), 4), b = min(max(hi - p, 0), 4);
    const uint32_t upto = b >= 4 ? 0xffffffffu : ((1u << (8 * b)) - 1u);
    const uint32_t from = a >= 4 ? 0xffffffffu : ((1u << (8 * a)) - 1u);
    return 0x01010101u & upto & ~from;
}

// Walks a row of `n` bytes in aligned 16-byte pieces (bytes outside the row read as zero): f(position, word)
template <int LANES, typename F>
__device__ __forceinline__ void walk_row(const uint8_t* row, int n, int lane, F f) {
    const uintptr_t start = reinterpret_cast<uintptr_t>(row);
    const int skew = static_cast<int>(start & 15u);
    const uint4* base = reinterpret_cast<const uint4*>(start - skew);
    const int pieces = (skew + n + 15) / 16;
    #pragma unroll 4
    for (int i = lane; i < pieces; i += LANES) {
        const uint4 v = __ldg(base + i);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int p = i * 16 + e * 4 - skew;
            const uint32_t inside = range_word(p, 0, n);
            if (inside != 0u) f(p, w[e] & (inside * 0xffu), inside);
        }
    }
}

struct RowShape {
    int lead, trail, count;
};

__device__ __forceinline__ RowShape row_shape(const uint8_t* row, int n, int lane) {
    int first_zero = n, last_zero = -1, count = 0;
    walk_row<32>(row, n, lane, [&](int p, uint32_t w, uint32_t inside) {
        const uint32_t ones = w & 0x01010101u;
        count += __popc(ones);
        const uint32_t zeros = inside & ~ones;
        if (zeros != 0u) {
            first_zero = min(first_zero, p + ((__ffs(zeros) - 1) >> 3));
            last_zero = max(last_zero, p + ((31 - __clz(zeros)) >> 3));
        }
    });
    for (int o = 16; o > 0; o >>= 1) {
        first_zero = min(first_zero, __shfl_xor_sync(0xffffffffu, first_zero, o));
        last_zero = max(last_zero, __shfl_xor_sync(0xffffffffu, last_zero, o));
        count += __shfl_xor_sync(0xffffffffu, count, o);
    }
    return RowShape{first_zero, n - 1 - last_zero, count};
}

__global__ void __launch_bounds__(kThreads)
mask_plan_kernel(const uint8_t* __restrict__ mask, int64_t sb, int64_t sh, int64_t sq, int heads, int lq, int lk,
                 int32_t* __restrict__ lens, int4* __restrict__ verdict) {
    chain_release();
    chain_wait();
    __shared__ RowShape s_row[3];   // row 0, the last row, the last row that sees key 0
    __shared__ int s_last0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint8_t* m = mask + blockIdx.x * sb;
    if (threadIdx.x == 0) s_last0 = 0;
    __syncthreads();
    if (warp < 2) {
        const RowShape r = row_shape(m + (warp == 0 ? 0 : lq - 1) * sq, lk, lane);
        if (lane == 0) s_row[warp] = r;
    }
    int last0 = 0;
    for (int q = threadIdx.x; q < lq; q += kThreads)
        if (m[q * sq] != 0) last0 = q;
    last0 = __reduce_max_sync(0xffffffffu, last0);
    if (lane == 0 && last0 > 0) atomicMax(&s_last0, last0);
    __syncthreads();
    last0 = s_last0;
    RowShape r = s_row[0];
    const RowShape r_end = s_row[1];
    int form = 1;
    bool identity = false;
    if (r.lead != r_end.lead || r.trail != r_end.trail || r.count != r_end.count) {   // rows differ: form 2 or nothing
        form = 2;
        if (last0 > 0) {
            if (warp == 0) {
                const RowShape x = row_shape(m + last0 * sq, lk, lane);
                if (lane == 0) s_row[2] = x;
            }
            __syncthreads();
            r = s_row[2];
        } else if (r_end.count >= 2) {
            r = r_end;
        } else {
            identity = true;
        }
        if (lq != lk) form = 0;
    }
    const int lead = identity ? 0 : r.lead;
    const int trail = identity || lead == lk ? 0 : r.trail;
    if (!identity && r.count != lead + trail) form = 0;
    if (form != 0) {
        const int ns = lk - trail;
        const int lg = threadIdx.x % kRowLanes;
        uint32_t diff = 0;
        for (int h = 0; h < heads; ++h)
            for (int q = threadIdx.x / kRowLanes; q < (form == 1 && sq == 0 ? 1 : lq); q += kThreads / kRowLanes) {
                int hi0 = lead, lo1 = ns, hi1 = lk;   // expected keys [0, hi0) and [lo1, hi1)
                if (form == 2) {
                    hi0 = min(lead, q + 1);
                    hi1 = q + 1;
                    if (q >= lead && q < ns) {        // padded: itself alone
                        hi0 = 0;
                        lo1 = q;
                    }
                }
                walk_row<kRowLanes>(m + h * sh + q * sq, lk, lg, [&](int p, uint32_t w, uint32_t) {
                    diff |= w ^ (range_word(p, 0, hi0) | range_word(p, lo1, hi1));
                });
            }
        if (__syncthreads_or(diff != 0u)) form = 0;
    }
    if (threadIdx.x == 0) {
        lens[blockIdx.x] = lead;
        verdict[blockIdx.x] = make_int4(form, lead, trail, identity ? 2 : (lead < lk ? 1 : 0));
    }
}

}  // namespace
}  // namespace tb200

extern "C" int tb200_mask_plan(const uint8_t* mask, int64_t stride_b, int64_t stride_h, int64_t stride_q, int32_t B, int32_t H,
                               int32_t Lq, int32_t Lk, int32_t* lens, int32_t* verdict, void* stream) {
    using namespace tb200;
    if (B < 1 || H < 1 || Lq < 1 || Lk < 1) return TB200_ERR_SHAPE;
    if (mask == nullptr || lens == nullptr || verdict == nullptr) return TB200_ERR_NULL;
    if (!aligned16(verdict)) return TB200_ERR_ALIGN;
    if (!device_info().valid) return TB200_ERR_DEVICE;
    launch_chained(mask_plan_kernel, B, kThreads, 0, static_cast<cudaStream_t>(stream), mask, stride_b, stride_h, stride_q, stride_h == 0 ? 1 : H, Lq,
                                                                            Lk, lens, reinterpret_cast<int4*>(verdict));
    count_launch();
    return launch_status();
}
