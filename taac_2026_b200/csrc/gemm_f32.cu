// Grouped fp32 GEMM on the tensor cores, for the engine's score-parity mode (fp32 weights, activations and results):
//     out[g] = act(a[g] w[g]^T + bias[g]) (+ residual[g])        a: [groups, M, K], out / residual: [groups, M, N], all fp32
//
// An fp32 value is the sum of three bf16 values, x = h + m + l (8 + 8 + 8 significant bits: h = bf16(x), m = bf16(x - h),
// l = bf16(x - h - m), the differences exact), and a product of two such sums is
//     xh yh + xh ym + xm yh + xm ym + xh yl + xl yh + terms below 2^-24 of it,
// which is the rounding of an fp32 multiplication.  The six kept products of bf16 values are exact in the tensor core, but its
// additions cut off what lies below the accumulator's last place instead of rounding.  So the tensor core only sums one K block of
// 64, the smallest products first, and the blocks are added up in fp32 registers with rounding: over the whole of K in the tensor
// core the error of a sum was 1.5e-6 at K = 256 and 1.7e-5 at K = 2560 (2-norm against float64; a library SGEMM: 2.9e-7 and
// 9.1e-7), with the blocks added in registers 8.8e-8 and 1.4e-7.  Six bf16 products at the tcgen05 rate are several times the rate of the fp32
// units: 74 000 x 256 x 128 ran at 47 TFLOP/s as a library SGEMM on the CUDA cores.
//
// Persistent CTAs of 512 threads on 128 x 128 tiles (column tiles fastest, so that the CTAs at work share activation rows):
//   warp 0          TMA producer of the weights, which are split once at load: [N, 3 K] bf16 = [h | m | l] per row
//   warp 1          MMA issuer: per 64-wide K block 6 x 4 tcgen05.mma of 128 x 128 x 16 into one of two accumulators
//   warps 2 .. 9    sums and epilogue: a thread owns half a row, adds the blocks' products to its 64 sums while the tensor cores
//                   fill the other accumulator (24 products take longer than the read), then bias, SiLU (exponential form),
//                   residual, 16-byte stores
//   warps 10 .. 15  read the fp32 activations (a block ahead, in registers), split them and write the three bf16 tiles with
//                   the 128-byte swizzle the MMA expects
// A row with an infinity, a NaN or a value that rounds to an infinite bf16 has no such split (inf - inf): its outputs are
// computed again in plain fp32.
// Two stages of {A: 3 x 16 KB, W: 3 x 16 KB}.  Every wait is bounded and reports through the status word.

#include "tb200_common.cuh"
#include "tb200_ptx.cuh"
#include "tb200_tmap.cuh"

namespace tb200 {
void count_launch();

namespace {

constexpr int kTile = 128;
constexpr int kBK = 64;
constexpr int kStages = 2;
constexpr int kSumThreads = 256;
constexpr int kSplitThreads = 192;
constexpr int kSplitRows = kSplitThreads / 16;                        // rows of 64 values that they take at a time
constexpr int kSplitSteps = (kTile + kSplitRows - 1) / kSplitRows;
constexpr int kThreads = 64 + kSumThreads + kSplitThreads;
constexpr int kFlagTiles = 8;      // tiles between the splitting warps and the sums: at most five (two stages, two accumulators)
constexpr uint32_t kPartBytes = kTile * kBK * 2;           // one bf16 tile of 128 x 64
constexpr uint32_t kStageBytes = 6 * kPartBytes;           // A: h, m, l; W: h, m, l
constexpr size_t kSmemBytes = kStages * kStageBytes + 1024;
constexpr uint32_t kTmemCols = 2 * kTile;

struct F32Args {
    const float* a;
    const __nv_bfloat16* w_split;
    const float* bias;
    const float* residual;
    float* out;
    int32_t* status;
    int64_t M;
    int32_t groups, N, K, act;
};

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float low_of(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float high_of(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

// four fp32 -> their three bf16 parts; false: one of them has none
__device__ __forceinline__ bool split4(const float4& x, uint2 (&part)[3]) {
    float4 r = x;
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        part[p] = make_uint2(pack_bf16(r.x, r.y), pack_bf16(r.z, r.w));
        r.x -= low_of(part[p].x);
        r.y -= high_of(part[p].x);
        r.z -= low_of(part[p].y);
        r.w -= high_of(part[p].y);
    }
    const float rest = (r.x + r.y) + (r.z + r.w);   // NaN where a part was not finite
    return rest == rest;
}

__global__ void __launch_bounds__(256)
split_weights_kernel(const float4* __restrict__ w, __nv_bfloat16* __restrict__ out, int64_t rows, int k) {
    chain_release();
    chain_wait();
    const int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;
    const int per_row = k / 4;
    if (i >= rows * per_row) return;
    const int64_t row = i / per_row;
    const int c = static_cast<int>(i - row * per_row) * 4;
    uint2 part[3];
    split4(w[i], part);
#pragma unroll
    for (int p = 0; p < 3; ++p) *reinterpret_cast<uint2*>(out + row * 3 * k + static_cast<int64_t>(p) * k + c) = part[p];
}

// 64 outputs of a row from column n0 on without the split
__device__ __noinline__ void plain_row(const F32Args& g, int grp, int64_t row, int n0) {
    const float* a = g.a + (static_cast<int64_t>(grp) * g.M + row) * g.K;
    for (int n = n0; n < n0 + kTile / 2; ++n) {
        const __nv_bfloat16* w = g.w_split + (static_cast<int64_t>(grp) * g.N + n) * 3 * g.K;
        float v = 0.f;
        for (int k = 0; k < g.K; ++k) v = fmaf(a[k], (__bfloat162float(w[k]) + __bfloat162float(w[g.K + k])) + __bfloat162float(w[2 * g.K + k]), v);
        if (g.bias != nullptr) v += g.bias[static_cast<int64_t>(grp) * g.N + n];
        if (g.act == 1) v = v / (1.0f + expf(-v));
        const int64_t at = (static_cast<int64_t>(grp) * g.M + row) * g.N + n;
        g.out[at] = v + (g.residual != nullptr ? g.residual[at] : 0.f);
    }
}

__global__ void __launch_bounds__(kThreads, 1)
gemm_f32_kernel(const __grid_constant__ CUtensorMap tmap_w, const F32Args g) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t full_bar[kStages], empty_bar[kStages], tmem_full[2], tmem_empty[2];
    __shared__ uint32_t tmem_base_slot;
    __shared__ uint8_t no_split[kFlagTiles][2][kTile];   // rows of a tile in flight whose outputs (left, right half) are computed in plain fp32
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t m_tiles = (g.M + kTile - 1) / kTile;
    const int n_tiles = g.N / kTile, k_blocks = g.K / kBK;
    const int64_t total = m_tiles * n_tiles * g.groups;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&full_bar[s], 1 + kSplitThreads);
            mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&tmem_full[b], 1);
            mbar_init(&tmem_empty[b], kSumThreads);
        }
        fence_mbar_init();
    }
    for (int i = threadIdx.x; i < kFlagTiles * 2 * kTile; i += kThreads) (&no_split[0][0][0])[i] = 0;
    if (warp == 1) {
        tmem_alloc(&tmem_base_slot, kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = tmem_base_slot;
    chain_release();   // not before every CTA holds its tensor memory (see launch_chained)
    chain_wait();

    auto decode = [&](int64_t t, int& n0, int64_t& m0, int& grp) {
        n0 = static_cast<int>(t % n_tiles) * kTile;
        const int64_t rest = t / n_tiles;
        m0 = rest % m_tiles * kTile;
        grp = static_cast<int>(rest / m_tiles);
    };
    bool ok = true;
    if (warp == 0) {
        if (lane == 0) {
            tma_prefetch_desc(&tmap_w);
            uint32_t it = 0;
            for (int64_t t = blockIdx.x; t < total && ok; t += gridDim.x) {
                int n0, grp;
                int64_t m0;
                decode(t, n0, m0, grp);
                for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                    const uint32_t s = it % kStages;
                    if (!mbar_wait_sleep(&empty_bar[s], ((it / kStages) & 1) ^ 1)) { ok = false; break; }
                    mbar_expect_tx(&full_bar[s], 3 * kPartBytes);
#pragma unroll
                    for (int p = 0; p < 3; ++p)
                        tma_load_3d(smem + s * kStageBytes + (3 + p) * kPartBytes, &tmap_w, (p * g.K + kb * kBK) * 2, n0, grp, &full_bar[s]);
                }
            }
        }
    } else if (warp == 1) {
        {   // all lanes walk the loop, an elected one issues (see mbar_wait_warp)
            const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
            const uint32_t idesc = umma_idesc(1, 1, 0, 0, kTile, kTile);
            const uint64_t desc0 = umma_desc_sw128(0, 1024, 16);
            const uint32_t base_lo = (smem_u32(smem) & 0x3FFFFu) >> 4;
            constexpr uint32_t kPart = kPartBytes >> 4;
            uint32_t it = 0;
            for (int64_t t = blockIdx.x; t < total && ok; t += gridDim.x) {
                for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                    const uint32_t s = it % kStages, buf = it & 1;
                    if (!mbar_wait_warp(&tmem_empty[buf], ((it >> 1) & 1) ^ 1) || !mbar_wait_warp(&full_bar[s], (it / kStages) & 1)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    const uint64_t at = desc0 + base_lo + s * (kStageBytes >> 4);
                    // (part of A, part of W), smallest products first
                    constexpr int pa[6] = {2, 1, 0, 1, 0, 0}, pw[6] = {0, 1, 2, 0, 1, 0};
                    if (elect_one()) {
#pragma unroll
                        for (int c = 0; c < 6; ++c)
#pragma unroll
                            for (int k = 0; k < kBK / 16; ++k)
                                mma_f16_ss(tmem + buf * kTile, at + pa[c] * kPart + 2 * k, at + (3 + pw[c]) * kPart + 2 * k, idesc,
                                           (c | k) != 0 ? 1u : 0u);
                        tc_commit(&empty_bar[s]);
                        tc_commit(&tmem_full[buf]);
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp < 2 + kSumThreads / 32) {
        const int quarter = warp & 3;                       // TMEM lanes [32 quarter, +32) are visible to this warp
        const int col0 = ((warp - 2) >> 2) * (kTile / 2);   // this thread's 64 columns
        const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
        uint32_t it = 0, tile = 0;
        for (int64_t t = blockIdx.x; t < total && ok; t += gridDim.x, ++tile) {
            int n0, grp;
            int64_t m0;
            decode(t, n0, m0, grp);
            float sum[kTile / 2];
#pragma unroll
            for (int i = 0; i < kTile / 2; ++i) sum[i] = 0.f;
#pragma unroll 1
            for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                const uint32_t buf = it & 1;
                if (!mbar_wait_sleep(&tmem_full[buf], (it >> 1) & 1)) ok = false;
                if (__any_sync(0xffffffffu, !ok)) { ok = false; break; }
                tc_fence_after_sync();
#pragma unroll
                for (int c = 0; c < kTile / 2; c += 16) {
                    uint32_t acc[16];
                    tmem_ld_x16(tmem_base + buf * kTile + lane_addr + col0 + c, acc);
                    tc_wait_ld(acc);
#pragma unroll
                    for (int i = 0; i < 16; ++i) sum[c + i] += __uint_as_float(acc[i]);
                }
                tc_fence_before_sync();
                mbar_arrive(&tmem_empty[buf]);
            }
            if (!ok) break;
            const int row_in_tile = quarter * 32 + lane;
            const int64_t row = m0 + row_in_tile;
            const bool live = row < g.M;
            const int64_t at = (static_cast<int64_t>(grp) * g.M + (live ? row : 0)) * g.N + n0 + col0;
            uint8_t& plain = no_split[tile % kFlagTiles][col0 != 0 ? 1 : 0][row_in_tile];
            const bool no_sum = plain != 0;
            if (no_sum) {
                plain = 0;      // for the tile eight later
                plain_row(g, grp, row, n0 + col0);
            }
            if (live && !no_sum) {
#pragma unroll
                for (int c0 = 0; c0 < kTile / 2; c0 += 16) {
                    float4 res[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        res[q] = g.residual != nullptr ? *reinterpret_cast<const float4*>(g.residual + at + c0 + 4 * q) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (g.bias != nullptr) b = __ldg(reinterpret_cast<const float4*>(g.bias + static_cast<int64_t>(grp) * g.N + n0 + col0 + c0 + 4 * q));
                        float v[4] = {sum[c0 + 4 * q] + b.x, sum[c0 + 4 * q + 1] + b.y, sum[c0 + 4 * q + 2] + b.z, sum[c0 + 4 * q + 3] + b.w};
                        if (g.act == 1) {
#pragma unroll
                            for (int e = 0; e < 4; ++e) v[e] = v[e] / (1.0f + expf(-v[e]));
                        }
                        *reinterpret_cast<float4*>(g.out + at + c0 + 4 * q) = make_float4(v[0] + res[q].x, v[1] + res[q].y, v[2] + res[q].z, v[3] + res[q].w);
                    }
                }
            }
            __syncwarp();
        }
    } else {
        const int tid = threadIdx.x - 64 - kSumThreads;
        const int col4 = tid & 15, row_in = tid >> 4;          // 16 threads per row of 64 values, rows row_in + 12 i
        uint32_t it = 0, tile = 0;
        float4 next[kSplitSteps];
        // the block that is read next: this thread's first value of it and the rows that exist (0 behind the last tile)
        const float* first = g.a;
        int rows = 0;
        auto locate = [&](int64_t t) {
            int n0, grp;
            int64_t m0;
            decode(t, n0, m0, grp);
            first = g.a + (static_cast<int64_t>(grp) * g.M + m0 + row_in) * g.K + col4 * 4;
            rows = static_cast<int>(g.M - m0 < kTile ? g.M - m0 : kTile);
        };
        const int64_t step = static_cast<int64_t>(kSplitRows) * g.K;
        if (blockIdx.x < total) locate(blockIdx.x);
        {
            const float* p = first;
#pragma unroll
            for (int i = 0; i < kSplitSteps; ++i, p += step) next[i] = row_in + kSplitRows * i < rows ? *reinterpret_cast<const float4*>(p) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        for (int64_t t = blockIdx.x; t < total && ok; t += gridDim.x, ++tile) {
            for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                const uint32_t s = it % kStages;
                if (kb + 1 < k_blocks) first += kBK;
                else if (t + gridDim.x < total) locate(t + gridDim.x);
                else rows = 0;
                if (!mbar_wait_sleep(&empty_bar[s], ((it / kStages) & 1) ^ 1)) { ok = false; break; }
                uint8_t* stage = smem + s * kStageBytes;
                const float* p = first;
#pragma unroll
                for (int i = 0; i < kSplitSteps; ++i, p += step) {
                    const int row = row_in + kSplitRows * i;
                    if (row >= kTile) break;
                    uint2 part[3];
                    if (!split4(next[i], part)) no_split[tile % kFlagTiles][0][row] = no_split[tile % kFlagTiles][1][row] = 1;
                    // requested as soon as its register has been split
                    next[i] = row < rows ? *reinterpret_cast<const float4*>(p) : make_float4(0.f, 0.f, 0.f, 0.f);
                    uint8_t* dst = stage + row * 128 + (((col4 >> 1) ^ (row & 7)) << 4) + (col4 & 1) * 8;
#pragma unroll
                    for (int q = 0; q < 3; ++q) *reinterpret_cast<uint2*>(dst + q * kPartBytes) = part[q];
                }
                fence_proxy_async_smem();
                mbar_arrive(&full_bar[s]);
            }
        }
    }
    if (!ok && g.status != nullptr) atomicExch(g.status, 1);
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

}  // namespace
}  // namespace tb200

extern "C" int tb200_split_f32_weights(const float* w, void* w_split, int64_t rows, int32_t K, void* stream) {
    using namespace tb200;
    if (rows < 0 || K < 4 || K % 4 != 0) return TB200_ERR_SHAPE;
    if (rows == 0) return TB200_OK;
    if (w == nullptr || w_split == nullptr) return TB200_ERR_NULL;
    if (!aligned16(w) || !aligned16(w_split)) return TB200_ERR_ALIGN;
    const int64_t blocks = (rows * (K / 4) + 255) / 256;
    if (blocks > 0x7FFFFFFFll) return TB200_ERR_SHAPE;
    if (!device_info().valid) return TB200_ERR_DEVICE;
    launch_chained(split_weights_kernel, static_cast<unsigned>(blocks), 256, 0, static_cast<cudaStream_t>(stream), reinterpret_cast<const float4*>(w),
                   static_cast<__nv_bfloat16*>(w_split), rows, K);
    count_launch();
    return launch_status();
}

extern "C" int tb200_gemm_f32_grouped(const float* a, const void* w_split, const float* bias, const float* residual, float* out, int32_t groups,
                                      int64_t M, int32_t N, int32_t K, int32_t act, int32_t* status_word, void* stream) {
    using namespace tb200;
    if (groups < 0 || M < 0 || N < kTile || N % kTile != 0 || K < kBK || K % kBK != 0) return TB200_ERR_SHAPE;
    if (act < 0 || act > 1) return TB200_ERR_UNSUPPORTED;
    if (groups == 0 || M == 0) return TB200_OK;
    if (a == nullptr || w_split == nullptr || out == nullptr) return TB200_ERR_NULL;
    for (const void* p : {static_cast<const void*>(a), w_split, static_cast<const void*>(out), static_cast<const void*>(bias),
                          static_cast<const void*>(residual)})
        if (!aligned16(p)) return TB200_ERR_ALIGN;
    if (M > 0x7FFFFF00ll || 6ll * K > 0x7FFFFFFFll) return TB200_ERR_SHAPE;
    const DeviceInfo& dev = device_info();
    if (!dev.valid) return TB200_ERR_DEVICE;
    const auto fn = encode_fn();
    if (fn == nullptr) return TB200_ERR_DRIVER;
    CUtensorMap tw;
    const cuuint64_t dims[3] = {6ull * K, static_cast<cuuint64_t>(N), static_cast<cuuint64_t>(groups)};
    const cuuint64_t strides[2] = {6ull * K, 6ull * K * N};
    const cuuint32_t box[3] = {128, kTile, 1};
    const cuuint32_t elem[3] = {1, 1, 1};
    if (fn(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(w_split), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return TB200_ERR_DRIVER;
    static bool attr_set[64] = {};
    if (!attr_set[dev.index]) {
        cudaFuncSetAttribute(gemm_f32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmemBytes));
        attr_set[dev.index] = true;
    }
    const F32Args g{a, static_cast<const __nv_bfloat16*>(w_split), bias, residual, out, status_word, M, groups, N, K, act};
    const int64_t tiles = (M + kTile - 1) / kTile * (N / kTile) * groups;
    const int64_t grid = tiles < dev.sm_count ? tiles : dev.sm_count;
    launch_chained(gemm_f32_kernel, static_cast<unsigned>(grid), kThreads, kSmemBytes, static_cast<cudaStream_t>(stream), tw, g);
    count_launch();
    return launch_status();
}
