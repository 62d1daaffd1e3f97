// Grouped fp32 GEMM on the tensor cores, for the engine's score-parity mode (fp32 weights, activations and results):
//     out[g] = act(a[g] w[g]^T + bias[g]) (+ residual[g])        a: [groups, M, K], out / residual: [groups, M, N], all fp32
//
// An fp32 value is the sum of three bf16 values, x = h + m + l (8 + 8 + 8 significant bits: h = bf16(x), m = bf16(x - h),
// l = bf16(x - h - m), the differences exact), and a product of two such sums is
//     xh yh + xh ym + xm yh + xm ym + xh yl + xl yh + terms below 2^-24 of it,
// which is the rounding of an fp32 multiplication.  The six kept products of bf16 values are exact in the tensor core and
// accumulate in fp32, the smallest first.  Six bf16 products at the tcgen05 rate are several times the rate of the fp32
// units: 74 000 x 256 x 128 ran at 47 TFLOP/s as a library SGEMM on the CUDA cores.
//
// Persistent CTAs of 448 threads on 128 x 128 tiles (column tiles fastest, so that the CTAs at work share activation rows):
//   warp 0        TMA producer of the weights, which are split once at load: [N, 3 K] bf16 = [h | m | l] per row
//   warp 1        MMA issuer: per 64-wide K block 6 x 4 tcgen05.mma of 128 x 128 x 16 into one of two accumulators
//   warps 2 .. 5  epilogue: a thread owns a row; bias, SiLU (exponential form), residual, 16-byte stores
//   warps 6 .. 13 read the fp32 activations (a block ahead, in registers), split them and write the three bf16 tiles with
//                 the 128-byte swizzle the MMA expects
// Two stages of {A: 3 x 16 KB, W: 3 x 16 KB}.  Every wait is bounded and reports through the status word.
#include <cudaTypedefs.h>

#include "tb200_common.cuh"
#include "tb200_ptx.cuh"

namespace tb200 {
void count_launch();

namespace {

constexpr int kTile = 128;
constexpr int kBK = 64;
constexpr int kStages = 2;
constexpr int kSplitThreads = 256;
constexpr int kThreads = 64 + 128 + kSplitThreads;
constexpr uint32_t kPartBytes = kTile * kBK * 2;           // one bf16 tile of 128 x 64
constexpr uint32_t kStageBytes = 6 * kPartBytes;           // A: h, m, l; W: h, m, l
constexpr size_t kSmemBytes = kStages * kStageBytes + 1024;
constexpr uint32_t kTmemCols = 2 * kTile;

struct F32Args {
    const float* a;
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

// four fp32 -> their three bf16 parts
__device__ __forceinline__ void split4(const float4& x, uint2 (&part)[3]) {
    float4 r = x;
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        part[p] = make_uint2(pack_bf16(r.x, r.y), pack_bf16(r.z, r.w));
        r.x -= low_of(part[p].x);
        r.y -= high_of(part[p].x);
        r.z -= low_of(part[p].y);
        r.w -= high_of(part[p].y);
    }
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

__global__ void __launch_bounds__(kThreads, 1)
gemm_f32_kernel(const __grid_constant__ CUtensorMap tmap_w, const F32Args g) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t full_bar[kStages], empty_bar[kStages], tmem_full[2], tmem_empty[2];
    __shared__ uint32_t tmem_base_slot;
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
            mbar_init(&tmem_empty[b], 128);
        }
        fence_mbar_init();
    }
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
            uint32_t it = 0, tile = 0;
            for (int64_t t = blockIdx.x; t < total && ok; t += gridDim.x, ++tile) {
                const uint32_t buf = tile & 1;
                if (!mbar_wait_warp(&tmem_empty[buf], ((tile >> 1) & 1) ^ 1)) { ok = false; break; }
                tc_fence_after_sync();
                for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                    const uint32_t s = it % kStages;
                    if (!mbar_wait_warp(&full_bar[s], (it / kStages) & 1)) { ok = false; break; }
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
                                           (kb | c | k) != 0 ? 1u : 0u);
                        tc_commit(&empty_bar[s]);
                    }
                    __syncwarp();
                }
                if (ok && elect_one()) tc_commit(&tmem_full[buf]);
                __syncwarp();
            }
        }
    } else if (warp < 6) {
        const int quarter = warp & 3;
        const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
        uint32_t tile = 0;
        for (int64_t t = blockIdx.x; t < total && ok; t += gridDim.x, ++tile) {
            int n0, grp;
            int64_t m0;
            decode(t, n0, m0, grp);
            const uint32_t buf = tile & 1;
            if (!mbar_wait_sleep(&tmem_full[buf], (tile >> 1) & 1)) ok = false;
            if (__any_sync(0xffffffffu, !ok)) { ok = false; break; }
            tc_fence_after_sync();
            const int64_t row = m0 + quarter * 32 + lane;
            const bool live = row < g.M;
            const int64_t at = (static_cast<int64_t>(grp) * g.M + (live ? row : 0)) * g.N + n0;
#pragma unroll 1
            for (int c0 = 0; c0 < kTile; c0 += 32) {
                uint32_t acc[32];
                tmem_ld_2x16(tmem_base + buf * kTile + lane_addr + c0, acc);
                float4 res[8];
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    res[q] = g.residual != nullptr && live ? *reinterpret_cast<const float4*>(g.residual + at + c0 + 4 * q) : make_float4(0.f, 0.f, 0.f, 0.f);
                tc_wait_ld(acc);
                if (c0 + 32 == kTile) {
                    tc_fence_before_sync();
                    mbar_arrive(&tmem_empty[buf]);
                }
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (g.bias != nullptr) b = __ldg(reinterpret_cast<const float4*>(g.bias + static_cast<int64_t>(grp) * g.N + n0 + c0 + 4 * q));
                    float v[4] = {__uint_as_float(acc[4 * q]) + b.x, __uint_as_float(acc[4 * q + 1]) + b.y, __uint_as_float(acc[4 * q + 2]) + b.z,
                                  __uint_as_float(acc[4 * q + 3]) + b.w};
                    if (g.act == 1) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) v[e] = v[e] / (1.0f + expf(-v[e]));
                    }
                    if (live)
                        *reinterpret_cast<float4*>(g.out + at + c0 + 4 * q) =
                            make_float4(v[0] + res[q].x, v[1] + res[q].y, v[2] + res[q].z, v[3] + res[q].w);
                }
            }
        }
    } else {
        const int tid = threadIdx.x - 192;
        const int col4 = tid & 15, row_in = tid >> 4;          // 16 threads per row of 64 values, rows row_in + 16 i
        uint32_t it = 0;
        float4 next[8];
        auto fetch = [&](int64_t t, int kb) {
            int n0, grp;
            int64_t m0;
            decode(t, n0, m0, grp);
            const float* base = g.a + static_cast<int64_t>(grp) * g.M * g.K + kb * kBK + col4 * 4;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int64_t row = m0 + row_in + 16 * i;
                next[i] = row < g.M ? *reinterpret_cast<const float4*>(base + row * g.K) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        };
        if (blockIdx.x < total) fetch(blockIdx.x, 0);
        for (int64_t t = blockIdx.x; t < total && ok; t += gridDim.x) {
            for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                const uint32_t s = it % kStages;
                float4 cur[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) cur[i] = next[i];
                if (kb + 1 < k_blocks) fetch(t, kb + 1);
                else if (t + gridDim.x < total) fetch(t + gridDim.x, 0);
                if (!mbar_wait_sleep(&empty_bar[s], ((it / kStages) & 1) ^ 1)) { ok = false; break; }
                uint8_t* stage = smem + s * kStageBytes;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int row = row_in + 16 * i;
                    uint2 part[3];
                    split4(cur[i], part);
                    uint8_t* dst = stage + row * 128 + (((col4 >> 1) ^ (row & 7)) << 4) + (col4 & 1) * 8;
#pragma unroll
                    for (int p = 0; p < 3; ++p) *reinterpret_cast<uint2*>(dst + p * kPartBytes) = part[p];
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

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = []() -> PFN_cuTensorMapEncodeTiled_v12000 {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult res;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &res) == cudaSuccess && res == cudaDriverEntryPointSuccess)
            return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
        cudaGetLastError();
        return nullptr;
    }();
    return fn;
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
    const F32Args g{a, bias, residual, out, status_word, M, groups, N, K, act};
    const int64_t tiles = (M + kTile - 1) / kTile * (N / kTile) * groups;
    const int64_t grid = tiles < dev.sm_count ? tiles : dev.sm_count;
    launch_chained(gemm_f32_kernel, static_cast<unsigned>(grid), kThreads, kSmemBytes, static_cast<cudaStream_t>(stream), tw, g);
    count_launch();
    return launch_status();
}
