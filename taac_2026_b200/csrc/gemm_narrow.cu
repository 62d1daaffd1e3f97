// Grouped bf16 GEMM for 9 .. 128 rows per group on tcgen05 with the operands' roles exchanged:
//     out[g]^T = act(w[g] a[g]^T + bias[g]) (+ residual[g]^T),   a: [groups, M, K], w: [groups, N, K]
// so that the 128-row side of the tensor-core tile is 128 output columns (always full) and its free side is M, padded to
// 16.  The layers are bound by streaming their weights: 9 groups of 1536 x 512 give 108 CTAs here instead of 54 tiles of
// 128 x 256, and where N is short (512 x 2048: 36 CTAs) a cluster of up to four CTAs splits K, so that most SMs have their
// share of the weights in flight at once.
//
// One tile per CTA, 192 threads: warp 0 fills a ring of {W 128 x 64, A M x 64} tiles by TMA (128-byte swizzle), warp 1 issues
// the MMAs, warps 2 .. 5 read the accumulator (lane = output column, TMEM column = row of M), add bias, activation and
// residual and store bf16: for one row of M the 32 lanes of a warp write 64 consecutive bytes.  With a split, every CTA leaves its
// fp32 partial tile in its own shared memory and the CTAs of the cluster each sum a share of the rows over the ranks in
// order through distributed shared memory.  Every wait is bounded; one that gives up raises the status word and the roles
// drain through the barriers.

#include "tb200_common.cuh"
#include "tb200_ptx.cuh"
#include "tb200_tmap.cuh"

namespace tb200 {
void count_launch();

namespace {

constexpr int kThreads = 192;
constexpr int kTile = 128;                      // output columns per CTA
constexpr uint32_t kWBytes = kTile * 128;       // a W tile: 128 rows x 64 bf16
constexpr uint32_t kRingBytes = 96 * 1024;      // W and A tiles; two CTAs fit an SM, so that the next kernel's are already set up
constexpr int kMaxStages = 10;
constexpr int kPartStride = kTile + 4;          // floats between rows of a partial tile

struct NarrowArgs {
    const float* bias;
    const __nv_bfloat16* residual;
    __nv_bfloat16* out;
    int32_t* status;
    int32_t M, N, K, act;
    int32_t m_pad;      // M rounded up to 16: columns of the MMA
    int32_t stages;
    uint32_t tmem_cols;
};

__device__ __forceinline__ float ld_peer(uint32_t smem_addr, uint32_t rank) {
    uint32_t at;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem_addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at));
    return v;
}

// Sixteen outputs of one column, rows `step` apart: all residual loads before the first store (`out` may be the residual)
__device__ __forceinline__ void load_residual(const NarrowArgs& g, int64_t at, int rows, int step, float (&res)[16]) {
#pragma unroll
    for (int i = 0; i < 16; ++i)
        res[i] = g.residual != nullptr && i < rows ? __bfloat162float(g.residual[at + static_cast<int64_t>(i * step) * g.N]) : 0.f;
}
__device__ __forceinline__ void store_rows(const NarrowArgs& g, int64_t at, int rows, int step, float bias, const float (&v)[16],
                                           const float (&res)[16]) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        float x = v[i] + bias;
        if (g.act == 1) {   // silu(x) = h tanh(h) + h, h = x / 2 (the result is rounded to bf16)
            const float h = 0.5f * x;
            float th;
            asm("tanh.approx.f32 %0, %1;" : "=f"(th) : "f"(h));
            x = fmaf(h, th, h);
        }
        if (i < rows) g.out[at + static_cast<int64_t>(i * step) * g.N] = __float2bfloat16_rn(x + res[i]);
    }
}

template <int SPLIT>
__global__ void __launch_bounds__(kThreads, 2)
gemm_narrow_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_w, const NarrowArgs g) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t full_bar[kMaxStages], empty_bar[kMaxStages], acc_full;
    __shared__ uint32_t tmem_base_slot;
    uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = SPLIT > 1 ? static_cast<int>(cluster_rank()) : 0;
    const int n0 = (blockIdx.x / SPLIT) * kTile;
    const int grp = blockIdx.y;
    const int k_blocks = g.K / 64;
    const int kb0 = k_blocks * rank / SPLIT, kb1 = k_blocks * (rank + 1) / SPLIT;
    const uint32_t a_bytes = static_cast<uint32_t>(g.m_pad) * 128;
    const uint32_t stage_bytes = kWBytes + a_bytes;

    if (threadIdx.x == 0) {
        for (int s = 0; s < g.stages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        mbar_init(&acc_full, 1);
        fence_mbar_init();
    }
    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tmap_a);
        tma_prefetch_desc(&tmap_w);
        for (int kb = kb0; kb < kb1; ++kb) tma_prefetch_3d(&tmap_w, kb * 128, n0, grp);   // into the L2, behind the preceding kernel
    }
    if (warp == 1) {
        tmem_alloc(&tmem_base_slot, g.tmem_cols);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = tmem_base_slot;
    chain_release();   // not before every CTA holds its tensor memory (see launch_chained)
    chain_wait();

    bool ok = true;
    if (warp == 0) {
        if (lane == 0) {
            for (int kb = kb0, it = 0; kb < kb1; ++kb, ++it) {
                const int s = it % g.stages;
                if (!mbar_wait_sleep(&empty_bar[s], ((it / g.stages) & 1) ^ 1)) { ok = false; break; }
                uint8_t* dst = ring + static_cast<size_t>(s) * stage_bytes;
                mbar_expect_tx(&full_bar[s], stage_bytes);
                tma_load_3d(dst, &tmap_w, kb * 128, n0, grp, &full_bar[s]);
                tma_load_3d(dst + kWBytes, &tmap_a, kb * 128, 0, grp, &full_bar[s]);
            }
        }
    } else if (warp == 1) {
        {   // all lanes walk the loop, an elected one issues (see mbar_wait_warp)
            const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem, 0);
            const uint32_t idesc = umma_idesc(1, 1, 0, 0, kTile, static_cast<uint32_t>(g.m_pad));
            const uint64_t desc0 = umma_desc_sw128(0, 1024, 16);
            const uint32_t ring_lo = (smem_u32(ring) & 0x3FFFFu) >> 4;
            for (int kb = kb0, it = 0; kb < kb1; ++kb, ++it) {
                const int s = it % g.stages;
                if (!mbar_wait_warp(&full_bar[s], (it / g.stages) & 1)) { ok = false; break; }
                tc_fence_after_sync();
                const uint64_t dw = desc0 + ring_lo + s * (stage_bytes >> 4);
                const uint64_t da = dw + (kWBytes >> 4);
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) mma_f16_ss(tmem_u, dw + 2 * k, da + 2 * k, idesc, (it | k) != 0 ? 1u : 0u);
                    tc_commit(&empty_bar[s]);
                }
                __syncwarp();
            }
            if (elect_one()) tc_commit(&acc_full);    // after a wait that gave up the partial products still end here, and the epilogue writes garbage
        }
    } else {
        ok = mbar_wait_sleep(&acc_full, 0);
        tc_fence_after_sync();
        const int quarter = warp & 3;
        const int col = quarter * 32 + lane;                     // output column inside the tile = TMEM lane
        const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
        const float bias = g.bias != nullptr ? g.bias[static_cast<int64_t>(grp) * g.N + n0 + col] : 0.f;
        float* part = reinterpret_cast<float*>(ring);            // every load has been consumed by now
        for (int m0 = 0; m0 < g.m_pad; m0 += 16) {
            const int64_t at = (static_cast<int64_t>(grp) * g.M + m0) * g.N + n0 + col;
            const int rows = min(g.M - m0, 16);
            float v[16], res[16];
            if (SPLIT == 1) load_residual(g, at, rows, 1, res);
            uint32_t r[16];
            tmem_ld_x16(tmem + lane_addr + m0, r);
            tc_wait_ld(r);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                v[i] = __uint_as_float(r[i]);
                if (SPLIT > 1) part[(m0 + i) * kPartStride + col] = v[i];
            }
            if (SPLIT == 1) store_rows(g, at, rows, 1, bias, v, res);
        }
    }
    if (SPLIT > 1) {
        __syncwarp();
        cluster_sync_all();                                      // every rank's partial tile is in place
        if (warp >= 2) {
            const int col = (warp & 3) * 32 + lane;
            const float bias = g.bias != nullptr ? g.bias[static_cast<int64_t>(grp) * g.N + n0 + col] : 0.f;
            const uint32_t part = smem_u32(ring);
            for (int m0 = rank; m0 < g.M; m0 += 16 * SPLIT) {      // sixteen of this rank's rows at a time: m0, m0 + SPLIT, ...
                const int64_t at = (static_cast<int64_t>(grp) * g.M + m0) * g.N + n0 + col;
                const int rows = min((g.M - m0 + SPLIT - 1) / SPLIT, 16);
                float v[16], res[16];
                load_residual(g, at, rows, SPLIT, res);
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    v[i] = 0.f;
                    if (i < rows) {
#pragma unroll
                        for (int r = 0; r < SPLIT; ++r) v[i] += ld_peer(part + ((m0 + i * SPLIT) * kPartStride + col) * 4, r);
                    }
                }
                store_rows(g, at, rows, SPLIT, bias, v, res);
            }
        }
        __syncwarp();
        cluster_sync_all();                                      // nobody leaves while its tile is being read
    }
    if (!ok && g.status != nullptr) atomicExch(g.status, 1);
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem, g.tmem_cols);
    }
}

// [groups, rows, row_bytes] bytes, boxes of box_rows x 128 bytes inside one group
bool make_map(CUtensorMap* map, const void* base, uint64_t row_bytes, uint64_t rows, uint64_t groups, uint32_t box_rows) {
    const auto fn = encode_fn();
    if (fn == nullptr) return false;
    const cuuint64_t dims[3] = {row_bytes, rows, groups};
    const cuuint64_t strides[2] = {row_bytes, row_bytes * rows};
    const cuuint32_t box[3] = {128, box_rows, 1};
    const cuuint32_t elem[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int SPLIT>
int launch(const CUtensorMap& ta, const CUtensorMap& tw, const NarrowArgs& g, int groups, size_t smem, cudaStream_t stream) {
    static bool attr_set[64] = {};
    const DeviceInfo& dev = device_info();
    if (!attr_set[dev.index]) {
        cudaFuncSetAttribute(gemm_narrow_kernel<SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kRingBytes + 1024));
        attr_set[dev.index] = true;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(g.N / kTile * SPLIT, groups);
    cfg.blockDim = kThreads;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2]{};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = SPLIT;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = SPLIT > 1 ? 2 : 1;
    cudaLaunchKernelEx(&cfg, gemm_narrow_kernel<SPLIT>, ta, tw, g);
    count_launch();
    return launch_status();
}

}  // namespace

// 1 <= M <= 128 (beyond that the 256-row tiles are faster), N % 128 == 0, K % 64 == 0, act 0 or 1
int gemm_narrow(const void* a, const void* w, const float* bias, const void* residual, void* out, int groups, int M, int N, int K, int act,
                int32_t* status, cudaStream_t stream) {
    NarrowArgs g{};
    g.bias = bias;
    g.residual = static_cast<const __nv_bfloat16*>(residual);
    g.out = static_cast<__nv_bfloat16*>(out);
    g.status = status;
    g.M = M;
    g.N = N;
    g.K = K;
    g.act = act;
    g.m_pad = (M + 15) / 16 * 16;
    g.tmem_cols = 32;
    while (g.tmem_cols < static_cast<uint32_t>(g.m_pad)) g.tmem_cols <<= 1;
    CUtensorMap ta, tw;
    if (!make_map(&ta, a, 2ull * K, M, groups, g.m_pad) || !make_map(&tw, w, 2ull * K, N, groups, kTile)) return TB200_ERR_DRIVER;
    // split K over a cluster while the CTAs still fit the chip once and every CTA keeps at least four 64-wide blocks
    const int ctas = N / kTile * groups, k_blocks = K / 64;
    int split = 1;
    while (split < 4 && ctas * split * 2 <= device_info().sm_count && k_blocks / (2 * split) >= 4) split *= 2;
    const uint32_t stage_bytes = kWBytes + static_cast<uint32_t>(g.m_pad) * 128;
    int stages = static_cast<int>(kRingBytes / stage_bytes);
    if (stages > kMaxStages) stages = kMaxStages;
    const int per_cta = (k_blocks + split - 1) / split;
    if (stages > per_cta) stages = per_cta;
    g.stages = stages;
    size_t smem = static_cast<size_t>(stages) * stage_bytes;
    const size_t part = split > 1 ? static_cast<size_t>(g.m_pad) * kPartStride * sizeof(float) : 0;
    if (smem < part) smem = part;
    smem += 1024;
    switch (split) {
        case 1: return launch<1>(ta, tw, g, groups, smem, stream);
        case 2: return launch<2>(ta, tw, g, groups, smem, stream);
        default: return launch<4>(ta, tw, g, groups, smem, stream);
    }
}

}  // namespace tb200
