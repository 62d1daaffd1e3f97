// Grouped bf16 GEMM for a handful of rows per group: the same layers as gemm_bf16.cu at request-sized batches,
//     out[g] = act(a[g] w[g]^T + bias[g]) (+ residual[g]),   a: [groups, M, K] with M <= 32, w: [groups, N, K].
//
// Bound by streaming the weights (9 groups of 1536 x 512: 14 MB, 2.2 us of HBM time); a 128 x 256 tile per CTA puts 54 of 148
// SMs to work and took 9 us (18 us for 512 x 2048, now 4.7 and 4.8).  Here a CTA owns 16 output columns of one group and its eight warps split K, so that every
// SM has many 16-byte weight loads in flight, and the partial sums meet in shared memory in a fixed order.  The weight
// rows are the 16-row operand of mma.sync m16n8k16 and the activations the 8-column one.  The order
// of k inside a product is free: lane t of a quad takes eight consecutive k of a row (one 16-byte load) for the two k
// halves of two products, on both sides alike, so operands go from global memory to registers without a transposition.
// The weights of the CTA are requested into the L2 before the wait on the preceding kernel.
#include "tb200_common.cuh"

namespace tb200 {
void count_launch();

namespace {

constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;
constexpr int kCols = 16;     // output columns of a CTA (times two for gated layers: gate and value)

struct SmallArgs {
    const __nv_bfloat16* a;
    const __nv_bfloat16* w;
    const float* bias;
    const __nv_bfloat16* residual;
    __nv_bfloat16* out;
    int32_t M, N, K, act;
    int64_t w_stride, bias_stride;       // elements between the groups' weights / biases (0: one for all groups)
    const __nv_bfloat16* norm_gamma;     // not NULL: the activations are rmsnorm(a + norm_bias) norm_gamma
    const __nv_bfloat16* norm_bias;      // may be NULL
    float norm_eps;
};

__device__ __forceinline__ uint4 ld_weights(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// pieces of eight values of a row, plus the bias in fp32
__device__ __forceinline__ void load_norm_input(const SmallArgs& g, const __nv_bfloat16* row, int piece, float (&f)[8]) {
    Vec16<__nv_bfloat16>::unpack(reinterpret_cast<const uint4*>(row)[piece], f);
    if (g.norm_bias != nullptr) {
        float b[8];
        Vec16<__nv_bfloat16>::unpack(reinterpret_cast<const uint4*>(g.norm_bias)[piece], b);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] += b[e];
    }
}

// MT: eight-row tiles of M; NT: 16-column tiles of W per CTA (2: a gate tile and its value tile 128 rows further)
template <int MT, int NT, bool NORM>
__global__ void __launch_bounds__(kThreads)
gemm_small_kernel(const SmallArgs g) {
    __shared__ float part[kWarps][NT][kCols][MT * 8 + 1];
    __shared__ float s_inv[NORM ? MT * 8 : 1];
    chain_release();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int gr = lane >> 2, t = lane & 3;
    const int64_t grp = blockIdx.y;
    // gated: 128 gate and 128 value rows alternate; CTA x owns gate rows [n0, n0 + 16) and the values 128 rows behind them
    const int n0 = NT == 1 ? blockIdx.x * kCols : (blockIdx.x / 8) * 256 + (blockIdx.x % 8) * kCols;
    const __nv_bfloat16* wg = g.w + grp * g.w_stride + static_cast<int64_t>(n0) * g.K;
    const int chunks = g.K / 32;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
        for (int i = threadIdx.x; i < kCols * (g.K / 64); i += kThreads) {   // 128 bytes per request
            const int r = i / (g.K / 64), c = i - r * (g.K / 64);
            asm volatile("prefetch.global.L2 [%0];" ::"l"(wg + static_cast<int64_t>(nt * 128 + r) * g.K + c * 64));
        }
    chain_wait();

    float acc[NT][MT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[nt][mt][e] = 0.f;
    const __nv_bfloat16* ag = g.a + grp * g.M * g.K;
    if (NORM) {   // every CTA takes the statistics of the group's few rows itself: a row per warp, out of the L2
        for (int m = warp; m < g.M; m += kWarps) {
            float sq = 0.f;
            for (int c = lane; c < g.K / 8; c += 32) {
                float f[8];
                load_norm_input(g, ag + static_cast<int64_t>(m) * g.K, c, f);
#pragma unroll
                for (int e = 0; e < 8; ++e) sq = fmaf(f[e], f[e], sq);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
            if (lane == 0) s_inv[m] = rsqrtf(sq / static_cast<float>(g.K) + g.norm_eps);
        }
        __syncthreads();
    }
    constexpr int U = MT == 1 ? 4 : 2;   // chunks of 32 k in flight per warp
    for (int c0 = warp; c0 < chunks; c0 += kWarps * U) {
        uint4 wv[U][NT][2], xv[U][MT];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int c = c0 + u * kWarps;
            if (c < chunks) {
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        wv[u][nt][h] = ld_weights(reinterpret_cast<const uint4*>(wg + static_cast<int64_t>(nt * 128 + gr + 8 * h) * g.K + c * 32 + t * 8));
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) {
                    const int m = mt * 8 + gr;
                    if (NORM) {
                        xv[u][mt] = make_uint4(0u, 0u, 0u, 0u);
                        if (m < g.M) {
                            float f[8], gm[8];
                            load_norm_input(g, ag + static_cast<int64_t>(m) * g.K, c * 4 + t, f);
                            Vec16<__nv_bfloat16>::unpack(reinterpret_cast<const uint4*>(g.norm_gamma)[c * 4 + t], gm);
                            const float inv = s_inv[m];
#pragma unroll
                            for (int e = 0; e < 8; ++e) f[e] = (f[e] * inv) * gm[e];
                            xv[u][mt] = Vec16<__nv_bfloat16>::pack(f);
                        }
                    } else {
                        xv[u][mt] = m < g.M ? *reinterpret_cast<const uint4*>(ag + static_cast<int64_t>(m) * g.K + c * 32 + t * 8) : make_uint4(0u, 0u, 0u, 0u);
                    }
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (c0 + u * kWarps >= chunks) break;
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) {
                    mma(acc[nt][mt], wv[u][nt][0].x, wv[u][nt][1].x, wv[u][nt][0].y, wv[u][nt][1].y, xv[u][mt].x, xv[u][mt].y);
                    mma(acc[nt][mt], wv[u][nt][0].z, wv[u][nt][1].z, wv[u][nt][0].w, wv[u][nt][1].w, xv[u][mt].z, xv[u][mt].w);
                }
        }
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int e = 0; e < 4; ++e) part[warp][nt][gr + 8 * (e >> 1)][mt * 8 + 2 * t + (e & 1)] = acc[nt][mt][e];
    __syncthreads();
    const int n_out = NT == 1 ? g.N : g.N / 2;
    const int o0 = NT == 1 ? n0 : (n0 / 256) * 128 + n0 % 256;
    auto total = [&](int nt, int c, int m) {   // the sum over K of one output, in the order of the warps
        float v = g.bias != nullptr ? g.bias[grp * g.bias_stride + n0 + nt * 128 + c] : 0.f;
#pragma unroll
        for (int k = 0; k < kWarps; ++k) v += part[k][nt][c][m];
        return v;
    };
    for (int i = threadIdx.x; i < kCols / 2 * g.M; i += kThreads) {   // two columns per thread
        const int m = i / (kCols / 2), c = 2 * (i - m * (kCols / 2));
        float v[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            v[e] = total(0, c + e, m);
            if (g.act >= 1) {   // silu(v) = h tanh(h) + h, h = v / 2 (the result is rounded to bf16)
                const float h = 0.5f * v[e];
                float th;
                asm("tanh.approx.f32 %0, %1;" : "=f"(th) : "f"(h));
                v[e] = fmaf(h, th, h);
            }
            if (NT == 2) v[e] *= total(NT - 1, c + e, m);
        }
        const int64_t at = (grp * g.M + m) * n_out + o0 + c;
        if (g.residual != nullptr) {
            const float2 r = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(g.residual + at));
            v[0] += r.x;
            v[1] += r.y;
        }
        *reinterpret_cast<__nv_bfloat162*>(g.out + at) = __floats2bfloat162_rn(v[0], v[1]);
    }
}

template <int MT, int NT, bool NORM>
int launch(const SmallArgs& g, int groups, cudaStream_t stream) {
    launch_chained(gemm_small_kernel<MT, NT, NORM>, dim3(g.N / (NT * kCols), groups), kThreads, 0, stream, g);
    count_launch();
    return launch_status();
}
template <int NT, bool NORM>
int launch_rows(const SmallArgs& g, int groups, cudaStream_t stream) {
    if (g.M <= 8) return launch<1, NT, NORM>(g, groups, stream);
    if (g.M <= 16) return launch<2, NT, NORM>(g, groups, stream);
    return launch<4, NT, NORM>(g, groups, stream);
}

}  // namespace

// Does this kernel serve the call?  It re-reads the activations in every CTA of 16 columns, so the more rows, the fewer of its
// CTAs may there be (measurements at the dispatch in gemm_bf16.cu).
bool gemm_small_serves(int groups, int64_t M, int N, int K) {
    const int64_t ctas = static_cast<int64_t>(groups) * (N / kCols);
    const int64_t sms = device_info().sm_count;
    return groups <= 65535 && (M <= 8 || (M <= 16 && ctas <= 6 * sms) || (M <= 32 && K <= 2048 && ctas <= 2 * sms));
}

int gemm_small(const void* a, const void* w, const float* bias, const void* residual, void* out, int groups, int M, int N, int K, int act,
               bool shared_w, const void* norm_gamma, const void* norm_bias, float norm_eps, cudaStream_t stream) {
    const SmallArgs g{static_cast<const __nv_bfloat16*>(a), static_cast<const __nv_bfloat16*>(w), bias, static_cast<const __nv_bfloat16*>(residual),
                      static_cast<__nv_bfloat16*>(out), M, N, K, act, shared_w ? 0 : static_cast<int64_t>(N) * K, shared_w ? 0 : N,
                      static_cast<const __nv_bfloat16*>(norm_gamma), static_cast<const __nv_bfloat16*>(norm_bias), norm_eps};
    if (act == 2) return launch_rows<2, false>(g, groups, stream);
    return norm_gamma != nullptr ? launch_rows<1, true>(g, groups, stream) : launch_rows<1, false>(g, groups, stream);
}

}  // namespace tb200

extern "C" int tb200_gemm_bf16_few_rows(const void* a, const void* w, const float* bias, const void* residual, void* out, int32_t groups, int64_t M,
                                        int32_t N, int32_t K, int32_t act, int32_t shared_w, const void* norm_gamma, const void* norm_bias,
                                        float norm_eps, void* stream) {
    using namespace tb200;
    if (groups < 0 || M < 0 || N < 256 || N % 256 != 0 || K < 64 || K % 64 != 0) return TB200_ERR_SHAPE;
    if (act < 0 || act > 1) return TB200_ERR_UNSUPPORTED;
    if (groups == 0 || M == 0) return TB200_OK;
    if (a == nullptr || w == nullptr || out == nullptr) return TB200_ERR_NULL;
    for (const void* p : {a, w, static_cast<const void*>(out), residual, norm_gamma, norm_bias})
        if (!aligned16(p)) return TB200_ERR_ALIGN;
    if (bias != nullptr && (reinterpret_cast<uintptr_t>(bias) & 3) != 0) return TB200_ERR_ALIGN;
    if (!device_info().valid) return TB200_ERR_DEVICE;
    if (!gemm_small_serves(groups, M, N, K)) return TB200_ERR_UNSUPPORTED;
    return gemm_small(a, w, bias, residual, out, groups, static_cast<int>(M), N, K, act, shared_w != 0, norm_gamma, norm_bias, norm_eps,
                      static_cast<cudaStream_t>(stream));
}
