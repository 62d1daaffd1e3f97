// Row kernels around the engine's blocks: the small projected tokens, the placement of the non-sequence rows, the pooled
// means and the classifier's last layer.  Each of them replaces a handful of one-line tensor operations whose launches
// cost more than their work; all are bound by launch latency at request sizes and by their row traffic at large ones.
#include "tb200_common.cuh"

namespace tb200 {
void count_launch();

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ---------------------------------------------------------------------------------------
// small_token: out[r, :] = LayerNorm(SiLU(W x_r + b)) with x_r = [values[r, :n], mask[r, :n] as 0 / 1 (optional)], all in fp32.
// Eight rows per CTA: a thread owns output columns and reads its weights (transposed: neighbouring threads, neighbouring
// addresses) once for the eight of them; the activated rows meet in shared memory, where one warp per row takes the
// statistics.
// ---------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(kThreads)
small_token_kernel(const float* __restrict__ values, int n, int64_t value_stride, const uint8_t* __restrict__ mask, int64_t mask_stride,
                   int in_dim, const float* __restrict__ w, const float* __restrict__ bias, const float* __restrict__ gamma,
                   const float* __restrict__ beta, T* __restrict__ out, int64_t out_stride, int64_t rows, int d, float eps) {
    chain_release();
    chain_wait();
    extern __shared__ float smem[];
    float* xs = smem;                       // [kWarps][in_dim]
    float* hs = smem + kWarps * in_dim;     // [kWarps][d]
    const int64_t row0 = static_cast<int64_t>(blockIdx.x) * kWarps;
    for (int i = threadIdx.x; i < kWarps * in_dim; i += kThreads) {
        const int r = i / in_dim, c = i - r * in_dim;
        float v = 0.f;
        if (row0 + r < rows) {
            if (c < n) v = values[(row0 + r) * value_stride + c];
            else if (mask != nullptr) v = mask[(row0 + r) * mask_stride + c - n] != 0 ? 1.f : 0.f;
        }
        xs[i] = v;
    }
    __syncthreads();
    for (int o = threadIdx.x; o < d; o += kThreads) {
        float acc[kWarps];
#pragma unroll
        for (int r = 0; r < kWarps; ++r) acc[r] = bias[o];
#pragma unroll 8
        for (int c = 0; c < in_dim; ++c) {
            const float wv = w[static_cast<int64_t>(c) * d + o];
#pragma unroll
            for (int r = 0; r < kWarps; ++r) acc[r] = fmaf(wv, xs[r * in_dim + c], acc[r]);
        }
#pragma unroll
        for (int r = 0; r < kWarps; ++r) hs[r * d + o] = acc[r] / (1.0f + expf(-acc[r]));
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (row0 + warp >= rows) return;
    const float* h = hs + warp * d;
    float sum = 0.f;
    for (int c = lane; c < d; c += 32) sum += h[c];
    const float mean = warp_sum(sum) / static_cast<float>(d);
    float sq = 0.f;
    for (int c = lane; c < d; c += 32) sq = fmaf(h[c] - mean, h[c] - mean, sq);
    const float inv = rsqrtf(warp_sum(sq) / static_cast<float>(d) + eps);
    T* y = out + (row0 + warp) * out_stride;
    for (int c = lane; c < d; c += 32) y[c] = from_float<T>(fmaf((h[c] - mean) * inv, gamma[c], beta[c]));
}

// ---------------------------------------------------------------------------------------
// ns_rows: the non-sequence tokens [B, ns, d] take their rows of the residual stream, and their RMS-normalised form takes
// its rows of the normalised matrix and the token-major copy [ns, B, d] that the per-token projections read.  The row ids
// are token-major.  Warp per row.
// ---------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(kThreads)
ns_rows_kernel(const T* __restrict__ ns_tokens, int64_t n, int ns, int64_t batch, int chunks, const T* __restrict__ gamma, float eps,
               const int64_t* __restrict__ token_rows, uint4* __restrict__ tokens, const int64_t* __restrict__ normed_rows,
               uint4* __restrict__ normed, uint4* __restrict__ token_major) {
    chain_release();
    chain_wait();
    constexpr int N = Vec16<T>::N;
    const int lane = threadIdx.x & 31;
    const int64_t i = static_cast<int64_t>(blockIdx.x) * kWarps + (threadIdx.x >> 5);
    if (i >= n) return;
    const int64_t b = i / ns, j = i - b * ns;
    const uint4* src = reinterpret_cast<const uint4*>(ns_tokens) + i * chunks;
    const int64_t m = j * batch + b;
    uint4* t_row = tokens + token_rows[m] * chunks;
    uint4* x_row = normed + normed_rows[m] * chunks;
    uint4* m_row = token_major + m * chunks;
    float sq = 0.f;
    for (int c = lane; c < chunks; c += 32) {
        const uint4 v = src[c];
        float f[N];
        Vec16<T>::unpack(v, f);
#pragma unroll
        for (int e = 0; e < N; ++e) sq = fmaf(f[e], f[e], sq);
        t_row[c] = v;
    }
    const float inv = rsqrtf(warp_sum(sq) / static_cast<float>(chunks * N) + eps);
    for (int c = lane; c < chunks; c += 32) {
        float f[N], g[N];
        Vec16<T>::unpack(src[c], f);
        Vec16<T>::unpack(reinterpret_cast<const uint4*>(gamma)[c], g);
#pragma unroll
        for (int e = 0; e < N; ++e) f[e] = (f[e] * inv) * g[e];
        const uint4 o = Vec16<T>::pack(f);
        x_row[c] = o;
        m_row[c] = o;
    }
}

// ---------------------------------------------------------------------------------------
// pool_rows: seq[b] = mean of rmsnorm(row) over the sample's sequence rows, ns[b] = the same over its ns non-sequence rows, in
// fp32 (no atomics: the order of the sum does not depend on scheduling).  With cu == nullptr the rows are token-major
// [ns, B, d] and there are no sequence rows.  The rows of a sample are dealt to the WPS warps that share it (8 where there are
// few samples and the chain of row loads is the time, 1 where there are many), each sums its own and the sums are added in the
// order of the warps.  Bound by the latency of the row loads: with one row at a time 8192 samples of 9 x 512 took 72 us,
// with four in flight and 16-byte stores 46 us.
// ---------------------------------------------------------------------------------------
template <typename T, int CPL, int WPS>
__global__ void __launch_bounds__(kThreads)
pool_rows_kernel(const uint4* __restrict__ rows, const int64_t* __restrict__ cu, const int64_t* __restrict__ counts, int64_t batch, int ns,
                 int chunks, const uint4* __restrict__ gamma, float eps, float* __restrict__ seq_out, float* __restrict__ ns_out) {
    chain_release();
    chain_wait();
    constexpr int N = Vec16<T>::N;
    extern __shared__ float sums[];          // [kWarps][d], WPS > 1 only
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t b = static_cast<int64_t>(blockIdx.x) * (kWarps / WPS) + warp / WPS;
    const bool live = b < batch;
    const int part = warp % WPS;
    const int d = chunks * N;
    const int64_t base = live ? (cu != nullptr ? cu[b] : b) : 0;
    const int64_t step = cu != nullptr ? 1 : batch;
    const int n_seq = live && cu != nullptr ? static_cast<int>(counts[b]) : 0;
    const float inv_d = 1.0f / static_cast<float>(d);
    float g[CPL][N];
#pragma unroll
    for (int k = 0; k < CPL; ++k) {
        const int c = lane + 32 * k;
#pragma unroll
        for (int e = 0; e < N; ++e) g[k][e] = 0.f;
        if (c < chunks) Vec16<T>::unpack(gamma[c], g[k]);
    }
    auto mean_of = [&](int first, int count, float* out) {
        float acc[CPL][N];
#pragma unroll
        for (int k = 0; k < CPL; ++k)
#pragma unroll
            for (int e = 0; e < N; ++e) acc[k][e] = 0.f;
        // U rows at a time: their loads and their reductions overlap, the sum keeps the order of the rows
        constexpr int U = WPS == 1 && CPL <= 2 ? 4 : 1;   // eight warps per sample have a row or two each
        for (int r0 = part; r0 < count; r0 += U * WPS) {
            float f[U][CPL][N], sq[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int r = r0 + u * WPS;
                const uint4* row = rows + (base + (first + (r < count ? r : r0)) * step) * chunks;
                sq[u] = 0.f;
#pragma unroll
                for (int k = 0; k < CPL; ++k) {
                    const int c = lane + 32 * k;
                    if (c < chunks) {
                        Vec16<T>::unpack(row[c], f[u][k]);
                    } else {
#pragma unroll
                        for (int e = 0; e < N; ++e) f[u][k][e] = 0.f;
                    }
#pragma unroll
                    for (int e = 0; e < N; ++e) sq[u] = fmaf(f[u][k][e], f[u][k][e], sq[u]);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) sq[u] = warp_sum(sq[u]);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (r0 + u * WPS < count) {
                    const float inv = rsqrtf(sq[u] * inv_d + eps);
#pragma unroll
                    for (int k = 0; k < CPL; ++k)
#pragma unroll
                        for (int e = 0; e < N; ++e) acc[k][e] += (f[u][k][e] * inv) * g[k][e];
                }
            }
        }
        const float denom = static_cast<float>(count > 0 ? count : 1);
        if (WPS > 1) {
#pragma unroll
            for (int k = 0; k < CPL; ++k) {
                const int c = lane + 32 * k;
                if (c < chunks) {
#pragma unroll
                    for (int e = 0; e < N; ++e) sums[warp * d + c * N + e] = acc[k][e];
                }
            }
            __syncthreads();
            if (live)
                for (int i = part * 32 + lane; i < d; i += 32 * WPS) {
                    float v = 0.f;
#pragma unroll
                    for (int w = 0; w < WPS; ++w) v += sums[(warp - part + w) * d + i];
                    out[b * d + i] = v / denom;
                }
            __syncthreads();
        } else if (live) {
#pragma unroll
            for (int k = 0; k < CPL; ++k) {
                const int c = lane + 32 * k;
                if (c < chunks) {
                    float* to = out + b * d + c * N;
                    if ((reinterpret_cast<uintptr_t>(out) & 15) == 0) {   // d is a multiple of 4: so is every row's start
#pragma unroll
                        for (int e = 0; e < N; e += 4)
                            *reinterpret_cast<float4*>(to + e) = make_float4(acc[k][e] / denom, acc[k][e + 1] / denom, acc[k][e + 2] / denom, acc[k][e + 3] / denom);
                    } else {
#pragma unroll
                        for (int e = 0; e < N; ++e) to[e] = acc[k][e] / denom;
                    }
                }
            }
        }
    };
    if (seq_out != nullptr) mean_of(0, n_seq, seq_out);
    mean_of(n_seq, live ? ns : 0, ns_out);
}

// embedding[b] = [seq[b] or zeros, ns[b]] in fp32, and as T for the classifier's GEMM (optional)
template <typename T>
__global__ void __launch_bounds__(kThreads)
join_summaries_kernel(const float* __restrict__ seq, const float* __restrict__ ns, float* __restrict__ joined, T* __restrict__ joined_t,
                      int64_t batch, int d) {
    chain_release();
    chain_wait();
    // whole rows per CTA and no 64-bit division: with one value per thread 8192 samples of 2 x 512 took 40 us, now 13 us
    const bool quads = d % 4 == 0 && ((reinterpret_cast<uintptr_t>(seq) | reinterpret_cast<uintptr_t>(ns) | reinterpret_cast<uintptr_t>(joined) |
                                       reinterpret_cast<uintptr_t>(joined_t)) & 15) == 0;
    const int width = quads ? d / 2 : 2 * d;                 // units of a joined row: four values, or one
    const int rows_here = width < kThreads ? kThreads / width : 1;
    const int own = width < kThreads ? static_cast<int>(threadIdx.x) / width : 0;
    if (own >= rows_here) return;
    for (int64_t b = static_cast<int64_t>(blockIdx.x) * rows_here + own; b < batch; b += static_cast<int64_t>(gridDim.x) * rows_here) {
        for (int i = static_cast<int>(threadIdx.x) - own * width; i < width; i += kThreads) {
            if (quads) {
                const int c = 4 * i;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (c >= d) v = *reinterpret_cast<const float4*>(ns + b * d + c - d);
                else if (seq != nullptr) v = *reinterpret_cast<const float4*>(seq + b * d + c);
                *reinterpret_cast<float4*>(joined + b * 2 * d + c) = v;
                if (joined_t != nullptr) {
                    T* to = joined_t + b * 2 * d + c;
                    to[0] = from_float<T>(v.x); to[1] = from_float<T>(v.y); to[2] = from_float<T>(v.z); to[3] = from_float<T>(v.w);
                }
            } else {
                const float v = i < d ? (seq != nullptr ? seq[b * d + i] : 0.f) : ns[b * d + i - d];
                joined[b * 2 * d + i] = v;
                if (joined_t != nullptr) joined_t[b * 2 * d + i] = from_float<T>(v);
            }
        }
    }
}

// logits[b, a] = h[b] . w[a] + bias[a], probs = sigmoid(logits), fp32.  Warp per sample.
template <typename T>
__global__ void __launch_bounds__(kThreads)
head_kernel(const T* __restrict__ h, const float* __restrict__ w, const float* __restrict__ bias, float* __restrict__ logits,
            float* __restrict__ probs, int64_t batch, int d, int actions) {
    chain_release();
    chain_wait();
    constexpr int N = Vec16<T>::N;
    const int lane = threadIdx.x & 31;
    const int64_t b = static_cast<int64_t>(blockIdx.x) * kWarps + (threadIdx.x >> 5);
    if (b >= batch) return;
    const uint4* row = reinterpret_cast<const uint4*>(h + b * d);
    for (int a = 0; a < actions; ++a) {
        float sum = 0.f;
        for (int c = lane; c < d / N; c += 32) {
            float f[N];
            Vec16<T>::unpack(row[c], f);
#pragma unroll
            for (int e = 0; e < N; ++e) sum = fmaf(f[e], w[static_cast<int64_t>(a) * d + c * N + e], sum);
        }
        sum = warp_sum(sum) + bias[a];
        if (lane == 0) {
            logits[b * actions + a] = sum;
            probs[b * actions + a] = 1.0f / (1.0f + expf(-sum));
        }
    }
}

unsigned warps_grid(int64_t n) { return static_cast<unsigned>((n + kWarps - 1) / kWarps); }

}  // namespace
}  // namespace tb200

#define TB200_BY_DTYPE(CALL)                                   \
    switch (dtype) {                                           \
        case TB200_F32: { using T = float; CALL; break; }      \
        case TB200_F16: { using T = __half; CALL; break; }     \
        case TB200_BF16: { using T = __nv_bfloat16; CALL; break; } \
        default: return TB200_ERR_DTYPE;                       \
    }

extern "C" int tb200_small_token_fwd(const float* values, int32_t n, int64_t value_stride, const uint8_t* mask, int64_t mask_stride,
                                     int32_t in_dim, const float* w, const float* bias, const float* gamma, const float* beta, void* out,
                                     int64_t out_stride, int64_t rows, int32_t d, float eps, int dtype, void* stream) {
    using namespace tb200;
    if (rows < 0 || n < 1 || d < 1 || in_dim < n || (mask != nullptr && in_dim != 2 * n) || out_stride < d) return TB200_ERR_SHAPE;
    if (rows == 0) return TB200_OK;
    if (values == nullptr || w == nullptr || bias == nullptr || gamma == nullptr || beta == nullptr || out == nullptr) return TB200_ERR_NULL;
    const size_t smem = static_cast<size_t>(kWarps) * (in_dim + d) * sizeof(float);
    if (smem > 48 * 1024 || rows > (1ll << 33)) return TB200_ERR_UNSUPPORTED;
    if (!device_info().valid) return TB200_ERR_DEVICE;
    TB200_BY_DTYPE((launch_chained(small_token_kernel<T>, warps_grid(rows), kThreads, smem, static_cast<cudaStream_t>(stream),
        values, n, value_stride, mask, mask_stride, in_dim, w, bias, gamma, beta, static_cast<T*>(out), out_stride, rows, d, eps)));
    count_launch();
    return launch_status();
}

extern "C" int tb200_ns_rows_fwd(const void* ns_tokens, int64_t batch, int32_t ns, int32_t d, const void* gamma, float eps,
                                 const int64_t* token_rows, void* tokens, const int64_t* normed_rows, void* normed, void* token_major,
                                 int dtype, void* stream) {
    using namespace tb200;
    if (batch < 0 || ns < 1 || d < 1) return TB200_ERR_SHAPE;
    if (batch == 0) return TB200_OK;
    const int es = dtype_size(dtype);
    if (es == 0) return TB200_ERR_DTYPE;
    if (ns_tokens == nullptr || gamma == nullptr || token_rows == nullptr || tokens == nullptr || normed_rows == nullptr ||
        normed == nullptr || token_major == nullptr)
        return TB200_ERR_NULL;
    if ((static_cast<int64_t>(d) * es) % 16 != 0 || !aligned16(ns_tokens) || !aligned16(gamma) || !aligned16(tokens) || !aligned16(normed) ||
        !aligned16(token_major))
        return TB200_ERR_ALIGN;
    if (batch * ns > (1ll << 33)) return TB200_ERR_SHAPE;
    if (!device_info().valid) return TB200_ERR_DEVICE;
    const int chunks = d * es / 16;
    TB200_BY_DTYPE((launch_chained(ns_rows_kernel<T>, warps_grid(batch * ns), kThreads, 0, static_cast<cudaStream_t>(stream),
        static_cast<const T*>(ns_tokens), batch * ns, ns, batch, chunks, static_cast<const T*>(gamma), eps, token_rows,
        static_cast<uint4*>(tokens), normed_rows, static_cast<uint4*>(normed), static_cast<uint4*>(token_major))));
    count_launch();
    return launch_status();
}

extern "C" int tb200_pool_rows_fwd(const void* rows, const int64_t* cu, const int64_t* counts, int64_t batch, int32_t ns, int32_t d,
                                   const void* gamma, float eps, float* seq_mean, float* ns_mean, int dtype, void* stream) {
    using namespace tb200;
    if (batch < 0 || ns < 1 || d < 1) return TB200_ERR_SHAPE;
    if (batch == 0) return TB200_OK;
    const int es = dtype_size(dtype);
    if (es == 0) return TB200_ERR_DTYPE;
    if (rows == nullptr || gamma == nullptr || ns_mean == nullptr || (cu != nullptr && (counts == nullptr || seq_mean == nullptr)))
        return TB200_ERR_NULL;
    if ((static_cast<int64_t>(d) * es) % 16 != 0 || !aligned16(rows) || !aligned16(gamma)) return TB200_ERR_ALIGN;
    const int chunks = d * es / 16;
    if (chunks > 256 || batch > (1ll << 33)) return TB200_ERR_UNSUPPORTED;
    if (!device_info().valid) return TB200_ERR_DEVICE;
    const bool few = batch < 8ll * device_info().sm_count && 8 * d * static_cast<int>(sizeof(float)) <= 48 * 1024;   // under eight samples per SM
    const dim3 grid = few ? dim3(static_cast<unsigned>(batch)) : dim3(warps_grid(batch));
    const size_t smem = few ? 8 * d * sizeof(float) : 0;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
#define TB200_POOL(CPL_)                                                                                                              \
    TB200_BY_DTYPE((launch_chained(few ? pool_rows_kernel<T, CPL_, 8> : pool_rows_kernel<T, CPL_, 1>, grid, kThreads, smem, st,       \
        static_cast<const uint4*>(rows), cu, counts, batch, ns, chunks, static_cast<const uint4*>(gamma), eps, seq_mean, ns_mean)))
    if (chunks <= 32) { TB200_POOL(1); }
    else if (chunks <= 64) { TB200_POOL(2); }
    else if (chunks <= 128) { TB200_POOL(4); }
    else { TB200_POOL(8); }
#undef TB200_POOL
    count_launch();
    return launch_status();
}

extern "C" int tb200_join_summaries(const float* seq, const float* ns, float* joined, void* joined_cast, int64_t batch, int32_t d, int dtype,
                                    void* stream) {
    using namespace tb200;
    if (batch < 0 || d < 1) return TB200_ERR_SHAPE;
    if (batch == 0) return TB200_OK;
    if (ns == nullptr || joined == nullptr) return TB200_ERR_NULL;
    if (batch * 2 * d > (1ll << 38)) return TB200_ERR_SHAPE;
    if (!device_info().valid) return TB200_ERR_DEVICE;
    const auto grid = static_cast<unsigned>(batch < (1 << 20) ? batch : (1 << 20));   // a CTA per sample at most; the kernel strides
    TB200_BY_DTYPE((launch_chained(join_summaries_kernel<T>, grid, kThreads, 0, static_cast<cudaStream_t>(stream), seq, ns, joined, static_cast<T*>(joined_cast),
                                                                                                     batch, d)));
    count_launch();
    return launch_status();
}

extern "C" int tb200_head_fwd(const void* h, const float* w, const float* bias, float* logits, float* probs, int64_t batch, int32_t d,
                              int32_t actions, int dtype, void* stream) {
    using namespace tb200;
    if (batch < 0 || d < 1 || actions < 1) return TB200_ERR_SHAPE;
    if (batch == 0) return TB200_OK;
    const int es = dtype_size(dtype);
    if (es == 0) return TB200_ERR_DTYPE;
    if (h == nullptr || w == nullptr || bias == nullptr || logits == nullptr || probs == nullptr) return TB200_ERR_NULL;
    if ((static_cast<int64_t>(d) * es) % 16 != 0 || !aligned16(h)) return TB200_ERR_ALIGN;
    if (batch > (1ll << 33)) return TB200_ERR_SHAPE;
    if (!device_info().valid) return TB200_ERR_DEVICE;
    TB200_BY_DTYPE((launch_chained(head_kernel<T>, warps_grid(batch), kThreads, 0, static_cast<cudaStream_t>(stream), static_cast<const T*>(h), w, bias, logits,
                                                                                                       probs, batch, d, actions)));
    count_launch();
    return launch_status();
}
