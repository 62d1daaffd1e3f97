// Attention backward on the tensor cores for 16-bit tensors in the padded (B, H, L, D) layout, head_dim 32 / 64 / 128:
// dq, dk, dv from q, k, v, o and the upstream gradient, every mask family of the forward kernels (valid prefix,
// always-valid suffix, causal, key-validity map, padded queries that return their own value row).
//
// Two kernels and no atomics, so the gradients do not depend on scheduling:
//   attn_bwd_dq_kernel    64 query rows per CTA.  First walk over the key tiles: S = Q K^T, row maximum and sum.  Second
//                         walk: P = exp2(S - lse), dP = dO V^T, dS = P (dP - delta), dQ += dS K.  Writes dq and, for the
//                         second kernel, lse (log2 domain) and delta = rowsum(dO O).
//   attn_bwd_dkv_kernel   64 keys per CTA, everything transposed so that the accumulators belong to the keys:
//                         S^T = K Q^T, dP^T = V dO^T, dV += P^T dO, dK += dS^T Q.
// The 16-bit operands q, k, v, dO enter the products as they are, with fp32 accumulation.  P and dS are fp32 values that
// the second products need as 16-bit operands: each is split into a leading and a remainder part (x = hi + lo, both
// 16-bit, 16 significant bits together for bf16 and 22 for fp16) and both parts are multiplied, so the gradients keep
// what an fp32 evaluation gives before their own rounding.  fp16 holds 2^-24 .. 65504 only, and dS is as large or as small as the
// upstream gradient (loss scaling makes it 1e4 and more): every row of P and dS is multiplied by a power of two that brings its largest
// value so far to 2^14 .. 2^15, the accumulators are kept in that unit like those of an online softmax and divided by it at the end
// (fit_unit).  Against float64, dQ of 256 rows of 64 with dO of 1e-4: relative error 7.8e-4 (split without the unit: 1.1e-3, fp32 form:
// 7.8e-4, which is the rounding of the result); with dO of 2e4: 2.5e-4 (without: NaN, fp32 form: 2.5e-4).  The unit costs fp16 7 %
// (64 x 8 heads of 256 rows of 64, causal: 190 -> 205 us); bf16 has the range and does without.
//
// What bounds it: issue slots (softmax arithmetic, operand splits) next to the mma.sync rate; K, V, Q, dO tiles come out
// of the L2 after their first read.  64 x 64 tiles and four warps keep the fp32 accumulators and both score tiles in
// registers at three CTAs per SM for head_dim 64.
#include "attn_bwd.cuh"
#include "attn_mma_tile.cuh"
#include "tb200_common.cuh"

namespace tb200 {
void count_launch();

namespace {

constexpr int kM = 64;         // rows of a CTA's own tile and of the tiles it walks over
constexpr int kThreads = 128;  // four warps, 16 own rows each

template <typename T>
__device__ __forceinline__ float2 unpack_pair(uint32_t w);
template <>
__device__ __forceinline__ float2 unpack_pair<__nv_bfloat16>(uint32_t w) {
    return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
}
template <>
__device__ __forceinline__ float2 unpack_pair<__half>(uint32_t w) {
    return __half22float2(*reinterpret_cast<const __half2*>(&w));
}

// (x, y) = hi + lo, both parts pairs of T
template <typename T>
__device__ __forceinline__ void split_pair(float x, float y, uint32_t& hi, uint32_t& lo) {
    hi = pack2<T>(x, y);
    const float2 h = unpack_pair<T>(hi);
    lo = pack2<T>(x - h.x, y - h.y);
}

// Whether the split operands need the unit, and the unit that any value above 2^-85 replaces
template <typename T>
constexpr bool kUnit = false;
template <>
constexpr bool kUnit<__half> = true;
constexpr float kFirstUnit = 1.2676506002282294e30f;   // 2^100

__device__ __forceinline__ float one_over(float unit) { return __uint_as_float((254u << 23) - __float_as_uint(unit)); }   // a power of two

// unit[hr]: the power of two of the thread's rows g (hr 0) and g + 8 (hr 1); the accumulators follow when it changes
template <int D, int NX>
__device__ __forceinline__ void fit_unit(const float (&x)[NX][4], float (&unit)[2], float (&acc)[D / 8][4]) {
#pragma unroll
    for (int hr = 0; hr < 2; ++hr) {
        float m = 0.f;
#pragma unroll
        for (int j = 0; j < NX; ++j) m = fmaxf(m, fmaxf(fabsf(x[j][2 * hr]), fabsf(x[j][2 * hr + 1])));
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
        if (m * unit[hr] >= 32768.f) {
            const float next = __uint_as_float((268u - (__float_as_uint(m) >> 23)) << 23);   // m next in [2^14, 2^15)
            const float f = next * one_over(unit[hr]);
            unit[hr] = next;
#pragma unroll
            for (int j = 0; j < D / 8; ++j) {
                acc[j][2 * hr] *= f;
                acc[j][2 * hr + 1] *= f;
            }
        }
    }
}
template <int D>
__device__ __forceinline__ void drop_unit(float (&acc)[D / 8][4], const float (&unit)[2]) {
#pragma unroll
    for (int j = 0; j < D / 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[j][e] *= one_over(unit[e >> 1]);
}

// rows [row0, row0 + 64) of a [*, D] strided matrix -> swizzled shared tile; rows >= n_rows are zero
template <typename T, int D>
__device__ __forceinline__ void load_rows(T* smem, const T* gmem, int64_t stride_l, int row0, int n_rows) {
    constexpr int CH = D / 8;
#pragma unroll
    for (int i = threadIdx.x; i < kM * CH; i += kThreads) {
        const int r = i / CH;
        const int c = i - r * CH;
        const bool ok = row0 + r < n_rows;
        cp_async16(smem + swz<D>(r, c), gmem + static_cast<int64_t>(ok ? row0 + r : 0) * stride_l + c * 8, ok);
    }
}

// c[j] (+)= A (16 rows of this warp, from registers) x B^T, B = 16 NJ rows x D of a shared tile (both K-major)
template <typename T, int D, int NJ>
__device__ __forceinline__ void product_nt(float (&c)[2 * NJ][4], const uint32_t (&af)[D / 16][4], const T* tile, int row0) {
    const int lane = threadIdx.x & 31, mi = lane >> 3;
#pragma unroll
    for (int j = 0; j < 2 * NJ; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) c[j][e] = 0.f;
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) {
#pragma unroll
        for (int jp = 0; jp < NJ; ++jp) {
            uint32_t b[4];
            ldsm_x4(b, tile + swz<D>(row0 + jp * 16 + (mi >> 1) * 8 + (lane & 7), kk * 2 + (mi & 1)));
            mma16816<T>(c[2 * jp], af[kk], b[0], b[1]);
            mma16816<T>(c[2 * jp + 1], af[kk], b[2], b[3]);
        }
    }
}

// acc += X (16 x 16 NK, fp32 accumulator layout, split into two 16-bit parts) x B, B = rows [row0, row0 + 16 NK) x D
template <typename T, int D, int NK>
__device__ __forceinline__ void product_nn(float (&acc)[D / 8][4], float (&x)[2 * NK][4], const T* tile, int row0, float (&unit)[2]) {
    if constexpr (kUnit<T>) {
        fit_unit<D, 2 * NK>(x, unit, acc);
#pragma unroll
        for (int j = 0; j < 2 * NK; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) x[j][e] *= unit[e >> 1];
    }
    const int lane = threadIdx.x & 31, mi = lane >> 3;
#pragma unroll
    for (int kk = 0; kk < NK; ++kk) {
        uint32_t hi[4], lo[4];
        split_pair<T>(x[2 * kk][0], x[2 * kk][1], hi[0], lo[0]);
        split_pair<T>(x[2 * kk][2], x[2 * kk][3], hi[1], lo[1]);
        split_pair<T>(x[2 * kk + 1][0], x[2 * kk + 1][1], hi[2], lo[2]);
        split_pair<T>(x[2 * kk + 1][2], x[2 * kk + 1][3], hi[3], lo[3]);
#pragma unroll
        for (int jp = 0; jp < D / 16; ++jp) {
            uint32_t b[4];
            ldsm_x4_t(b, tile + swz<D>(row0 + kk * 16 + (mi & 1) * 8 + (lane & 7), jp * 2 + (mi >> 1)));
            mma16816<T>(acc[2 * jp], hi, b[0], b[1]);
            mma16816<T>(acc[2 * jp + 1], hi, b[2], b[3]);
            mma16816<T>(acc[2 * jp], lo, b[0], b[1]);
            mma16816<T>(acc[2 * jp + 1], lo, b[2], b[3]);
        }
    }
}

template <typename T, int D>
__device__ __forceinline__ void load_frags(uint32_t (&f)[D / 16][4], const T* tile) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) ldsm_x4(f[kk], tile + swz<D>(warp * 16 + (lane & 15), kk * 2 + (lane >> 4)));
}

// the warp's 16 x D accumulators, scaled -> T in the shared tile (rows warp * 16 ..), for 16-byte stores
template <typename T, int D>
__device__ __forceinline__ void stage_rows(T* tile, const float (&acc)[D / 8][4], float scale) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int j = 0; j < D / 8; ++j) {
        *reinterpret_cast<uint32_t*>(tile + swz<D>(warp * 16 + g, j) + 2 * t) = pack2<T>(acc[j][0] * scale, acc[j][1] * scale);
        *reinterpret_cast<uint32_t*>(tile + swz<D>(warp * 16 + g + 8, j) + 2 * t) = pack2<T>(acc[j][2] * scale, acc[j][3] * scale);
    }
}
template <typename T, int D>
__device__ __forceinline__ void store_rows(T* gmem, int64_t stride_l, const T* tile, int row0, int n_rows) {
    constexpr int CH = D / 8;
    for (int i = threadIdx.x; i < kM * CH; i += kThreads) {
        const int r = i / CH;
        const int c = i - r * CH;
        if (row0 + r < n_rows)
            *reinterpret_cast<uint4*>(gmem + static_cast<int64_t>(row0 + r) * stride_l + c * 8) = *reinterpret_cast<const uint4*>(tile + swz<D>(r, c));
    }
}

template <typename T, int D>
__global__ void __launch_bounds__(kThreads, D <= 64 ? 3 : 2)
attn_bwd_dq_kernel(const BwdArgs g) {
    chain_release();
    chain_wait();
    extern __shared__ __align__(128) uint8_t smem_raw[];
    __shared__ float s_delta[kM];
    T* sQ = reinterpret_cast<T*>(smem_raw);
    T* sG = sQ + kM * D;
    T* sK = sG + kM * D;       // two stages
    T* sV = sK + 2 * kM * D;   // two stages
    const AttnArgs& a = g.a;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int gr = lane >> 2, t = lane & 3;
    const int b = blockIdx.z, h = blockIdx.y;
    // later query tiles see more keys under a causal mask: they go first
    const int m0 = (static_cast<int>(gridDim.x) - 1 - static_cast<int>(blockIdx.x)) * kM;
    const int m_end = min(m0 + kM, a.Lq);
    const RowMask mask = make_mask(a, b);
    const T* q = static_cast<const T*>(a.q) + b * a.q_sb + h * a.q_sh;
    const T* k = static_cast<const T*>(a.k) + b * a.k_sb + h * a.k_sh;
    const T* v = static_cast<const T*>(a.v) + b * a.v_sb + h * a.v_sh;
    const T* o = static_cast<const T*>(a.o) + b * a.o_sb + h * a.o_sh;
    const T* d_o = static_cast<const T*>(g.d_o) + b * a.o_sb + h * a.o_sh;
    T* dq = static_cast<T*>(g.dq) + b * a.q_sb + h * a.q_sh;
    const int64_t row_base = (static_cast<int64_t>(b) * a.H + h) * a.Lq;

    const int kv_end = mask.causal ? min(a.Lk, m_end) : a.Lk;
    const int n_tiles = (kv_end + kM - 1) / kM;
    const bool self_rows = a.padded_query_self != 0;
    const bool all_padded = self_rows && mask.kvalid == nullptr && m0 >= mask.valid_len && m_end <= mask.ns_start;
    auto next_live = [&](int n) {
        for (++n; n < n_tiles; ++n)
            if (mask.kvalid != nullptr || n * kM < mask.valid_len || n * kM + kM > mask.ns_start) break;
        return n;
    };
    const int first = all_padded ? n_tiles : next_live(-1);

    float acc[D / 8][4];
#pragma unroll
    for (int j = 0; j < D / 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;

    if (first < n_tiles) {
        load_rows<T, D>(sQ, q, a.q_sl, m0, a.Lq);
        load_rows<T, D>(sG, d_o, a.o_sl, m0, a.Lq);
        load_rows<T, D>(sK, k, a.k_sl, first * kM, a.Lk);
        cp_async_commit();
    }
    // delta = rowsum(dO O), two threads per row
    {
        const int r = threadIdx.x >> 1, half = threadIdx.x & 1;
        float sum = 0.f;
        if (m0 + r < a.Lq) {
            const uint4* op = reinterpret_cast<const uint4*>(o + static_cast<int64_t>(m0 + r) * a.o_sl) + half * (D / 16);
            const uint4* gp = reinterpret_cast<const uint4*>(d_o + static_cast<int64_t>(m0 + r) * a.o_sl) + half * (D / 16);
#pragma unroll
            for (int c = 0; c < D / 16; ++c) {
                float x[8], y[8];
                Vec16<T>::unpack(op[c], x);
                Vec16<T>::unpack(gp[c], y);
#pragma unroll
                for (int e = 0; e < 8; ++e) sum = fmaf(x[e], y[e], sum);
            }
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        if (half == 0) s_delta[r] = sum;
    }

    float unit[2] = {kFirstUnit, kFirstUnit};
    float lse[2] = {INFINITY, INFINITY};   // +inf: every probability of the row is 0
    if (first < n_tiles) {
        uint32_t qf[D / 16][4];
        float row_m[2] = {-INFINITY, -INFINITY}, row_l[2] = {0.f, 0.f};
        auto scores = [&](float (&s)[8][4], const T* tile, int n) {
            product_nt<T, D, 4>(s, qf, tile, 0);
            const int n0 = n * kM;
            const bool full = mask.kvalid == nullptr && (n0 + kM <= mask.valid_len || n0 >= mask.ns_start) && n0 + kM <= a.Lk &&
                              (!mask.causal || n0 + kM - 1 <= m0);
            if (!full) {
#pragma unroll
                for (int j = 0; j < 8; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int r = m0 + warp * 16 + gr + ((e >> 1) << 3), c = n0 + j * 8 + 2 * t + (e & 1);
                        if (c >= a.Lk || !mask.sees(r, c)) s[j][e] = -INFINITY;
                    }
            }
        };
        // first walk: row maximum and sum
        int stage = 0;
        bool have_q = false;
        for (int n = first; n < n_tiles;) {
            const int next = next_live(n);
            if (next < n_tiles) load_rows<T, D>(sK + (stage ^ 1) * kM * D, k, a.k_sl, next * kM, a.Lk);
            cp_async_commit();
            cp_async_wait<1>();
            __syncthreads();
            if (!have_q) {
                load_frags<T, D>(qf, sQ);
                have_q = true;
            }
            float s[8][4];
            scores(s, sK + stage * kM * D, n);
#pragma unroll
            for (int hr = 0; hr < 2; ++hr) {
                float mx = row_m[hr];
#pragma unroll
                for (int j = 0; j < 8; ++j) mx = fmaxf(mx, fmaxf(s[j][2 * hr], s[j][2 * hr + 1]));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
                const float ms = (mx == -INFINITY ? 0.f : mx) * a.scale_log2;
                float sum = 0.f;
#pragma unroll
                for (int j = 0; j < 8; ++j) sum += ex2_approx(fmaf(s[j][2 * hr], a.scale_log2, -ms)) + ex2_approx(fmaf(s[j][2 * hr + 1], a.scale_log2, -ms));
                row_l[hr] = row_l[hr] * ex2_approx(row_m[hr] * a.scale_log2 - ms) + sum;
                row_m[hr] = mx;
            }
            __syncthreads();
            stage ^= 1;
            n = next;
        }
        load_rows<T, D>(sK + stage * kM * D, k, a.k_sl, first * kM, a.Lk);
        load_rows<T, D>(sV + stage * kM * D, v, a.v_sl, first * kM, a.Lk);
        cp_async_commit();
        float delta[2];
#pragma unroll
        for (int hr = 0; hr < 2; ++hr) {
            float l = row_l[hr];
            l += __shfl_xor_sync(0xffffffffu, l, 1);
            l += __shfl_xor_sync(0xffffffffu, l, 2);
            const int r = m0 + warp * 16 + gr + 8 * hr;
            const bool padded = self_rows && r < a.Lq && r < a.Lk && mask.padded_query(r);
            if (l > 0.f && !padded) lse[hr] = row_m[hr] * a.scale_log2 + log2f(l);
            delta[hr] = s_delta[warp * 16 + gr + 8 * hr];
        }
        // second walk: dQ
        uint32_t gf[D / 16][4];
        load_frags<T, D>(gf, sG);
        for (int n = first; n < n_tiles;) {
            const int next = next_live(n);
            if (next < n_tiles) {
                load_rows<T, D>(sK + (stage ^ 1) * kM * D, k, a.k_sl, next * kM, a.Lk);
                load_rows<T, D>(sV + (stage ^ 1) * kM * D, v, a.v_sl, next * kM, a.Lk);
            }
            cp_async_commit();
            cp_async_wait<1>();
            __syncthreads();
            float s[8][4], dp[8][4];
            scores(s, sK + stage * kM * D, n);
            product_nt<T, D, 4>(dp, gf, sV + stage * kM * D, 0);
#pragma unroll
            for (int j = 0; j < 8; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float p = ex2_approx(fmaf(s[j][e], a.scale_log2, -lse[e >> 1]));
                    s[j][e] = p * (dp[j][e] - delta[e >> 1]);
                }
            product_nn<T, D, 4>(acc, s, sK + stage * kM * D, 0, unit);
            __syncthreads();
            stage ^= 1;
            n = next;
        }
        cp_async_wait<0>();
    }
    __syncthreads();
    if (t == 0) {
#pragma unroll
        for (int hr = 0; hr < 2; ++hr) {
            const int r = warp * 16 + gr + 8 * hr;
            if (m0 + r < a.Lq) {
                g.lse[row_base + m0 + r] = lse[hr];
                g.delta[row_base + m0 + r] = s_delta[r];
            }
        }
    }
    if constexpr (kUnit<T>) drop_unit<D>(acc, unit);
    stage_rows<T, D>(sQ, acc, g.scale);
    __syncthreads();
    store_rows<T, D>(dq, a.q_sl, sQ, m0, a.Lq);
}

template <typename T, int D>
__global__ void __launch_bounds__(kThreads, D <= 64 ? 3 : 2)
attn_bwd_dkv_kernel(const BwdArgs g) {
    chain_release();
    chain_wait();
    extern __shared__ __align__(128) uint8_t smem_raw[];
    __shared__ __align__(16) float s_lse[2][kM];
    __shared__ __align__(16) float s_delta[2][kM];
    T* sK = reinterpret_cast<T*>(smem_raw);
    T* sV = sK + kM * D;
    T* sQ = sV + kM * D;       // two stages
    T* sG = sQ + 2 * kM * D;   // two stages
    const AttnArgs& a = g.a;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int gr = lane >> 2, t = lane & 3;
    const int b = blockIdx.z, h = blockIdx.y;
    const int k0 = blockIdx.x * kM;     // under a causal mask the first keys are seen by most queries: they go first
    const RowMask mask = make_mask(a, b);
    const T* q = static_cast<const T*>(a.q) + b * a.q_sb + h * a.q_sh;
    const T* k = static_cast<const T*>(a.k) + b * a.k_sb + h * a.k_sh;
    const T* v = static_cast<const T*>(a.v) + b * a.v_sb + h * a.v_sh;
    const T* d_o = static_cast<const T*>(g.d_o) + b * a.o_sb + h * a.o_sh;
    T* dk = static_cast<T*>(g.dk) + b * a.k_sb + h * a.k_sh;
    T* dv = static_cast<T*>(g.dv) + b * a.v_sb + h * a.v_sh;
    const float* lse = g.lse + (static_cast<int64_t>(b) * a.H + h) * a.Lq;
    const float* delta = g.delta + (static_cast<int64_t>(b) * a.H + h) * a.Lq;

    const bool self_rows = a.padded_query_self != 0;
    const bool dead = mask.kvalid == nullptr && k0 >= mask.valid_len && k0 + kM <= mask.ns_start;   // no key of the tile is visible
    const int n_tiles = dead ? 0 : (a.Lq + kM - 1) / kM;
    auto next_live = [&](int n) {   // query tiles with a row that may see a key of this tile
        for (++n; n < n_tiles; ++n) {
            const int q_end = min(n * kM + kM, a.Lq);
            if (mask.causal && q_end <= k0) continue;
            if (self_rows && mask.kvalid == nullptr && n * kM >= mask.valid_len && q_end <= mask.ns_start) continue;
            break;
        }
        return n;
    };
    auto load_queries = [&](int stage, int n) {
        load_rows<T, D>(sQ + stage * kM * D, q, a.q_sl, n * kM, a.Lq);
        load_rows<T, D>(sG + stage * kM * D, d_o, a.o_sl, n * kM, a.Lq);
    };
    auto load_stats = [&](int stage, int n) {
        if (threadIdx.x < kM) {
            const int r = n * kM + threadIdx.x;
            s_lse[stage][threadIdx.x] = r < a.Lq ? lse[r] : INFINITY;
            s_delta[stage][threadIdx.x] = r < a.Lq ? delta[r] : 0.f;
        }
    };

    float acc_k[D / 8][4], acc_v[D / 8][4];
#pragma unroll
    for (int j = 0; j < D / 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc_k[j][e] = acc_v[j][e] = 0.f;

    float unit_k[2] = {kFirstUnit, kFirstUnit}, unit_v[2] = {kFirstUnit, kFirstUnit};
    const int first = next_live(-1);
    if (first < n_tiles) {
        load_rows<T, D>(sK, k, a.k_sl, k0, a.Lk);
        load_rows<T, D>(sV, v, a.v_sl, k0, a.Lk);
        load_queries(0, first);
        load_stats(0, first);
        cp_async_commit();
        int stage = 0;
        constexpr bool kKeep = D <= 64;           // the K / V fragments stay in registers where they fit
        uint32_t kf[D / 16][4], vf[D / 16][4];
        bool have = false;
        for (int n = first; n < n_tiles;) {
            const int next = next_live(n);
            if (next < n_tiles) {
                load_queries(stage ^ 1, next);
                load_stats(stage ^ 1, next);
            }
            cp_async_commit();
            cp_async_wait<1>();
            __syncthreads();
            if (kKeep && !have) {
                load_frags<T, D>(kf, sK);
                load_frags<T, D>(vf, sV);
                have = true;
            }
            const T* tq = sQ + stage * kM * D;
            const T* tg = sG + stage * kM * D;
            const int q0 = n * kM;
            const bool full = mask.kvalid == nullptr && (k0 + kM <= mask.valid_len || k0 >= mask.ns_start) && k0 + kM <= a.Lk &&
                              (!mask.causal || k0 + kM - 1 <= q0);
#pragma unroll 1
            for (int part = 0; part < 2; ++part) {   // 32 queries at a time: half the score registers
                float s[4][4], dp[4][4];
                if (!kKeep) load_frags<T, D>(kf, sK);
                product_nt<T, D, 2>(s, kf, tq, part * 32);
                if (!kKeep) load_frags<T, D>(vf, sV);
                product_nt<T, D, 2>(dp, vf, tg, part * 32);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int cq = part * 32 + j * 8 + 2 * t;
                    const float2 l2 = *reinterpret_cast<const float2*>(&s_lse[stage][cq]);
                    const float2 d2 = *reinterpret_cast<const float2*>(&s_delta[stage][cq]);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        float p = ex2_approx(fmaf(s[j][e], a.scale_log2, -((e & 1) ? l2.y : l2.x)));
                        if (!full) {
                            const int key = k0 + warp * 16 + gr + ((e >> 1) << 3), row = q0 + cq + (e & 1);
                            if (key >= a.Lk || !mask.sees(row, key)) p = 0.f;
                        }
                        s[j][e] = p;
                        dp[j][e] = p * (dp[j][e] - ((e & 1) ? d2.y : d2.x));
                    }
                }
                product_nn<T, D, 2>(acc_v, s, tg, part * 32, unit_v);
                product_nn<T, D, 2>(acc_k, dp, tq, part * 32, unit_k);
            }
            __syncthreads();
            stage ^= 1;
            n = next;
        }
        cp_async_wait<0>();
    }
    __syncthreads();
    if constexpr (kUnit<T>) {
        drop_unit<D>(acc_k, unit_k);
        drop_unit<D>(acc_v, unit_v);
    }
    if (self_rows) {   // a padded query returned its own value row: its gradient goes straight there
#pragma unroll
        for (int hr = 0; hr < 2; ++hr) {
            const int r = k0 + warp * 16 + gr + 8 * hr;
            if (r < a.Lk && r < a.Lq && mask.padded_query(r)) {
#pragma unroll
                for (int j = 0; j < D / 8; ++j) {
                    const float2 x = unpack_pair<T>(*reinterpret_cast<const uint32_t*>(d_o + static_cast<int64_t>(r) * a.o_sl + j * 8 + 2 * t));
                    acc_v[j][2 * hr] += x.x;
                    acc_v[j][2 * hr + 1] += x.y;
                }
            }
        }
    }
    stage_rows<T, D>(sK, acc_k, g.scale);
    stage_rows<T, D>(sV, acc_v, 1.f);
    __syncthreads();
    store_rows<T, D>(dk, a.k_sl, sK, k0, a.Lk);
    store_rows<T, D>(dv, a.v_sl, sV, k0, a.Lk);
}

template <typename T, int D>
int launch(const BwdArgs& g, cudaStream_t stream) {
    const AttnArgs& a = g.a;
    const size_t smem = static_cast<size_t>(6) * kM * D * sizeof(T);
    static bool attr_set[64] = {};
    const DeviceInfo& dev = device_info();
    if (!attr_set[dev.index]) {
        cudaFuncSetAttribute(attn_bwd_dq_kernel<T, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        cudaFuncSetAttribute(attn_bwd_dkv_kernel<T, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        attr_set[dev.index] = true;
    }
    launch_chained(attn_bwd_dq_kernel<T, D>, dim3((a.Lq + kM - 1) / kM, a.H, a.B), kThreads, smem, stream, g);
    count_launch();
    const int code = launch_status();
    if (code != TB200_OK) return code;
    launch_chained(attn_bwd_dkv_kernel<T, D>, dim3((a.Lk + kM - 1) / kM, a.H, a.B), kThreads, smem, stream, g);
    count_launch();
    return launch_status();
}

template <typename T>
int launch_dim(const BwdArgs& g, int D, cudaStream_t stream) {
    switch (D) {
        case 32: return launch<T, 32>(g, stream);
        case 64: return launch<T, 64>(g, stream);
        default: return launch<T, 128>(g, stream);
    }
}

}  // namespace

// 16-bit tensors whose rows start on 16-byte boundaries, head_dim 32 / 64 / 128 (grid limits: B and H up to 65535)
bool attn_bwd_mma_supported(const BwdArgs& g, int D, int dtype) {
    const AttnArgs& a = g.a;
    if ((dtype != TB200_BF16 && dtype != TB200_F16) || (D != 32 && D != 64 && D != 128) || a.B > 65535) return false;
    for (const void* p : {a.q, a.k, a.v, static_cast<const void*>(a.o), g.d_o, static_cast<const void*>(g.dq), static_cast<const void*>(g.dk),
                          static_cast<const void*>(g.dv)})
        if (!aligned16(p)) return false;
    for (int64_t s : {a.q_sb, a.q_sh, a.q_sl, a.k_sb, a.k_sh, a.k_sl, a.v_sb, a.v_sh, a.v_sl, a.o_sb, a.o_sh, a.o_sl})
        if (s % 8 != 0) return false;
    return true;
}
int attn_bwd_mma(const BwdArgs& g, int D, int dtype, cudaStream_t stream) {
    return dtype == TB200_BF16 ? launch_dim<__nv_bfloat16>(g, D, stream) : launch_dim<__half>(g, D, stream);
}

}  // namespace tb200
