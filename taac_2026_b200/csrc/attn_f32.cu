// Attention forward in plain fp32 for the score-parity mode: fp32 q, k, v and o, every product, the softmax and
// the weighted sum in fp32, no tensor cores.  It exists so that a model whose dense layers run in fp32 can be
// compared with the reference's fp32 torch path without a 16-bit rounding of q, k and v in between.
//
// Head dims 32, 64 and 128 take attn_f32_tile_kernel.  A warp owns 16 queries of a (sample, head) and walks over 32-key tiles that it
// brings into its own shared memory by cp.async (no block-wide barrier).  A lane holds 4 x 4 scores (four queries, the keys c, c + 8,
// ...) and 4 x D / 8 outputs: per 16-byte shared-memory read eight multiply-adds, which leaves the fp32 units the bound; online softmax in
// registers.  512 samples of 16 .. 256 keys, 4 heads of 32, some 60 queries each: one query per warp took 137 us.
//
// Other head dims take attn_f32_kernel.  A warp owns one (sample, head, query): pass 1 gives every lane the keys j = lane, lane + 32, ... — the scaled
// dot products of the visible ones go to the warp's slice of shared memory — then the row maximum and the sum of
// exp2 are reduced across the lanes; pass 2 gives every lane the output dimensions d = lane, lane + 32, ... and
// walks all keys (coalesced reads of the value rows).  Same mask rule as the other kernels: valid prefix,
// always-valid suffix, causal, padded queries returning their own value row, packed batches with separate query
// offsets, or an explicit key-validity map.
#include "attn_common.cuh"
#include "tb200_common.cuh"

namespace tb200 {
void count_launch();

namespace {

constexpr int kWarps = 4;
constexpr int kMaxD = 256;

__global__ void __launch_bounds__(kWarps * 32)
attn_f32_kernel(const AttnArgs a, const int D, const int lk_cap) {
    chain_release();
    chain_wait();
    extern __shared__ float smem[];
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    float* qs = smem + warp * (kMaxD + lk_cap);   // the query row, then one score per key
    float* ps = qs + kMaxD;
    const int b = blockIdx.x;
    const int h = blockIdx.y;
    const int r = blockIdx.z * kWarps + warp;     // query index inside the sample

    const bool packed = a.cu_rows != nullptr;
    int lq = a.Lq, lk = a.Lk;
    int64_t row_base = 0, q_base = 0;
    if (packed) {
        row_base = a.cu_rows[b];
        lq = lk = a.cu_rows[b + 1] - static_cast<int32_t>(row_base);
        q_base = row_base;
        if (a.cu_rows_q != nullptr) {
            q_base = a.cu_rows_q[b];
            lq = a.cu_rows_q[b + 1] - static_cast<int32_t>(q_base);
        }
    }
    if (r >= lq) return;
    lk = min(lk, lk_cap);
    const int off = (packed && a.cu_rows_q != nullptr) ? max(lk - lq, 0) : 0;   // position of query 0 among the keys
    const int pos = r + off;
    const int valid_len = (a.seq_len != nullptr && !packed) ? min(max(a.seq_len[b], 0), lk) : lk;
    const int ns_start = packed ? lk : min(a.ns_start, lk);
    const bool causal = a.causal != 0;
    const uint8_t* kvalid = (a.key_valid != nullptr && !packed) ? a.key_valid + static_cast<int64_t>(b) * a.Lk : nullptr;

    const float* qp = static_cast<const float*>(a.q) + (packed ? q_base * a.q_sl : static_cast<int64_t>(b) * a.q_sb) +
                      static_cast<int64_t>(h) * a.q_sh + static_cast<int64_t>(r) * a.q_sl;
    const float* kp = static_cast<const float*>(a.k) + (packed ? row_base * a.k_sl : static_cast<int64_t>(b) * a.k_sb) + static_cast<int64_t>(h) * a.k_sh;
    const float* vp = static_cast<const float*>(a.v) + (packed ? row_base * a.v_sl : static_cast<int64_t>(b) * a.v_sb) + static_cast<int64_t>(h) * a.v_sh;
    float* op = static_cast<float*>(a.o) + (packed ? q_base * a.o_sl : static_cast<int64_t>(b) * a.o_sb) +
                static_cast<int64_t>(h) * a.o_sh + static_cast<int64_t>(r) * a.o_sl;

    // a padded query returns its own value row
    if (a.padded_query_self && !packed && pos < lk) {
        const bool padded_query = kvalid != nullptr ? kvalid[pos] == 0 : (pos >= valid_len && pos < ns_start);
        if (padded_query) {
            for (int d = lane; d < D; d += 32) op[d] = vp[static_cast<int64_t>(pos) * a.v_sl + d];
            return;
        }
    }
    for (int d = lane; d < D; d += 32) qs[d] = qp[d];
    __syncwarp();

    float row_max = -INFINITY;
    for (int j = lane; j < lk; j += 32) {
        const bool seen = kvalid != nullptr ? (kvalid[j] != 0 && (!causal || j <= pos))
                                            : attn_visible(pos, j, valid_len, ns_start, lk, causal);
        float s = -INFINITY;
        if (seen) {
            const float* kr = kp + static_cast<int64_t>(j) * a.k_sl;
            float dot = 0.f;
            for (int d = 0; d < D; ++d) dot = fmaf(qs[d], kr[d], dot);
            s = dot * a.scale_log2;
        }
        ps[j] = s;
        row_max = fmaxf(row_max, s);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) row_max = fmaxf(row_max, __shfl_xor_sync(0xffffffffu, row_max, o));
    if (row_max == -INFINITY) {   // no visible key: zeros
        for (int d = lane; d < D; d += 32) op[d] = 0.f;
        return;
    }
    float sum = 0.f;
    for (int j = lane; j < lk; j += 32) {
        const float p = exp2f(ps[j] - row_max);   // exp2f(-inf) = 0 for hidden keys
        ps[j] = p;
        sum += p;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    __syncwarp();
    const float inv = 1.0f / sum;
    const int last = causal ? min(lk, pos + 1) : lk;   // keys beyond the causal limit carry p = 0
    for (int d = lane; d < D; d += 32) {
        float acc = 0.f;
        for (int j = 0; j < last; ++j) acc = fmaf(ps[j], vp[static_cast<int64_t>(j) * a.v_sl + d], acc);
        op[d] = acc * inv;
    }
}

constexpr int kTileQ = 16;      // queries of a warp
constexpr int kTileK = 32;      // keys of a tile

__device__ __forceinline__ void cp16(float* smem, const float* gmem, bool ok) {
    const uint32_t at = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at), "l"(gmem), "r"(ok ? 16 : 0) : "memory");
}

template <int D>
constexpr int tile_floats() { return (2 * kTileK + kTileQ) * (D + 4) + kTileQ * (kTileK + 4); }   // K, V, Q, P of a warp

template <int D>
__global__ void __launch_bounds__(kWarps * 32)
attn_f32_tile_kernel(const AttnArgs a, const int q_tiles) {
    chain_release();
    chain_wait();
    constexpr int LD = D + 4;            // row stride in floats: eight lanes on eight rows hit eight different bank groups
    constexpr int LP = kTileK + 4;
    constexpr int DL = D / 8;            // output dimensions of a lane: d = c * 4 + 32 * i + (0 .. 3)
    extern __shared__ __align__(16) float f32_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t item = static_cast<int64_t>(blockIdx.x) * kWarps + warp;
    if (item >= static_cast<int64_t>(a.B) * a.H * q_tiles) return;
    const int b = static_cast<int>(item / (a.H * q_tiles));
    const int rem = static_cast<int>(item - static_cast<int64_t>(b) * a.H * q_tiles);
    const int h = rem / q_tiles, r0 = (rem - h * q_tiles) * kTileQ;

    const bool packed = a.cu_rows != nullptr;
    int lq = a.Lq, lk = a.Lk;
    int64_t row_base = 0, q_base = 0;
    if (packed) {
        row_base = a.cu_rows[b];
        lq = lk = a.cu_rows[b + 1] - static_cast<int32_t>(row_base);
        q_base = row_base;
        if (a.cu_rows_q != nullptr) {
            q_base = a.cu_rows_q[b];
            lq = a.cu_rows_q[b + 1] - static_cast<int32_t>(q_base);
        }
    }
    if (r0 >= lq) return;
    const int off = (packed && a.cu_rows_q != nullptr) ? max(lk - lq, 0) : 0;   // position of query 0 among the keys
    const int valid_len = (a.seq_len != nullptr && !packed) ? min(max(a.seq_len[b], 0), lk) : lk;
    const int ns_start = packed ? lk : min(a.ns_start, lk);
    const bool causal = a.causal != 0;
    const uint8_t* kvalid = (a.key_valid != nullptr && !packed) ? a.key_valid + static_cast<int64_t>(b) * a.Lk : nullptr;
    const float* qp = static_cast<const float*>(a.q) + (packed ? q_base * a.q_sl : static_cast<int64_t>(b) * a.q_sb) + static_cast<int64_t>(h) * a.q_sh;
    const float* kp = static_cast<const float*>(a.k) + (packed ? row_base * a.k_sl : static_cast<int64_t>(b) * a.k_sb) + static_cast<int64_t>(h) * a.k_sh;
    const float* vp = static_cast<const float*>(a.v) + (packed ? row_base * a.v_sl : static_cast<int64_t>(b) * a.v_sb) + static_cast<int64_t>(h) * a.v_sh;
    float* op = static_cast<float*>(a.o) + (packed ? q_base * a.o_sl : static_cast<int64_t>(b) * a.o_sb) + static_cast<int64_t>(h) * a.o_sh;

    float* sK = f32_smem + warp * tile_floats<D>();
    float* sV = sK + kTileK * LD;
    float* sQ = sV + kTileK * LD;
    float* sP = sQ + kTileQ * LD;
    const int rg = lane >> 3, c = lane & 7;     // queries 4 rg .. 4 rg + 3; keys c + 8 j
    auto load_rows = [&](float* dst, const float* src, int64_t stride, int row0, int n, int limit) {
        for (int i = lane; i < n * (D / 4); i += 32) {
            const int r = i / (D / 4), d4 = i - r * (D / 4);
            const bool ok = row0 + r < limit;
            cp16(dst + r * LD + d4 * 4, src + static_cast<int64_t>(ok ? row0 + r : 0) * stride + d4 * 4, ok);
        }
    };
    load_rows(sQ, qp, a.q_sl, r0, kTileQ, lq);

    const int q_end = min(r0 + kTileQ, lq);
    const int kv_end = causal ? min(lk, q_end + off) : lk;
    float acc[4][DL], m_run[4], l_run[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m_run[i] = -INFINITY;
        l_run[i] = 0.f;
#pragma unroll
        for (int e = 0; e < DL; ++e) acc[i][e] = 0.f;
    }
    for (int k0 = 0; k0 < kv_end; k0 += kTileK) {
        if (kvalid == nullptr && k0 >= valid_len && k0 + kTileK <= ns_start) continue;      // nothing visible
        load_rows(sK, kp, a.k_sl, k0, kTileK, lk);
        asm volatile("cp.async.commit_group;" ::: "memory");
        load_rows(sV, vp, a.v_sl, k0, kTileK, lk);
        asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        float s[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 4
        for (int d4 = 0; d4 < D / 4; ++d4) {
            float4 qv[4], kv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) qv[i] = *reinterpret_cast<const float4*>(sQ + (rg * 4 + i) * LD + d4 * 4);
#pragma unroll
            for (int j = 0; j < 4; ++j) kv[j] = *reinterpret_cast<const float4*>(sK + (c + 8 * j) * LD + d4 * 4);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    s[i][j] = fmaf(qv[i].x, kv[j].x, s[i][j]);
                    s[i][j] = fmaf(qv[i].y, kv[j].y, s[i][j]);
                    s[i][j] = fmaf(qv[i].z, kv[j].z, s[i][j]);
                    s[i][j] = fmaf(qv[i].w, kv[j].w, s[i][j]);
                }
        }
        const bool full = kvalid == nullptr && (k0 + kTileK <= valid_len || k0 >= ns_start) && k0 + kTileK <= lk &&
                          (!causal || k0 + kTileK - 1 <= r0 + off);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int pos = r0 + rg * 4 + i + off;
            float mx = -INFINITY;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int key = k0 + c + 8 * j;
                s[i][j] *= a.scale_log2;
                if (!full) {
                    const bool seen = key < lk && (kvalid != nullptr ? (kvalid[key] != 0 && (!causal || key <= pos))
                                                                     : attn_visible(pos, key, valid_len, ns_start, lk, causal));
                    if (!seen) s[i][j] = -INFINITY;
                }
                mx = fmaxf(mx, s[i][j]);
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const float m_new = fmaxf(m_run[i], mx);
            const float ref = m_new == -INFINITY ? 0.f : m_new;
            const float corr = exp2f(m_run[i] - ref);
            m_run[i] = m_new;
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float p = exp2f(s[i][j] - ref);
                sum += p;
                sP[(rg * 4 + i) * LP + c + 8 * j] = p;
            }
            l_run[i] = l_run[i] * corr + sum;
#pragma unroll
            for (int e = 0; e < DL; ++e) acc[i][e] *= corr;
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
#pragma unroll 2
        for (int j4 = 0; j4 < kTileK / 4; ++j4) {
            float4 pv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) pv[i] = *reinterpret_cast<const float4*>(sP + (rg * 4 + i) * LP + j4 * 4);
#pragma unroll
            for (int jj = 0; jj < 4; ++jj)
#pragma unroll
                for (int e4 = 0; e4 < DL / 4; ++e4) {
                    const float4 vv = *reinterpret_cast<const float4*>(sV + (j4 * 4 + jj) * LD + e4 * 32 + c * 4);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float p = jj == 0 ? pv[i].x : (jj == 1 ? pv[i].y : (jj == 2 ? pv[i].z : pv[i].w));
                        acc[i][e4 * 4 + 0] = fmaf(p, vv.x, acc[i][e4 * 4 + 0]);
                        acc[i][e4 * 4 + 1] = fmaf(p, vv.y, acc[i][e4 * 4 + 1]);
                        acc[i][e4 * 4 + 2] = fmaf(p, vv.z, acc[i][e4 * 4 + 2]);
                        acc[i][e4 * 4 + 3] = fmaf(p, vv.w, acc[i][e4 * 4 + 3]);
                    }
                }
        }
        __syncwarp();       // the tile is free for the next copies
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float l = l_run[i];
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
        const int r = r0 + rg * 4 + i;
        if (r >= lq) continue;
        const float inv = l > 0.f ? 1.0f / l : 0.f;      // no visible key: zeros
        const int pos = r + off;
        // a padded query returns its own value row
        const bool self = a.padded_query_self && !packed && pos < lk && (kvalid != nullptr ? kvalid[pos] == 0 : (pos >= valid_len && pos < ns_start));
#pragma unroll
        for (int e4 = 0; e4 < DL / 4; ++e4) {
            float4 o4 = make_float4(acc[i][e4 * 4] * inv, acc[i][e4 * 4 + 1] * inv, acc[i][e4 * 4 + 2] * inv, acc[i][e4 * 4 + 3] * inv);
            if (self) o4 = *reinterpret_cast<const float4*>(vp + static_cast<int64_t>(pos) * a.v_sl + e4 * 32 + c * 4);
            *reinterpret_cast<float4*>(op + static_cast<int64_t>(r) * a.o_sl + e4 * 32 + c * 4) = o4;
        }
    }
}

template <int D>
int launch_tiles(const AttnArgs& a, int max_lq, cudaStream_t stream) {
    const size_t smem = static_cast<size_t>(kWarps) * tile_floats<D>() * sizeof(float);
    static bool attr_set[64] = {};
    const DeviceInfo& dev = device_info();
    if (!attr_set[dev.index]) {
        cudaFuncSetAttribute(attn_f32_tile_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        attr_set[dev.index] = true;
    }
    const int q_tiles = (max_lq + kTileQ - 1) / kTileQ;
    const int64_t grid = (static_cast<int64_t>(a.B) * a.H * q_tiles + kWarps - 1) / kWarps;
    if (grid > 0x7FFFFFFFll) return TB200_ERR_SHAPE;
    launch_chained(attn_f32_tile_kernel<D>, static_cast<unsigned>(grid), kWarps * 32, smem, stream, a, q_tiles);
    count_launch();
    return launch_status();
}

}  // namespace

// fp32 tensors, head_dim up to 256, at most 8192 keys per sample.
int attn_f32_forward(const AttnArgs& a, int head_dim, int max_lq, int max_lk, cudaStream_t stream) {
    if (head_dim > kMaxD || max_lk > 8192) return TB200_ERR_UNSUPPORTED;
    switch (head_dim) {
        case 32: return launch_tiles<32>(a, max_lq, stream);
        case 64: return launch_tiles<64>(a, max_lq, stream);
        case 128: return launch_tiles<128>(a, max_lq, stream);
        default: break;
    }
    const int lk_cap = max_lk < 1 ? 1 : max_lk;
    const size_t smem = static_cast<size_t>(kWarps) * (kMaxD + lk_cap) * sizeof(float);
    static bool attr_set[64] = {};
    const DeviceInfo& dev = device_info();
    if (!attr_set[dev.index]) {
        cudaFuncSetAttribute(attn_f32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(kWarps * (kMaxD + 8192) * sizeof(float)));
        attr_set[dev.index] = true;
    }
    const unsigned row_blocks = static_cast<unsigned>((max_lq + kWarps - 1) / kWarps);
    if (a.H > 65535 || row_blocks > 65535) return TB200_ERR_SHAPE;
    dim3 grid(static_cast<unsigned>(a.B), static_cast<unsigned>(a.H), row_blocks);
    launch_chained(attn_f32_kernel, grid, kWarps * 32, smem, stream, a, head_dim, lk_cap);
    count_launch();
    return launch_status();
}

}  // namespace tb200
