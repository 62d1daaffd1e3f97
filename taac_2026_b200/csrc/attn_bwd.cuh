// Argument block and mask rule shared by the attention backward kernels.
#pragma once
#include "attn_common.cuh"

namespace tb200 {

struct BwdArgs {
    AttnArgs a;                 // q, k, v, o and their strides, the mask
    const void* d_o;            // strides of o
    void* dq;                   // strides of q
    void* dk;                   // strides of k
    void* dv;                   // strides of v
    float* lse;                 // [B, H, Lq]
    float* delta;               // [B, H, Lq]
    float scale;
};

struct RowMask {
    int valid_len, ns_start, lk;
    bool causal;
    const uint8_t* kvalid;
    __device__ __forceinline__ bool sees(int query, int key) const {
        return kvalid != nullptr ? (kvalid[key] != 0 && (!causal || key <= query))
                                 : attn_visible(query, key, valid_len, ns_start, lk, causal);
    }
    __device__ __forceinline__ bool padded_query(int pos) const {
        return kvalid != nullptr ? kvalid[pos] == 0 : (pos >= valid_len && pos < ns_start);
    }
};

__device__ __forceinline__ RowMask make_mask(const AttnArgs& a, int b) {
    RowMask m;
    m.lk = a.Lk;
    m.valid_len = a.seq_len != nullptr ? min(max(a.seq_len[b], 0), a.Lk) : a.Lk;
    m.ns_start = min(a.ns_start, a.Lk);
    m.causal = a.causal != 0;
    m.kvalid = a.key_valid != nullptr ? a.key_valid + static_cast<int64_t>(b) * a.Lk : nullptr;
    return m;
}

bool attn_bwd_mma_supported(const BwdArgs& g, int D, int dtype);
int attn_bwd_mma(const BwdArgs& g, int D, int dtype, cudaStream_t stream);

}  // namespace tb200
