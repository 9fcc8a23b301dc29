// CACHED_ATTENTION's operands and what its kernels share: which keys a query sees, how a position finds its row, what becomes of a
// score, and the softmax's closing factor (mixops.cu: the f32 kernels; attention_tc.cu: the tensor-core form).
#pragma once
#include "seq_common.cuh"

namespace {

// first position a query at p can see
__device__ __forceinline__ uint32_t mask_low(uint32_t p, uint32_t kind, uint32_t size) {
    if (kind == 1 || kind == 3) return p + 1 >= size ? p + 1 - size : 0;
    if (kind == 2) return p - p % size;
    return 0;
}
// mask 3: beside its window a query at p sees the mean row of every block of `pool` positions that lies wholly before the window
__device__ __forceinline__ uint32_t pooled_seen(uint32_t p, uint32_t size, uint32_t pool) { return p + 1 > size ? (p + 1 - size) / pool : 0; }
struct CaArgs {
    float* dst; const float* q; const float* kc; const float* vc; const float* ctl;
    uint32_t T, H, G, maps, dk, dv, q_rs, q_off, kw, k_off, vw, v_off, R, kind, size;
    float scale;
    const float* tab;      // score table [H * maps, tab_rs] by distance, or null
    uint32_t tab_rs, wkind;   // weights: 0 softmax over the visible keys, 1 sigmoid of every visible key (not normalised)
    float cap;             // > 0: the scaled score passes cap * tanh(s / cap)
    const void* sink;      // a learned score per (head, map) that joins the softmax's denominator only, or null
    uint32_t sink_bf16;    // its weight type
    float out_scale;       // the result is multiplied by it
    uint32_t dst_rs;       // row stride of dst (its first column is folded into the pointer)
    const float* kp; const float* vp;   // POOL: pooled rows [slots, pool_rows, kw] (laid out like the cache's), their key and value columns
    uint32_t pool, pool_rows;
    uint32_t early;        // (few rows) the cache's rows of earlier positions may be read before the launch's predecessor has completed
    uint32_t unslotted;    // the caches belong to the step (rows recomputed by the program), not to a state slot
};
__device__ __forceinline__ uint32_t ca_slot(const CaArgs& a) { return a.unslotted ? 0u : (uint32_t)ctl_word(a.ctl, ZG_CTL_SLOT); }
__device__ __forceinline__ float ca_score(const CaArgs& a, float dot) {
    const float s = dot * a.scale;
    return a.cap > 0.0f ? a.cap * tanhf(s / a.cap) : s;
}
__device__ __forceinline__ float ca_sink(const CaArgs& a, uint32_t hm) {
    return a.sink_bf16 ? __bfloat162float(reinterpret_cast<const bf16*>(a.sink)[hm]) : reinterpret_cast<const float*>(a.sink)[hm];
}
// 1 / (sum + exp(sink - max)): the sink's share of the denominator, in the frame of the running maximum
__device__ __forceinline__ float ca_inv_sum(const CaArgs& a, uint32_t hm, float mx, float l) {
    if (a.sink) l += expf(ca_sink(a, hm) - mx);
    return 1.0f / l;
}
// weight of a visible key under the unnormalised kind
__device__ __forceinline__ float ca_sigmoid(float s) { return __frcp_rn(1.0f + expf(-s)); }
constexpr int kCaMaxDv = 1024;   // 32 channels per lane in the per-query kernel
// Keys as a kernel counts them: positions of the cache, or (POOL) the pooled blocks some row of the tile can see, followed by the
// positions from k_lo on.  One softmax runs over both.
template <bool POOL>
struct CaKeys {
    const float* cache; const float* pooled;
    uint32_t R, width, k_lo, n_pool;
    __device__ __forceinline__ uint32_t first() const { return POOL ? 0u : k_lo; }
    __device__ __forceinline__ uint32_t count(uint32_t p_max) const { return p_max - k_lo + 1 + (POOL ? n_pool : 0u); }
    __device__ __forceinline__ bool is_pooled(uint32_t u) const { return POOL && u < n_pool; }
    __device__ __forceinline__ uint32_t position(uint32_t u) const { return POOL ? u - n_pool + k_lo : u; }
    __device__ __forceinline__ const float* row(uint32_t u) const { return is_pooled(u) ? pooled + (size_t)u * width : cache + (size_t)(position(u) % R) * width; }
    // whether a row at position p, whose window starts at lo and that sees nb blocks, sees key u
    __device__ __forceinline__ bool seen(uint32_t u, uint32_t p, uint32_t lo, uint32_t nb) const {
        if (is_pooled(u)) return u < nb;
        const uint32_t j = position(u);
        return j <= p && j >= lo;
    }
};
template <bool POOL>
__device__ __forceinline__ CaKeys<POOL> ca_keys(const float* cache, const float* pooled, uint32_t R, uint32_t width, uint32_t k_lo, uint32_t n_pool) {
    CaKeys<POOL> k;
    k.cache = cache; k.pooled = pooled; k.R = R; k.width = width; k.k_lo = k_lo; k.n_pool = POOL ? n_pool : 0u;
    return k;
}

}  // namespace
