// Arguments of the chunked-prefill kernels over one sequence's slab and the visible range of a query.
#pragma once

#include "common.cuh"

namespace vfkv {

struct PrefillParams {
    const uint8_t *k, *v;              // rows of the slot: [pos][kv_head][dim]
    const float *k_scales, *v_scales;  // [pos][kv_head] or null
    const float *q;                    // [m][n_q_heads][dim]
    float *out;                        // [m][n_q_heads][dim]
    uint64_t row_bytes;
    uint32_t n_q_heads, n_kv_heads, group, head_dim, m, q_start, n_kv, kv_start, window;
    float scale, softcap;
};

// f32-accurate tiled kernel on CUDA cores (attn_prefill_f32.cu): every dtype, scales, any group size
bool prefill_f32_supported(uint32_t head_dim);
int32_t launch_prefill_f32(vfkv_ctx *ctx, uint32_t dtype, const PrefillParams &p, cudaStream_t st);

#ifdef __CUDACC__
// Visible range [lo, hi) of query i (flash_attn_batch.comp:116-119,141-144; window: per-query bound).
__device__ __forceinline__ void query_range(const PrefillParams &p, uint32_t i, uint32_t *lo, uint32_t *hi)
{
    uint32_t c = p.q_start + i + 1u;
    if (c > p.n_kv) c = p.n_kv;
    uint32_t l = p.kv_start;
    if (p.window != 0u && c > p.window && c - p.window > l) l = c - p.window;
    if (l > c) l = c;
    *lo = l; *hi = c;
}
#endif

}  // namespace vfkv
