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
    bool whole;                        // host side only: leave no pieces (the call is being captured)
};

// f32-accurate tiled kernel on CUDA cores (attn_prefill_f32.cu): every dtype, scales, any group size
bool prefill_f32_supported(uint32_t head_dim);
int32_t launch_prefill_f32(vfkv_ctx *ctx, uint32_t dtype, const PrefillParams &p, cudaStream_t st);

// tcgen05 kernel with one Q tile of 128 rows a CTA (attn_prefill_tc5s.cu): F8 (scaled or not) and F16 rows of 64,
// 128 or 256 dims, any group size.  split_q: F16 with Q as two half-precision terms (always for 64 and 256 dims)
bool prefill_one_tile_supported(const vfkv_ctx *ctx, uint32_t dtype, uint32_t head_dim);
int32_t launch_prefill_one_tile(vfkv_ctx *ctx, uint32_t dtype, bool split_q, const PrefillParams &p, cudaStream_t st);

// expected time of the call, in us
double prefill_one_tile_us(const vfkv_ctx *ctx, uint32_t dtype, bool split_q, const PrefillParams &p);

// shared by the tcgen05 kernels (attn_prefill_tc5.cu)
float *prefill_scratch(vfkv_ctx *ctx, cudaStream_t st, uint64_t *floats);
void prefill_scratch_used(vfkv_ctx *ctx, cudaStream_t st, const float *scratch);
bool encode_rows_map(vfkv_ctx *ctx, CUtensorMap *out, const void *base, uint64_t row_bytes, uint32_t rows, uint32_t box_rows);

#ifdef __CUDACC__
// Visible range [lo, hi) of query i (flash_attn_batch.comp:116-119,141-144; window: per-query bound).
__host__ __device__ __forceinline__ void query_range(const PrefillParams &p, uint32_t i, uint32_t *lo, uint32_t *hi)
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
