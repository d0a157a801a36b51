// RoPE-NeoX fused with the KV append, and the same rotation for Q rows.
//
// In the reference one layer's K goes through a rope dispatch (run_rope_neox*, host
// src/backend/vulkan/forward/runs.rs:647-720, math vk_shaders/rope_funcs.glsl:73-107), a pipeline
// barrier, and then kv_store_fp8 / kv_copy_fp16 (executor/attention.rs:435-530, :546-596): the
// rotated row makes a round trip through memory in f32.  Here the rotation happens in the
// registers of the thread that encodes the cache bytes, and K and V share one launch.
//
// The angle follows the CPU form the reference grades against (tests/correctness.rs:827-838):
// theta_i = pos * theta_scale^i with theta_scale = freq_base^(-2 / n_dims) computed once in f32
// and the powers taken by repeated multiplication.  They depend on the row and the pair alone, so a
// block makes the sines and cosines of its rows once, in shared memory, and all heads use them;
// what is left is the rows' own traffic.  (A chain of up to n_dims / 2 multiplications and a sincosf
// for every element had the time: Q of 2048 rows, 32 heads of 128: 36 us; 67 MB are 10 us.)
#include <cmath>

#include "../../include/vfkv_next.h"
#include "common.cuh"
#include "fp8_codec.cuh"

namespace vfkv {

struct RopeAppendParams {
    const float *k, *v;
    uint8_t *k_dst, *v_dst;                // layer base (slot 0)
    float *k_rot;                          // optional f32 copy of the rotated K rows
    const uint32_t *slot_ids, *positions;  // batch mode when positions != null
    uint64_t slot_stride_bytes;
    uint32_t row_elems, head_dim, n_kv_heads, max_seq, n_slots, n_rows, slot, base_pos;
    uint32_t n_dims;
    float theta_scale, freq_scale;
    uint32_t *status;
};

template <int DT> struct Pack;
template <> struct Pack<VFKV_F8> {
    static constexpr int kElems = 16, kBytes = 1;
    __device__ static uint4 run(const float *x)
    {
        return make_uint4(f32x4_to_e4m3x4(x[0], x[1], x[2], x[3]), f32x4_to_e4m3x4(x[4], x[5], x[6], x[7]),
                          f32x4_to_e4m3x4(x[8], x[9], x[10], x[11]), f32x4_to_e4m3x4(x[12], x[13], x[14], x[15]));
    }
};
template <> struct Pack<VFKV_F16> {
    static constexpr int kElems = 8, kBytes = 2;
    __device__ static uint4 run(const float *x)
    {
        return make_uint4(f32x2_to_f16x2(x[0], x[1]), f32x2_to_f16x2(x[2], x[3]), f32x2_to_f16x2(x[4], x[5]),
                          f32x2_to_f16x2(x[6], x[7]));
    }
};
template <> struct Pack<VFKV_F32> {
    static constexpr int kElems = 4, kBytes = 4;
    __device__ static uint4 run(const float *x)
    {
        return make_uint4(__float_as_uint(x[0]), __float_as_uint(x[1]), __float_as_uint(x[2]), __float_as_uint(x[3]));
    }
};

constexpr uint32_t kRopeThreads = 256;
constexpr uint32_t kMaxTable = 2048;                    // angles a block keeps (16 KB)

// {cos, sin} of `rows` x half angles from row row0 on, row-major, and the powers they are made of.
template <typename PosOf>
__device__ __forceinline__ void rope_table(float2 *table, float *freqs, uint32_t rows, uint32_t half, float theta_scale,
                                           float freq_scale, PosOf pos_of)
{
    for (uint32_t i = threadIdx.x; i < half; i += kRopeThreads) {
        float f = 1.0f;
        for (uint32_t k = 0; k < i; ++k) f = __fmul_rn(f, theta_scale);
        freqs[i] = f;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < rows * half; i += kRopeThreads) {
        const uint32_t r = i / half, w = i - r * half;
        float s, c;
        sincosf(__fmul_rn(__fmul_rn(float(pos_of(r)), freq_scale), freqs[w]), &s, &c);
        table[i] = make_float2(c, s);
    }
    __syncthreads();
}
// (x_i, x_{i+half}) <- (a c - b s, a s + b c), products rounded separately as on the CPU
__device__ __forceinline__ float rope_lo(float a, float b, float2 cs) { return __fsub_rn(__fmul_rn(a, cs.x), __fmul_rn(b, cs.y)); }
__device__ __forceinline__ float rope_hi(float a, float b, float2 cs) { return __fadd_rn(__fmul_rn(a, cs.y), __fmul_rn(b, cs.x)); }

// K rotated and stored, V stored as it is.  A block takes rows_per_block rows; a thread's unit is one
// 16-byte cache store of V, or the two stores of K whose elements pair up (or one of dims that pass through).
template <int DT>
__global__ void __launch_bounds__(kRopeThreads) rope_append_kernel(const RopeAppendParams p, uint32_t rows_per_block)
{
    constexpr int E = Pack<DT>::kElems;
    extern __shared__ float2 table[];
    const uint32_t half = p.n_dims / 2;
    float *const freqs = reinterpret_cast<float *>(table + rows_per_block * half);
    const uint32_t row0 = blockIdx.x * rows_per_block, rows = min(rows_per_block, p.n_rows - row0);
    if (p.positions) pdl_wait();                        // the positions may be the predecessor's
    rope_table(table, freqs, rows, half, p.theta_scale, p.freq_scale,
               [&](uint32_t r) { return p.positions ? p.positions[row0 + r] : p.base_pos + row0 + r; });
    if (!p.positions) pdl_wait();
    const uint32_t pairs = half / E, tail = (p.head_dim - p.n_dims) / E, k_units = p.n_kv_heads * (pairs + tail);
    const uint32_t v_units = p.row_elems / E, units = k_units + v_units;
    const uint64_t row_bytes = uint64_t(p.row_elems) * Pack<DT>::kBytes;
    for (uint32_t i = threadIdx.x; i < rows * units; i += kRopeThreads) {
        const uint32_t r = i / units, u = i - r * units, row = row0 + r;
        uint32_t slot, pos;
        if (p.positions) { slot = p.slot_ids ? p.slot_ids[row] : row; pos = p.positions[row]; }
        else { slot = p.slot; pos = p.base_pos + row; }
        if (slot >= p.n_slots || pos >= p.max_seq) { atomicOr(p.status, 2u); continue; }
        const uint64_t dst = uint64_t(slot) * p.slot_stride_bytes + uint64_t(pos) * row_bytes;
        float x[E];
        auto load = [&](const float *src) {
#pragma unroll
            for (int j = 0; j < E; j += 4) {
                const float4 f = *reinterpret_cast<const float4 *>(src + j);
                x[j] = f.x; x[j + 1] = f.y; x[j + 2] = f.z; x[j + 3] = f.w;
            }
        };
        auto store = [&](const float *y, uint8_t *base, uint32_t e0, bool rot) {
            if (rot && p.k_rot) {
                float *o = p.k_rot + uint64_t(row) * p.row_elems + e0;
#pragma unroll
                for (int j = 0; j < E; j += 4) *reinterpret_cast<float4 *>(o + j) = make_float4(y[j], y[j + 1], y[j + 2], y[j + 3]);
            }
            *reinterpret_cast<uint4 *>(base + dst + uint64_t(e0) * Pack<DT>::kBytes) = Pack<DT>::run(y);
        };
        if (u >= k_units) {
            const uint32_t e0 = (u - k_units) * E;
            load(p.v + uint64_t(row) * p.row_elems + e0);
            store(x, p.v_dst, e0, false);
            continue;
        }
        const uint32_t head = u / (pairs + tail), c = u - head * (pairs + tail);
        const uint32_t d0 = c < pairs ? c * E : p.n_dims + (c - pairs) * E;
        const float *const src = p.k + uint64_t(row) * p.row_elems + uint64_t(head) * p.head_dim;
        load(src + d0);
        if (c < pairs) {
            float hi[E];
            const float2 *const cs = table + r * half + d0;
#pragma unroll
            for (int j = 0; j < E; j += 4) {
                const float4 f = *reinterpret_cast<const float4 *>(src + half + d0 + j);
                const float b[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float a = x[j + q];
                    x[j + q] = rope_lo(a, b[q], cs[j + q]);
                    hi[j + q] = rope_hi(a, b[q], cs[j + q]);
                }
            }
            store(hi, p.k_dst, head * p.head_dim + half + d0, true);
        }
        store(x, p.k_dst, head * p.head_dim + d0, true);
    }
}

// Q rows (or any [rows][heads][head_dim] f32): four pairs a thread, x and out 16-byte aligned, in place
// or not.  grid.y cuts the heads of a few rows over several blocks.
__global__ void __launch_bounds__(kRopeThreads)
rope_rows_kernel(const float *x, float *out, uint32_t n_rows, uint32_t n_heads, uint32_t head_dim, uint32_t heads_per_block,
                 const uint32_t *positions, uint32_t base_pos, uint32_t n_dims, float theta_scale,
                 float freq_scale, uint32_t rows_per_block)
{
    extern __shared__ float2 table[];
    const uint32_t half = n_dims / 2;
    float *const freqs = reinterpret_cast<float *>(table + rows_per_block * half);
    const uint32_t row0 = blockIdx.x * rows_per_block, rows = min(rows_per_block, n_rows - row0);
    const uint32_t head0 = blockIdx.y * heads_per_block, heads = min(heads_per_block, n_heads - head0);
    if (positions) pdl_wait();
    rope_table(table, freqs, rows, half, theta_scale, freq_scale,
               [&](uint32_t r) { return positions ? positions[row0 + r] : base_pos + row0 + r; });
    if (!positions) pdl_wait();
    const uint32_t quads = half / 4, tail = (head_dim - n_dims) / 4, per_head = quads + tail, units = heads * per_head;
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < rows * units; i += kRopeThreads) {
        const uint32_t r = i / units, u = i - r * units, h = u / per_head, c = u - h * per_head;
        const uint64_t at = (uint64_t(row0 + r) * n_heads + head0 + h) * head_dim;
        if (c >= quads) {
            const uint64_t d = at + n_dims + 4 * (c - quads);
            *reinterpret_cast<float4 *>(out + d) = *reinterpret_cast<const float4 *>(x + d);
            continue;
        }
        const float4 a = *reinterpret_cast<const float4 *>(x + at + 4 * c), b = *reinterpret_cast<const float4 *>(x + at + half + 4 * c);
        const float2 *const t = table + r * half + 4 * c;
        const float2 cs[4] = {t[0], t[1], t[2], t[3]};
        *reinterpret_cast<float4 *>(out + at + 4 * c) = make_float4(rope_lo(a.x, b.x, cs[0]), rope_lo(a.y, b.y, cs[1]), rope_lo(a.z, b.z, cs[2]), rope_lo(a.w, b.w, cs[3]));
        *reinterpret_cast<float4 *>(out + at + half + 4 * c) = make_float4(rope_hi(a.x, b.x, cs[0]), rope_hi(a.y, b.y, cs[1]), rope_hi(a.z, b.z, cs[2]), rope_hi(a.w, b.w, cs[3]));
    }
}

// The same for shapes or buffers that do not come in 16-byte pieces: one thread per pair.
__global__ void __launch_bounds__(256)
rope_neox_kernel(const float *x, float *out, uint64_t n_rows, uint32_t n_heads, uint32_t head_dim,
                 const uint32_t *positions, uint32_t base_pos, uint32_t n_dims, float theta_scale, float freq_scale)
{
    const uint32_t half = n_dims / 2, tail = head_dim - n_dims;
    const uint32_t per_head = half + tail;              // work items per head: pairs, then pass-through dims
    const uint64_t total = n_rows * n_heads * per_head;
    pdl_wait();
    for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < total; i += uint64_t(gridDim.x) * blockDim.x) {
        const uint32_t w = uint32_t(i % per_head);
        const uint64_t rh = i / per_head, row = rh / n_heads;
        const float *src = x + rh * head_dim;
        float *dst = out + rh * head_dim;
        if (w >= half) { dst[n_dims + (w - half)] = src[n_dims + (w - half)]; continue; }
        const uint32_t pos = positions ? positions[row] : base_pos + uint32_t(row);
        float freq = 1.0f;
        for (uint32_t k = 0; k < w; ++k) freq = __fmul_rn(freq, theta_scale);
        float s, c;
        sincosf(__fmul_rn(__fmul_rn(float(pos), freq_scale), freq), &s, &c);
        const float a = src[w], b = src[w + half];
        dst[w] = rope_lo(a, b, make_float2(c, s));
        dst[w + half] = rope_hi(a, b, make_float2(c, s));
    }
}

// Rows a block takes: enough blocks for four on every SM, at most eight rows, a table that fits.
static uint32_t rows_per_block(const vfkv_ctx *ctx, uint64_t n_rows, uint32_t half)
{
    uint64_t r = n_rows / (uint64_t(ctx->sm_count) * 4);
    if (r > 8) r = 8;
    if (r > kMaxTable / half) r = kMaxTable / half;
    return r < 1 ? 1u : uint32_t(r);
}

static float theta_scale_of(const vfkv_rope_params &r)
{
    return powf(1.0f / r.freq_base, 2.0f / float(r.n_dims));     // setup.rs:786-788 in f32
}

template <int DT>
static int32_t launch_rope_append_t(vfkv_ctx *ctx, const RopeAppendParams &p, cudaStream_t st)
{
    const uint32_t half = p.n_dims / 2, rpb = rows_per_block(ctx, p.n_rows, half);
    const size_t smem = rpb * half * sizeof(float2) + half * sizeof(float);
    ProfScope ps(ctx, VFKV_PROF_KV_STORE, st);
    const cudaError_t e = launch_dependent(ctx, rope_append_kernel<DT>, dim3((p.n_rows + rpb - 1) / rpb), dim3(kRopeThreads), smem, st, p, rpb);
    ctx->count_launch();
    ctx->set_written(p.k_dst, uint64_t(p.n_slots) * p.slot_stride_bytes);
    return check_cuda(ctx, e, "rope_append launch");
}

}  // namespace vfkv

using namespace vfkv;

namespace {

struct Guard {
    int prev = -1;
    explicit Guard(int dev) { cudaGetDevice(&prev); if (prev != dev) cudaSetDevice(dev); else prev = -1; }
    ~Guard() { if (prev >= 0) cudaSetDevice(prev); }
};

int32_t check_rope(vfkv_ctx *ctx, const vfkv_rope_params *r, uint32_t head_dim, const char *fn)
{
    if (!r) return set_error(ctx, VFKV_ERR_INVALID, std::string(fn) + ": null rope parameters");
    if (r->n_dims == 0 || r->n_dims % 2 != 0 || r->n_dims > head_dim)
        return set_error(ctx, VFKV_ERR_INVALID, std::string(fn) + ": n_dims must be even and at most head_dim");
    if (!(r->freq_base > 0.f) || !(r->freq_scale > 0.f))
        return set_error(ctx, VFKV_ERR_INVALID, std::string(fn) + ": freq_base and freq_scale must be positive");
    return VFKV_OK;
}

int32_t rope_append_common(vfkv_cache *cache, uint32_t layer, const float *d_k, const float *d_v, uint32_t n_rows,
                           uint32_t slot, uint32_t base_pos, const uint32_t *d_slot_ids, const uint32_t *d_positions,
                           const vfkv_rope_params *rope, float *d_k_rot, void *stream, const char *fn)
{
    if (!cache) return VFKV_ERR_INVALID;
    vfkv_ctx *ctx = cache->ctx;
    KvCache &kv = cache->kv;
    if (layer >= kv.config.n_layers) return set_error(ctx, VFKV_ERR_INVALID, std::string(fn) + ": layer out of range");
    if (!d_k || !d_v) return set_error(ctx, VFKV_ERR_INVALID, std::string(fn) + ": null K or V");
    if ((reinterpret_cast<uintptr_t>(d_k) | reinterpret_cast<uintptr_t>(d_v) | reinterpret_cast<uintptr_t>(d_k_rot)) % 16 != 0)
        return set_error(ctx, VFKV_ERR_INVALID, std::string(fn) + ": K, V and the rotated-K output must be 16-byte aligned");
    const uint32_t hd = kv.head_dim_for(layer), hkv = kv.kv_heads_for(layer);
    int32_t rc = check_rope(ctx, rope, hd, fn);
    if (rc) return rc;
    if (n_rows == 0) return VFKV_OK;
    const uint32_t dt = uint32_t(kv.kv_dtype);
    const uint32_t E = dt == VFKV_F8 ? 16 : dt == VFKV_F16 ? 8 : 4;
    const bool fusable = !kv.k_scales && (rope->n_dims / 2) % E == 0 && hd % E == 0 && rope->n_dims / 2 <= kMaxTable;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (!fusable) {
        // shapes the fused kernel does not tile (or a cache with scale planes): rotate into the
        // caller's buffer, then the ordinary append
        if (!d_k_rot) return set_error(ctx, VFKV_ERR_UNSUPPORTED, std::string(fn) + ": this shape needs the d_k_rot buffer");
        rc = vfkv_rope_neox(ctx, d_k, d_k_rot, n_rows, hkv, hd, d_positions, base_pos, rope, stream);
        if (rc) return rc;
        return d_positions ? vfkv_append_batch(cache, layer, d_k_rot, d_v, d_slot_ids, d_positions, n_rows, stream)
                           : vfkv_append(cache, layer, d_k_rot, d_v, n_rows, slot, base_pos, stream);
    }
    RopeAppendParams p{};
    p.k = d_k; p.v = d_v; p.k_rot = d_k_rot;
    const uint64_t off = kv.layer_offset_bytes(layer);
    p.k_dst = static_cast<uint8_t *>(kv.k_buffer) + off;
    p.v_dst = static_cast<uint8_t *>(kv.v_buffer) + off;
    p.slot_ids = d_slot_ids; p.positions = d_positions;
    p.slot_stride_bytes = kv.layer_size_bytes(layer);
    p.row_elems = hkv * hd; p.head_dim = hd; p.n_kv_heads = hkv;
    p.max_seq = kv.config.max_seq_len; p.n_slots = kv.config.n_slots;
    p.n_rows = n_rows; p.slot = slot; p.base_pos = base_pos;
    p.n_dims = rope->n_dims; p.theta_scale = theta_scale_of(*rope); p.freq_scale = rope->freq_scale;
    p.status = ctx->d_status;
    Guard g(ctx->device);
    switch (dt) {
    case VFKV_F8: return launch_rope_append_t<VFKV_F8>(ctx, p, st);
    case VFKV_F16: return launch_rope_append_t<VFKV_F16>(ctx, p, st);
    case VFKV_F32: return launch_rope_append_t<VFKV_F32>(ctx, p, st);
    }
    return set_error(ctx, VFKV_ERR_INVALID, "unknown dtype");
}

}  // namespace

extern "C" {

int32_t vfkv_rope_append(vfkv_cache *cache, uint32_t layer, const float *d_k, const float *d_v, uint32_t n_tokens,
                         uint32_t slot, uint32_t base_pos, const vfkv_rope_params *rope, float *d_k_rot, void *stream)
{
    if (!cache) return VFKV_ERR_INVALID;
    if (slot >= cache->kv.config.n_slots)
        return set_error(cache->ctx, VFKV_ERR_INVALID, "vfkv_rope_append: slot out of range");
    if (uint64_t(base_pos) + n_tokens > cache->kv.config.max_seq_len)
        return set_error(cache->ctx, VFKV_ERR_INVALID, "vfkv_rope_append: base_pos + n_tokens exceeds max_seq_len");
    return rope_append_common(cache, layer, d_k, d_v, n_tokens, slot, base_pos, nullptr, nullptr, rope, d_k_rot, stream,
                              "vfkv_rope_append");
}

int32_t vfkv_rope_append_batch(vfkv_cache *cache, uint32_t layer, const float *d_k, const float *d_v,
                               const uint32_t *d_slot_ids, const uint32_t *d_positions, uint32_t n_seqs,
                               const vfkv_rope_params *rope, float *d_k_rot, void *stream)
{
    if (!cache) return VFKV_ERR_INVALID;
    if (!d_positions) return set_error(cache->ctx, VFKV_ERR_INVALID, "vfkv_rope_append_batch: null positions");
    return rope_append_common(cache, layer, d_k, d_v, n_seqs, 0, 0, d_slot_ids, d_positions, rope, d_k_rot, stream,
                              "vfkv_rope_append_batch");
}

int32_t vfkv_rope_neox(vfkv_ctx *ctx, const float *d_x, float *d_out, uint32_t n_rows, uint32_t n_heads,
                       uint32_t head_dim, const uint32_t *d_positions, uint32_t base_pos, const vfkv_rope_params *rope,
                       void *stream)
{
    if (!ctx) return VFKV_ERR_INVALID;
    if (!d_x || !d_out) return set_error(ctx, VFKV_ERR_INVALID, "vfkv_rope_neox: null argument");
    if (head_dim == 0 || n_heads == 0) return set_error(ctx, VFKV_ERR_INVALID, "vfkv_rope_neox: empty shape");
    int32_t rc = check_rope(ctx, rope, head_dim, "vfkv_rope_neox");
    if (rc) return rc;
    if (n_rows == 0) return VFKV_OK;
    Guard g(ctx->device);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const uint32_t half = rope->n_dims / 2;
    cudaError_t e;
    if (half % 4 == 0 && head_dim % 4 == 0 && half <= kMaxTable &&
        (reinterpret_cast<uintptr_t>(d_x) | reinterpret_cast<uintptr_t>(d_out)) % 16 == 0) {
        const uint32_t rpb = rows_per_block(ctx, n_rows, half);
        const uint32_t hpb = n_rows >= uint32_t(ctx->sm_count) * 2 || n_heads < 8 ? n_heads : 8;
        const size_t smem = rpb * half * sizeof(float2) + half * sizeof(float);
        e = launch_dependent(ctx, rope_rows_kernel, dim3((n_rows + rpb - 1) / rpb, (n_heads + hpb - 1) / hpb), dim3(kRopeThreads),
                             smem, st, d_x, d_out, n_rows, n_heads, head_dim, hpb, d_positions, base_pos, rope->n_dims,
                             theta_scale_of(*rope), rope->freq_scale, rpb);
    } else {
        const uint64_t total = uint64_t(n_rows) * n_heads * (half + head_dim - rope->n_dims);
        uint64_t blocks = (total + 255) / 256;
        const uint64_t cap = uint64_t(ctx->sm_count) * 16;
        if (blocks > cap) blocks = cap;
        e = launch_dependent(ctx, rope_neox_kernel, dim3(unsigned(blocks)), dim3(256), 0, st, d_x, d_out, uint64_t(n_rows), n_heads,
                             head_dim, d_positions, base_pos, rope->n_dims, theta_scale_of(*rope), rope->freq_scale);
    }
    ctx->count_launch();
    return check_cuda(ctx, e, "rope_neox launch");
}

}  // extern "C"
