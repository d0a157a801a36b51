// Log-sum-exp merge of split-K partials and the attention dispatcher.
//
// Replaces vk_shaders/flash_attn_reduce.comp and the host half of
// Forward::run_flash_attn_split_reduce (src/backend/vulkan/forward/runs.rs:1463-1571).
#include "attn_params.cuh"

#include <algorithm>

namespace vfkv {

// flash_attn_reduce.comp:51-80: out = sum_i o_i e^(m_i - M) / sum_i l_i e^(m_i - M) with M the
// maximum of the partial maxima; the final multiply by 1/sum is skipped when
// the caller wants the unnormalised triple (sequence-dimension sharding).
// Partial i of row r: m and l at i*ml_part + r*ml_row, o at i*o_part + r*o_row (+ dim), all in floats.
// Output row of partial row r when a launch carries several layers (see SeqArgs); the identity otherwise.
struct LayerRows { uint32_t per_layer; uint16_t layer_ids[kMaxLaunchLayers]; };

__global__ void __launch_bounds__(128)
merge_kernel(const float *pm, const float *pl, const float *po,
             uint32_t n_parts, uint64_t ml_part, uint64_t ml_row, uint64_t o_part, uint64_t o_row, uint32_t head_dim,
             float *out, float *out_m, float *out_l, float *out_o, const LayerRows lr)
{
    const uint64_t row = blockIdx.x;
    uint64_t orow = row;
    if (lr.per_layer != 0u) {
        const uint32_t i = blockIdx.x / lr.per_layer;
        orow = uint64_t(lr.layer_ids[i]) * lr.per_layer + (blockIdx.x - i * lr.per_layer);
    }
    pdl_wait();
    if (n_parts == 0u) {                                // nothing to merge: an empty range
        const uint32_t d = blockIdx.y * 128 + threadIdx.x;
        if (d < head_dim) {
            if (out) out[orow * head_dim + d] = 0.f;
            if (out_o) out_o[orow * head_dim + d] = 0.f;
        }
        if (out_o && d == 0) { out_m[orow] = kMaskedScore; out_l[orow] = 0.f; }
        return;
    }
    __shared__ float s_red[4], s_sum[4], s_acc[4][128];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // The shader walks the partials with a running (max, sum, acc); the same result, up to
    // rounding, comes from taking the maximum first and then one weighted sum, which leaves
    // every load independent of the others.  The launch is a chain of L2 round trips and nothing
    // else: a warp takes four parts at a time (its first four are on their way behind the maximum), lane: dims
    // lane + 32 j of the block's 128, every load unconditional.  (One thread a dim walking all parts, with a
    // condition on the dim, serialised them: 64 parts of 16 rows of 512, 59 us.)
    constexpr int U = 4;
    float pv[U][4], pw[U];
    auto fetch = [&](uint32_t i0) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t i = min(i0 + u, n_parts - 1);
            pw[u] = pm[uint64_t(i) * ml_part + row * ml_row];
            const float *const o = po + uint64_t(i) * o_part + row * o_row;
#pragma unroll
            for (int j = 0; j < 4; ++j) pv[u][j] = o[min(blockIdx.y * 128 + lane + 32 * j, head_dim - 1)];
        }
    };
    fetch(warp * U);
    float gmax = kMaskedScore;
    float m_own[2] = {kMaskedScore, kMaskedScore}, l_own[2] = {0.f, 0.f};      // parts tid and tid + 128
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const uint32_t i = threadIdx.x + 128 * k;
        if (i < n_parts) {
            const uint64_t pi = uint64_t(i) * ml_part + row * ml_row;
            m_own[k] = pm[pi];
            l_own[k] = pl[pi];
        }
    }
    gmax = fmaxf(m_own[0], m_own[1]);
    for (uint32_t i = threadIdx.x + 256; i < n_parts; i += 128) gmax = fmaxf(gmax, pm[uint64_t(i) * ml_part + row * ml_row]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) gmax = fmaxf(gmax, __shfl_xor_sync(0xffffffffu, gmax, o));
    if (lane == 0) s_red[warp] = gmax;
    __syncthreads();
    gmax = fmaxf(fmaxf(s_red[0], s_red[1]), fmaxf(s_red[2], s_red[3]));
    float gsum = fmaf(l_own[0], __expf(m_own[0] - gmax), l_own[1] * __expf(m_own[1] - gmax));
    for (uint32_t i = threadIdx.x + 256; i < n_parts; i += 128) {
        const uint64_t pi = uint64_t(i) * ml_part + row * ml_row;
        gsum = fmaf(pl[pi], __expf(pm[pi] - gmax), gsum);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) gsum += __shfl_xor_sync(0xffffffffu, gsum, o);
    if (lane == 0) s_sum[warp] = gsum;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    for (uint32_t i0 = warp * U; i0 < n_parts; i0 += 4 * U) {
        if (i0 != warp * U) fetch(i0);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (i0 + u < n_parts) {
                const float kn = __expf(pw[u] - gmax);
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[j] = fmaf(pv[u][j], kn, acc[j]);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) s_acc[warp][lane + 32 * j] = acc[j];
    __syncthreads();
    gsum = (s_sum[0] + s_sum[1]) + (s_sum[2] + s_sum[3]);
    const float inv = gsum > 0.f ? 1.0f / gsum : 0.f;   // an empty range yields zeros, not NaN
    const uint32_t t = threadIdx.x, d = blockIdx.y * 128 + t;
    const float o = (s_acc[0][t] + s_acc[1][t]) + (s_acc[2][t] + s_acc[3][t]);
    if (d < head_dim) {
        if (out) out[orow * head_dim + d] = o * inv;
        if (out_o) out_o[orow * head_dim + d] = o;
    }
    if (out_o && d == 0) { out_m[orow] = gmax; out_l[orow] = gsum; }
}

int32_t launch_merge_ws(vfkv_ctx *ctx, vfkv_workspace *ws, const AttnArgs &a, uint32_t n_splits,
                        cudaStream_t st)
{
    const uint32_t rows = a.seq.units() * a.n_q_heads;
    LayerRows lr{};
    if (a.seq.layer_ids) {
        lr.per_layer = a.seq.n_seqs * a.n_q_heads;
        for (uint32_t i = 0; i < a.seq.n_layers; ++i) lr.layer_ids[i] = a.seq.layer_ids[i];
    }
    ProfScope ps(ctx, VFKV_PROF_FA_REDUCE, st);
    const uint64_t D = a.kv.head_dim;
    const cudaError_t e = launch_dependent(ctx, merge_kernel, dim3(rows, (a.kv.head_dim + 127) / 128), dim3(128), 0, st, ws->part_m, ws->part_l, ws->part_o,
                                           n_splits, uint64_t(1), uint64_t(n_splits), D, n_splits * D, a.kv.head_dim, a.out,
                                           a.out_m, a.out_l, a.out_o, lr);
    ctx->count_launch(a.seq.n_layers);
    return check_cuda(ctx, e, "merge launch");
}

int32_t launch_merge_partials(vfkv_ctx *ctx, const float *m, const float *l, const float *o,
                              uint32_t n_parts, uint32_t n_rows, uint32_t head_dim, float *out,
                              cudaStream_t st)
{
    if (n_rows == 0) return VFKV_OK;
    ProfScope ps(ctx, VFKV_PROF_FA_REDUCE, st);
    merge_kernel<<<dim3(n_rows, (head_dim + 127) / 128), 128, 0, st>>>(m, l, o, n_parts, n_rows, 1, uint64_t(n_rows) * head_dim, head_dim,
                                        head_dim, out, nullptr, nullptr, nullptr, LayerRows{});
    ctx->count_launch();
    return check_cuda(ctx, cudaGetLastError(), "merge_partials launch");
}

// One block of n_rows*(head_dim+2) floats per part: m[n_rows], l[n_rows], o[n_rows][head_dim] --
// the layout an all-gather of per-GPU partials produces.
int32_t launch_merge_partials_packed(vfkv_ctx *ctx, const float *packed, uint32_t n_parts, uint32_t n_rows,
                                     uint32_t head_dim, float *out, cudaStream_t st)
{
    if (n_rows == 0) return VFKV_OK;
    const uint64_t block = uint64_t(n_rows) * (head_dim + 2);
    ProfScope ps(ctx, VFKV_PROF_FA_REDUCE, st);
    merge_kernel<<<dim3(n_rows, (head_dim + 127) / 128), 128, 0, st>>>(packed, packed + n_rows, packed + 2 * uint64_t(n_rows), n_parts, block, 1,
                                        block, head_dim, head_dim, out, nullptr, nullptr, nullptr, LayerRows{});
    ctx->count_launch();
    return check_cuda(ctx, cudaGetLastError(), "merge_partials_packed launch");
}

// The most tiles of a sequence that the tensor-core kernel gives to a warp by itself (attn_mma.cu, launch_c), by the CTAs of
// the launch.  0 up to as many as are resident with 4 warps.  Up to twice that, a warp with more than eight tiles (ten of F16)
// pays only if all sequences are equally long, and the longest, which the caller names, says nothing of the others; from two and a
// half times on sixteen pay either way.  Times of four warps / of one, all as long and spread from a 32nd to that, of 128 dims:
//   520 CTAs, FP8   8 tiles 1.14 0.97   10 1.15 0.87   16 0.97 0.72        F16   10 1.23 0.99   12 1.11 0.91   16 1.03 0.81
//   896             12 1.16 1.06   14 1.23 0.98   16 1.12 0.93             F16   16 1.13 1.09
//   1184            16 1.09 1.06                                           F16   16 1.11 1.22
// 64 dims, four CTAs an SM: 720 8 0.97 0.98, 10 0.95 0.95; 1184 12 1.04 1.04, 16 0.97 0.94.  256 dims, two CTAs an SM: 520, FP8, 8
// 1.12 0.98, 10 1.22 0.92; 600 12 1.19 0.94; 720 12 1.18 1.02, 16 1.15 0.99; F16, 600 16 1.26 1.06; at three an SM, where it begins, 8 1.11 0.96.
uint32_t one_warp_tiles(const vfkv_ctx *ctx, uint32_t dtype, uint32_t head_dim, uint64_t ctas)
{
    const uint64_t n_sm = uint64_t(ctx->sm_count), resident = n_sm * (head_dim == 64 ? 4u : head_dim == 128 ? 3u : 2u);
    const bool f16 = dtype == VFKV_F16;
    if (ctas <= (head_dim == 64 ? resident : 3 * n_sm)) return 0u;
    if (2 * ctas > 5 * resident) return 16u;
    if (ctas > 2 * resident) return f16 && head_dim != 64 ? 16u : 12u;
    return f16 && head_dim == 128 ? 10u : 8u;
}

// Expected time (us) of a tensor-core decode launch with n splits of sequences of len positions, base (sequence, kv-head)
// pairs: a wave of CTAs costs 8 us and its stream, splits cost their merge.  An SM streams 39 KB a us with one CTA of 8 warps, 27
// with two of 4 and 17 with one of those (HBM, shared, is in that); a CTA works through its positions in rounds of a tile for
// each warp.  The numbers are a fit to 280 grids of 9 to 295 pairs (23 to 130 000 positions, all dtypes and groups), each
// timed with 1 to 64 splits.
static double split_us(const vfkv_ctx *ctx, const AttnArgs &a, uint32_t len, uint64_t base, uint32_t n)
{
    const uint32_t es = a.kv.dtype == VFKV_F8 ? 1 : 2, tp = a.kv.dtype == VFKV_F8 ? 32 : 16, per = (len + n - 1) / n;
    const double row = 2.0 * a.kv.head_dim * es;
    const uint64_t ctas = base * n, n_sm = uint64_t(ctx->sm_count);
    auto wave = [&](uint32_t warps, double rate) {
        const uint32_t round = warps * tp;
        return 8.0 + double((per + round - 1) / round * round) * row / rate;
    };
    double us = n > 1 ? 4.0 + 0.11 * n : 0.0;
    if (a.kv.head_dim < 256 && ctas <= n_sm) return us + wave(8, 39400.0);
    const uint64_t full = ctas / (2 * n_sm), last = ctas % (2 * n_sm);
    us += double(full) * wave(4, 27000.0 / 2);
    if (last) us += wave(4, last <= n_sm ? 17000.0 : 27000.0 / 2);
    return us;
}

// The same where one sequence is that long and the others are short: its CTAs, few to an SM, stream 80 KB a us each with 8 warps
// and 42 with 4, and the others' cost 2.4 us for every three an SM, whatever they find to do.
static double split_us_alone(const vfkv_ctx *ctx, const AttnArgs &a, uint32_t len, uint64_t base, uint32_t n)
{
    const double row = 2.0 * a.kv.head_dim * (a.kv.dtype == VFKV_F8 ? 1 : 2);
    const double rate = a.kv.head_dim < 256 && base * n <= uint64_t(ctx->sm_count) ? 80000.0 : 42000.0;
    return (n > 1 ? 4.0 + 0.11 * n : 0.0) + 8.0 + double((len + n - 1) / n) * row / rate +
           2.4 * double(base * n) / double(3 * uint64_t(ctx->sm_count));
}

// Split count when the caller passes 0.  The reference always cuts at 64
// positions (runs.rs:766-769); here the count only has to fill the GPU: aim
// for about two CTAs per SM, never cut below 256 positions per split (128 on the tensor cores
// with an F16 cache).
uint32_t choose_splits(const vfkv_ctx *ctx, const AttnArgs &a, uint32_t tile)
{
    uint32_t max_len = a.seq.max_len_hint ? a.seq.max_len_hint : a.kv.max_seq;
    if (!a.seq.seq_lens && !a.seq.positions) max_len = a.seq.seq_len_scalar - a.seq.kv_start_scalar;
    if (a.seq.window && max_len > a.seq.window) max_len = a.seq.window;
    // One split per (sequence, kv-head) once that alone gives every SM two CTAs: the stream is
    // HBM-bound, so a ragged last wave costs little, while every extra split costs a partial
    // write, a ticket and a merge.  Smaller grids are cut until about two CTAs per SM exist, but
    // never below 256 positions per split.
    const uint32_t parts = tile >= 128 ? attn_mma_parts(a.kv.dtype, a.n_q_heads / a.kv.n_kv_heads) : 1u;
    const uint64_t base = uint64_t(a.seq.units()) * a.kv.n_kv_heads * parts;
    const uint64_t slots = uint64_t(ctx->sm_count) * 2;
    // (an 8-warp CTA of the tensor-core kernel takes 8 tiles at a time: 256 positions of an FP8
    // cache, 128 of an F16 cache, where 16 splits of 128 measured 6.2 us against 6.6 us with 8 of 256
    // on 32 q / 8 kv / 128 at 2048 positions)
    const uint32_t min_chunk = (tile >= 128 && a.kv.dtype == VFKV_F16) ? 128 : tile < 256 ? 256 : tile;
    uint64_t cap = (uint64_t(max_len) + min_chunk - 1) / min_chunk;
    if (cap < 1) cap = 1;
    if (cap > 64) cap = 64;
    uint64_t want = base ? (slots + base - 1) / base : 1;
    // The CTA that merges reads every split's partial: beyond 16 splits that tail costs more than
    // the extra CTAs save (one sequence of 16384 positions, 64 q-heads: 15.9 us with 16 splits,
    // 19.5 us with 37), unless the length rule below asks for more.
    // (The wide-row kernel -- tile 64 -- leaves the merge to a launch with a CTA for each row.)
    if (want > 16 && tile != 64) want = 16;
    // Fewer than eight groups (one long sequence whose kv-heads are spread over several GPUs): the
    // merge is then shared by up to sixteen CTAs of the group, each combining its outputs with a
    // team of lanes, and one CTA per SM pays: 148 / groups splits.
    const bool few_groups = base > 0 && base * 32 <= uint64_t(ctx->sm_count) && tile >= 128;
    if (few_groups) {
        want = uint64_t(ctx->sm_count) / base;
        if (want > 255) want = 255;
        cap = (uint64_t(max_len) + min_chunk - 1) / min_chunk;
        if (cap < 1) cap = 1;
        if (want > cap) want = cap;
        // a CTA of 8 warps takes 256 positions per round of tiles: the fewest splits that need no
        // more rounds than that count does (131 072 positions on one kv-head: 128 splits of 4
        // rounds, 14.1 us, where 148 ragged ones took 15.6 us)
        const uint64_t rounds = ((uint64_t(max_len) + want - 1) / want + 255) / 256;
        const uint64_t fewest = (uint64_t(max_len) + rounds * 256 - 1) / (rounds * 256);
        if (fewest >= 1 && fewest < want) want = fewest;
    }
    // A CTA keeps at most its own ring of stages in flight, which bounds one CTA's stream to a few
    // tens of GB/s: in a ragged batch a sequence much longer than the rest would finish last on
    // its own.  No CTA gets more than 8192 positions, 4096 once contexts beyond 8192 are possible
    // (measured: 64 sequences of 512..16384 tokens 5.0 / 5.5 / 6.1 TB/s with 1 / 2 / 4 splits;
    // 64 x 8192 uniform 6.3 / 6.0 / 5.9 TB/s).
    // The rule is for batches that fill the GPU by themselves; a single long sequence is better off
    // with its 16 splits on 8-warp CTAs, one per SM (131 072 positions, 8 kv-heads: 46.3 us with
    // 16 splits of 8 warps, 51.1 us with 32 splits of 4 warps).
    const uint64_t per_cta = max_len > 8192 ? 4096 : 8192;
    const uint64_t by_len = (uint64_t(max_len) + per_cta - 1) / per_cta;
    if (want < by_len && base >= slots) want = by_len;
    if (want > cap) want = cap;
    if (want < 1) want = 1;
    // A stream-bound grid that spills a few CTAs into another wave pays for a whole wave: 64
    // (sequence, kv-head) pairs x 5 splits = 320 CTAs on 296 slots took 571 us where 9 splits (576
    // CTAs, two full waves) took 354 us and 4 splits (one wave, 86 % full) 379 us (F16, head_dim
    // 256, 8 x 32768 positions).  So when the count above overshoots the slots, take the nearby
    // count that fills its waves best, with a small price per split for the merge.
    if (base * want > slots && base < slots) {
        double best = -1.0;
        uint64_t pick = want;
        const uint64_t hi = cap < 4 * want ? cap : 4 * want;
        for (uint64_t n = want > 1 ? want - 1 : 1; n <= hi; ++n) {
            const uint64_t ctas = base * n, waves = (ctas + slots - 1) / slots;
            const double score = double(ctas) / double(waves * slots) - 0.008 * double(n);
            if (score > best) { best = score; pick = n; }
        }
        want = pick;
    }
    // Between nine pairs (fewer are a layer at a time, whose calls the host bounds) and two CTAs an SM the count of the rules
    // above gives way to the one that the model of the launch finds, if it promises a tenth or more (128 pairs of 3000 28.0 -> 18.4;
    // scaled, 256 pairs of 2001 to 4099 57 -> 49; F16, 192 pairs of at most 319, sixteen q-heads each 24 -> 11; over the 280 grids a
    // tenth on average, one of them 6 % slower, one 2).
    // Not for 64-dim rows, of which four CTAs share an SM, nor for more than 700 MB, where only HBM and every SM count (64 pairs of
    // 41 443, F16: 9 splits 208 us, 2 216; at 820 to 980 MB 0.95 to 1.05 of the time with the model's count, one case 0.90) and the
    // clock that the GPU keeps up decides (64 q / 8 kv heads over FP8, 8 layers x 131 072 positions: 9 splits 363 to 383 us, 2 329
    // for the first milliseconds, 399 where the power limit then holds).  At 300 to 660 MB it gains 2 to 16 %.
    const bool hbm_bound = double(max_len) * double(base) * 2.0 * a.kv.head_dim * (a.kv.dtype == VFKV_F8 ? 1 : 2) > 7e8;
    // The model knows of one length, the longest.  In a batch whose other sequences are short, fewer splits leave the longest to
    // a few CTAs while the other SMs stand idle (4 layers x 4 sequences, FP8, one of 16 384 and three of 600: 1 split 70 us, 9 42),
    // so what it promises if all are as long has to be 2.4 times what that would cost.  53 grids of 2 to 32 sequences, each with
    // all as long / down to half of it / down to a 32nd / half of them a 16th / all but one, in times of the rules' counts:
    // always the model's 1.14 / 1.10 / 1.05 / 1.06 / 0.88 as fast (at worst 0.99 / 0.92 / 0.76 / 0.80 / 0.38), so
    // 1.11 / 1.09 / 1.07 / 1.07 / 1.01 (1.00 / 0.97 / 0.86 / 0.83 / 0.70).
    if (tile >= 128 && base > 8 && base < slots && a.kv.head_dim != 64 && !hbm_bound) {
        const uint32_t rules = uint32_t(want);
        const double rules_us = split_us(ctx, a, max_len, base, rules), rules_alone = split_us_alone(ctx, a, max_len, base, rules);
        double best = 0.9 * rules_us;
        for (uint32_t n = 1; n == 1 || (n <= 64 && base * n <= 3 * uint64_t(ctx->sm_count) && uint64_t(n) * 128 <= max_len); ++n) {
            const double us = split_us(ctx, a, max_len, base, n);
            if (a.seq.n_seqs > 1u && n < rules && rules_us - us < 2.4 * (split_us_alone(ctx, a, max_len, base, n) - rules_alone)) continue;
            if (us < best) { best = us; want = n; }
        }
    }
    return uint32_t(want);
}

int32_t launch_attention(vfkv_ctx *ctx, vfkv_workspace *ws, const AttnArgs &a, cudaStream_t st)
{
    if (a.seq.n_seqs == 0) return VFKV_OK;
    if (a.kv.n_kv_heads == 0 || a.n_q_heads == 0 || a.n_q_heads % a.kv.n_kv_heads != 0)
        return set_error(ctx, VFKV_ERR_INVALID, "n_q_heads must be a non-zero multiple of n_kv_heads");
    const bool mma_ok = attn_mma_supported(a);
    if (ctx->attn_impl == 2 && !mma_ok)
        return set_error(ctx, VFKV_ERR_UNSUPPORTED, "shape outside the tensor-core attention kernel");
    const bool use_mma = mma_ok && ctx->attn_impl != 1, use_wide = !mma_ok && ctx->attn_impl != 1 && attn_wide_supported(a);

    uint32_t n_splits = a.n_splits ? a.n_splits : choose_splits(ctx, a, use_mma ? 128 : use_wide ? 64 : 32);
    if (n_splits > 1) {
        if (!ws) return set_error(ctx, VFKV_ERR_INVALID, "a workspace is required when n_splits > 1");
        if (n_splits > ws->max_splits) n_splits = ws->max_splits;
        if (a.seq.n_seqs > ws->max_seqs || a.n_q_heads > ws->n_q_heads || a.kv.head_dim > ws->head_dim)
            return set_error(ctx, VFKV_ERR_INVALID, "workspace too small for this call");
        // the workspace is sized for max_splits of each sequence of one layer; a launch of several layers shares it out
        if (a.seq.n_layers > 1) {
            const uint32_t parts = use_mma ? attn_mma_parts(a.kv.dtype, a.n_q_heads / a.kv.n_kv_heads) : 1u;
            const uint64_t groups = uint64_t(a.seq.units()) * a.kv.n_kv_heads * parts, g = a.n_q_heads / (a.kv.n_kv_heads * parts);
            const uint64_t most = use_mma ? (groups <= ws->n_counters ? ws->tag_words / (groups * (g * (a.kv.head_dim + 2) + 2)) : 1)
                                          : uint64_t(ws->max_seqs) * ws->max_splits / a.seq.units();
            if (n_splits > most) n_splits = most > 1 ? uint32_t(most) : 1u;
        }
    }
    int32_t rc = use_mma    ? launch_attn_mma(ctx, ws, a, n_splits, st)
                 : use_wide ? launch_attn_wide(ctx, ws, a, n_splits, st)
                            : launch_attn_generic(ctx, ws, a, n_splits, st);
    if (rc != VFKV_OK) return rc;
    // the tensor-core kernel merges its own partials (last CTA of each kv-head)
    if (n_splits > 1 && !use_mma) rc = launch_merge_ws(ctx, ws, a, n_splits, st);
    return rc;
}

}  // namespace vfkv
