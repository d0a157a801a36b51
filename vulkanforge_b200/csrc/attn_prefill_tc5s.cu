// Chunked-prefill causal attention on tcgen05 with one Q tile of 128 rows a CTA: the shapes that the
// two-tile kernel of attn_prefill_tc5.cu does not hold (head_dim 64 and 256, Q as two half-precision
// terms, FP8 rows with a scale per position and head) and chunks with few rows.
//
// CTA = 128 rows (128 / g consecutive queries x the g q-heads of a kv-head) x K/V tiles of 64 positions.
//   warps 0-3   softmax: thread = row; scores out of tensor memory, P back over them
//   warp  4     one thread issues every MMA: S(t + 1) = Q K^T as soon as its K is there, O += P V(t) as soon
//               as its P is, whichever comes first (two S buffers, so the products of one tile run under the
//               softmax of another)
//   warps 5-10  K and V rows into a ring of stages each: FP8 fetched, widened and placed by three warps
//               each, one tile ahead in registers; F16 copied by TMA
// 64 positions a tile, because Q of 256 dims in two terms takes 128 KB and leaves room for three stages (two
// of K, whose products come a tile earlier, and one of V).
// A row's exponents refer to a maximum that is moved, and O rescaled, only when the true one has outgrown
// it by a few binary orders.  The largest p is then any number up to 2^8 and not 1, so a row's sum is taken of the
// p as they go into the product, rounded to half precision: a row that one position dominates is that position's V
// whatever its p was rounded to (with the sum of the unrounded p: off by up to 2^-12; 32.3 -> 33.0 us for 333 queries at
// 1000 positions, F16).
//
// SPLITQ: Q = high + low half-precision term, scaled per row by a power of two (two products for S).
// SC: the scales of K multiply the scores, those of V multiply P, in f32; P is then also fed as two terms,
// relative to the largest power of two among the V scales so far (all of it exact but the terms' own
// 2^-22), which makes the result as accurate as f32 tiles on the CUDA cores.
//
// The tiles of a row block are cut over n_split CTAs when the blocks leave SMs idle; the pieces go to
// scratch and prefill_pieces_kernel puts them together (flash_attn_reduce.comp:51-80, maximum first).
// Every wait is bounded; one that runs out sets status bit 0 and the CTA leaves.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>

#include "fp8_codec.cuh"
#include "prefill_params.cuh"
#include "softcap.cuh"
#include "tcgen05.cuh"

namespace vfkv {
namespace {

constexpr float kLog2e = 1.4426950408889634f;
constexpr int BM = 128, BN = 64;
constexpr uint32_t kThreads = 352;
constexpr uint32_t SLAB_Q = 128 * 128, SLAB_KV = 64 * 128;      // [rows][64 halves], 128-byte swizzle
constexpr uint32_t kSmall = 3072;                               // barriers, row multipliers, tile scales
constexpr float kPUnit = 1024.0f;                               // SC: P terms are fed as p * v_scale / reference * 2^10

struct OneTileParams {
    PrefillParams a;
    uint32_t n_split, n_rb;
    float *scratch;                    // pieces {O [128][D], reference maxima [128], sums [128]} of n_split > 1
    uint32_t *status;
};

template <int D, bool SPLITQ> struct OneTile {
    static constexpr uint32_t QT = BM * D * 2, Q = QT * (SPLITQ ? 2 : 1), STAGE = BN * D * 2;
    static constexpr uint32_t ROOM = 227 * 1024 - kSmall - Q, NST = ROOM / STAGE < 8 ? ROOM / STAGE : 8;
    static constexpr uint32_t NK = (NST + 1) / 2, NV = NST / 2;  // stages of K, stages of V behind them
    static constexpr uint32_t SMEM = Q + NST * STAGE + kSmall;
    // Columns of tensor memory: S of even and odd tiles, then O.  With 32 products a tile (256 dims, Q in two
    // terms) those of S go to two accumulators in turn, which the softmax adds: MMAs into one wait for each
    // other (1.85 -> 1.73 us a tile; with 16 products the addition costs as much as it saves).
    static constexpr bool ACC2 = D > 128 && SPLITQ;
    static constexpr uint32_t S_COLS = ACC2 ? 128 : 64, O_COL = 2 * S_COLS, TMEM = O_COL + D > 256 ? 512 : 256;
    static constexpr uint64_t PIECE = uint64_t(BM) * (D + 2);
};

// Row block rb (0 = the latest queries): its first row, the first position of its tiles, their number.
__host__ __device__ __forceinline__ void block_extent(const PrefillParams &p, uint32_t n_rb, uint32_t rb, uint32_t *row0,
                                                      uint32_t *c_lo, uint32_t *n_tiles)
{
    const uint32_t r0 = (n_rb - 1u - rb) * uint32_t(BM);
    uint32_t qb = (r0 + uint32_t(BM) - 1u) / p.group, lo, hi, x;
    if (qb >= p.m) qb = p.m - 1u;
    query_range(p, r0 / p.group, &lo, &x);
    query_range(p, qb, &x, &hi);
    lo = lo / uint32_t(BN) * uint32_t(BN);
    *row0 = r0; *c_lo = lo;
    *n_tiles = hi > lo ? (hi - lo + uint32_t(BN) - 1u) / uint32_t(BN) : 0u;
}

// byte offset of 16-byte chunk c of row r in a tile of slabs of `slab` bytes
__device__ __forceinline__ uint32_t chunk_off(uint32_t r, uint32_t c, uint32_t slab)
{
    return (c >> 3) * slab + r * 128u + (((c & 7u) ^ (r & 7u)) << 4);
}

// One row by one warp over positions [lo, hi), each read only if the row sees it; to dst as the rows of the kernel below,
// final or (m != null) as a piece.  For rows that came out of the products as infinities or NaN: 0 x V of a position that
// a row does not see is not 0 when that V is not finite, and the tiles multiply all rows with all positions.
template <int DT, int D>
__device__ __noinline__ void row_alone(const PrefillParams *params, uint32_t r, uint32_t kvh, uint32_t lo, uint32_t hi, float *dst, float *m_out, float *l_out)
{
    const PrefillParams &p = *params;
    constexpr int N = D / 32;
    const uint32_t lane = threadIdx.x & 31u, g = p.group;
    const float *const q = p.q + (uint64_t(r / g) * p.n_q_heads + kvh * g + r % g) * D + lane;
    auto element = [&](const uint8_t *row, int j) {
        if constexpr (DT == VFKV_F16) return __half2float(reinterpret_cast<const __half *>(row)[lane + 32 * j]);
        else return e4m3x2_to_float2(row[lane + 32 * j]).x;
    };
    float m = kMaskedScore, l = 0.f, o[N];
#pragma unroll
    for (int j = 0; j < N; ++j) o[j] = 0.f;
    for (uint32_t pos = lo; pos < hi; ++pos) {
        const uint64_t at = uint64_t(pos) * p.row_bytes + uint64_t(kvh) * D * (DT == VFKV_F16 ? 2 : 1);
        float s = 0.f;
#pragma unroll
        for (int j = 0; j < N; ++j) s = fmaf(q[32 * j], element(p.k + at, j), s);
#pragma unroll
        for (int x = 16; x > 0; x >>= 1) s += __shfl_xor_sync(0xffffffffu, s, x);
        if (p.k_scales) s *= p.k_scales[uint64_t(pos) * p.n_kv_heads + kvh];
        s *= p.scale;
        if (p.softcap > 0.f) s = softcap_any(s, p.softcap, 1.0f / p.softcap);
        const float mn = fmaxf(m, s), corr = __expf(m - mn), e = __expf(s - mn);
        const float pv = p.v_scales ? e * p.v_scales[uint64_t(pos) * p.n_kv_heads + kvh] : e;
        l = l * corr + e;
#pragma unroll
        for (int j = 0; j < N; ++j) o[j] = o[j] * corr + pv * element(p.v + at, j);
        m = mn;
    }
    const float f = m_out ? 1.0f : l > 0.f ? 1.0f / l : 0.f;
#pragma unroll
    for (int j = 0; j < N; ++j) dst[lane + 32 * j] = o[j] * f;
    if (m_out && lane == 0u) { *m_out = m * kLog2e; *l_out = l; }
}

template <int DT, int D, bool SPLITQ, bool SC, bool CAP>
__global__ void __launch_bounds__(kThreads, 1)
prefill_one_tile_kernel(const __grid_constant__ OneTileParams op, const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v)
{
    using T = OneTile<D, SPLITQ>;
    static_assert(!SC || (SPLITQ && DT == VFKV_F8), "scales belong to FP8 caches and keep f32 accuracy");
    constexpr bool FP8 = DT == VFKV_F8;
    constexpr uint32_t NST = T::NST, NK = T::NK, NV = T::NV, ES = FP8 ? 1 : 2;
    const PrefillParams &p = op.a;
    extern __shared__ __align__(1024) uint8_t sm[];
    const uint32_t base = smem_addr(sm), q_sm = base, ring = base + T::Q, small = ring + NST * T::STAGE;
    uint8_t *const sm_small = sm + T::Q + NST * T::STAGE;
    float *const s_mult = reinterpret_cast<float *>(sm_small + 256);            // [128]
    float *const s_scales = s_mult + BM;                                       // SC: [warp][64 K scales, 64 V scales]
    volatile uint32_t *const s_ctl = reinterpret_cast<uint32_t *>(sm_small + 240);     // tensor memory address, abort flag
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t g = p.group, n_rows = p.m * g;
    // barriers: 0-1 S ready (commit)   2-3 P ready (128)   4-5 P V done (commit)   6.. stage full   6 + NST.. stage
    // free (commit); those that come in pairs belong to even and odd tiles, so that a wait on a phase parity is
    // never more than one phase away from the barrier's state
    auto bar = [&](uint32_t i) { return small + 8u * i; };
    const uint32_t full0 = 6u, free0 = 6u + NST;
    if ((base & 1023u) != 0u) {                // the swizzle counts on it; the array's alignment provides it
        if (tid == 0) atomicOr(op.status, 1u);
        return;
    }
    if (tid == 0) {
        mbar_init(bar(0), 1); mbar_init(bar(1), 1);
        mbar_init(bar(2), BM); mbar_init(bar(3), BM);
        mbar_init(bar(4), 1); mbar_init(bar(5), 1);
        for (uint32_t i = 0; i < NST; ++i) { mbar_init(bar(full0 + i), FP8 ? 96u : 1u); mbar_init(bar(free0 + i), 1); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_ctl[1] = 0u;
    }
    if (warp == 4) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(small + 240u), "n"(T::TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // blocks in the order (row block, kv-head, piece), on the one grid axis that holds any number of them
    const uint32_t line = blockIdx.x / op.n_split, split = blockIdx.x - line * op.n_split;
    const uint32_t rb = line / p.n_kv_heads, kvh = line - rb * p.n_kv_heads;
    uint32_t row0, c_lo, n_tiles;
    block_extent(p, op.n_rb, rb, &row0, &c_lo, &n_tiles);
    if (op.n_split > 1u) {
        const uint32_t first = uint32_t(uint64_t(n_tiles) * split / op.n_split), last = uint32_t(uint64_t(n_tiles) * (split + 1u) / op.n_split);
        c_lo += first * BN;
        n_tiles = last - first;
    }
    pdl_wait();

    // ---- K/V rows of FP8 caches: 96 threads for K, 96 for V, the first tile requested before Q is -----
    constexpr uint32_t PIECES = BN * D / 16;                    // 16-code pieces of a stage
    constexpr uint32_t NP = (PIECES + 95) / 96;
    const bool is_v = warp >= 8u;
    const uint32_t pt = tid - (is_v ? 256u : 160u);
    uint4 raw[FP8 ? NP : 1];
    auto fetch = [&](uint32_t it) {
        const uint8_t *src = (is_v ? p.v : p.k) + uint64_t(kvh) * D;
        const uint32_t t0 = c_lo + it * BN;
#pragma unroll
        for (uint32_t i = 0; i < NP; ++i) {
            const uint32_t idx = pt + 96u * i, pos = t0 + idx / (D / 16), c = idx % (D / 16);
            const bool in = idx < PIECES && pos < p.n_kv;
            raw[i] = in ? *reinterpret_cast<const uint4 *>(src + uint64_t(pos) * p.row_bytes + c * 16) : make_uint4(0u, 0u, 0u, 0u);
        }
    };
    if constexpr (FP8)
        if (warp >= 5u && n_tiles > 0u) fetch(0);

    // ---- Q -> shared memory, all warps: D / 8 neighbouring lanes hold a row --------------------------
    {
        constexpr uint32_t CHUNKS = BM * D / 8 / 32, QB = 4;
        const float q_mult = p.scale * (CAP ? 1.0f : kLog2e);
        for (uint32_t c0 = warp; c0 < CHUNKS; c0 += 11u * QB) {
            float4 a[QB], b[QB];
#pragma unroll
            for (uint32_t u = 0; u < QB; ++u) {
                const uint32_t idx = (c0 + 11u * u) * 32u + lane, r = row0 + idx / (D / 8), c = idx % (D / 8);
                const bool in = c0 + 11u * u < CHUNKS && r < n_rows;
                const float4 *src = reinterpret_cast<const float4 *>(p.q + (uint64_t(r / g) * p.n_q_heads + kvh * g + r % g) * D + 8 * c);
                a[u] = in ? *src : make_float4(0.f, 0.f, 0.f, 0.f);
                b[u] = in ? src[1] : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (uint32_t u = 0; u < QB; ++u) {
                if (c0 + 11u * u >= CHUNKS) break;
                const uint32_t idx = (c0 + 11u * u) * 32u + lane, r = idx / (D / 8), c = idx % (D / 8);
                float qs = q_mult;
                if constexpr (SPLITQ) {
                    // rows scaled by a power of two into [128, 256); the inverse goes to the scores
                    float top = fmaxf(fmaxf(fmaxf(fabsf(a[u].x), fabsf(a[u].y)), fmaxf(fabsf(a[u].z), fabsf(a[u].w))),
                                      fmaxf(fmaxf(fabsf(b[u].x), fabsf(b[u].y)), fmaxf(fabsf(b[u].z), fabsf(b[u].w))));
#pragma unroll
                    for (int o = 1; o < D / 8; o <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
                    int e = int((__float_as_uint(top) >> 23) & 0xFF) - 127;
                    e = top > 0.f ? max(-100, min(100, e)) : 7;
                    qs = __uint_as_float(uint32_t(7 - e + 127) << 23);
                    if (c == 0u) s_mult[r] = q_mult * __uint_as_float(uint32_t(e - 7 + 127) << 23);
                }
                const float x[8] = {a[u].x * qs, a[u].y * qs, a[u].z * qs, a[u].w * qs, b[u].x * qs, b[u].y * qs, b[u].z * qs, b[u].w * qs};
                uint32_t hi[4], lo[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    hi[j] = pack_half2(x[2 * j], x[2 * j + 1]);
                    const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&hi[j]));
                    lo[j] = pack_half2(x[2 * j] - f.x, x[2 * j + 1] - f.y);
                }
                uint8_t *const dst = sm + chunk_off(r, c, SLAB_Q);
                *reinterpret_cast<uint4 *>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                if constexpr (SPLITQ) *reinterpret_cast<uint4 *>(dst + T::QT) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            }
        }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_ctl[0];
    bool ok = true;

    if (warp < 4u) {
        // ================= softmax: thread tid owns row tid =================================================
        const uint32_t r = row0 + tid;
        const bool r_ok = r < n_rows;
        uint32_t r_lo = 0u, r_hi = 0u;
        if (r_ok) query_range(p, r / g, &r_lo, &r_hi);
        const uint32_t t_lane = (warp * 32u) << 16, tm_o = tmem + T::O_COL + t_lane;
        const float mult = SPLITQ ? s_mult[tid] : 1.0f, inv_cap = CAP ? 1.0f / p.softcap : 0.f;
        constexpr float GROW = SC ? 4.0f : 8.0f;
        float mref = kMaskedScore, lrow = 0.f;
        uint32_t vs_ref = 0u;                      // SC: exponent bits of the largest V scale so far
        float *const my_scales = s_scales + warp * 128u;
        float ks_next[2] = {1.f, 1.f}, vs_next[2] = {0.f, 0.f};
        auto load_scales = [&](uint32_t it) {
#pragma unroll
            for (uint32_t i = 0; i < 2; ++i) {
                const uint32_t pos = c_lo + it * BN + lane + 32u * i;
                const bool in = it < n_tiles && pos < p.n_kv;
                ks_next[i] = in ? p.k_scales[uint64_t(pos) * p.n_kv_heads + kvh] : 1.f;
                vs_next[i] = in ? p.v_scales[uint64_t(pos) * p.n_kv_heads + kvh] : 0.f;
            }
        };
        if constexpr (SC) load_scales(0);
        for (uint32_t it = 0; it < n_tiles; ++it) {
            float vs_corr = 1.f;
            if constexpr (SC) {
                const uint32_t top = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(vs_next[0], vs_next[1]))) & 0x7f800000u;
                if (top > vs_ref) {
                    vs_corr = vs_ref != 0u && top - vs_ref < (127u << 23) ? __uint_as_float((127u << 23) - (top - vs_ref)) : 0.f;
                    vs_ref = top;
                }
                const float to_ref = __uint_as_float((254u << 23) - vs_ref) * kPUnit;
                __syncwarp();                      // the previous tile's have been read
#pragma unroll
                for (uint32_t i = 0; i < 2; ++i) {
                    my_scales[lane + 32u * i] = ks_next[i];
                    my_scales[64u + lane + 32u * i] = vs_next[i] * to_ref;
                }
                __syncwarp();
                load_scales(it + 1);
            }
            const uint32_t buf = it & 1u, tm_s = tmem + buf * T::S_COLS + t_lane, t0 = c_lo + it * BN;
            if (!mbar_wait(bar(buf), (it >> 1) & 1u)) { ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float s[64];
            tmem_ld64(tm_s, s);
            if constexpr (T::ACC2) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float x[32];
                    tmem_ld32(tm_s + 64u + 32u * h, x);
#pragma unroll
                    for (int j = 0; j < 32; ++j) s[32 * h + j] += x[j];
                }
            }
            if constexpr (SC) {
#pragma unroll
                for (int j = 0; j < 64; j += 4) {
                    const float4 k4 = *reinterpret_cast<const float4 *>(my_scales + j);
                    s[j] *= mult * k4.x; s[j + 1] *= mult * k4.y; s[j + 2] *= mult * k4.z; s[j + 3] *= mult * k4.w;
                }
            } else if constexpr (SPLITQ) {
#pragma unroll
                for (int j = 0; j < 64; ++j) s[j] *= mult;
            }
            if constexpr (CAP) {
                softcap_all(s, p.softcap, inv_cap);
#pragma unroll
                for (int j = 0; j < 64; ++j) s[j] *= kLog2e;
            }
            const bool full = t0 >= r_lo && t0 + BN <= r_hi;
            const bool warp_full = __all_sync(0xffffffffu, full);
            if (!warp_full) {
#pragma unroll
                for (int j = 0; j < 64; ++j)
                    if (t0 + j < r_lo || t0 + j >= r_hi) s[j] = kMaskedScore;
            }
            float mx = kMaskedScore;
#pragma unroll
            for (int j = 0; j < 64; j += 2) mx = fmaxf(mx, fmaxf(s[j], s[j + 1]));
            const bool grow = mx > mref + GROW;
            if (__any_sync(0xffffffffu, grow) || (SC && vs_corr != 1.f)) {
                const float mnew = grow ? mx : mref, alpha = fast_exp2(mref - mnew);
                lrow *= alpha;
                mref = mnew;
                if (it > 0u) {                     // O is touched only between products: the last one has to be complete
                    if (!mbar_wait(bar(4u + (buf ^ 1u)), ((it - 1u) >> 1) & 1u)) { ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const float f = SC ? alpha * vs_corr : alpha;
#pragma unroll 1
                    for (int c = 0; c < D / 32; ++c) {
                        float o[32];
                        tmem_ld32(tm_o + 32 * c, o);
#pragma unroll
                        for (int j = 0; j < 32; ++j) o[j] *= f;
                        tmem_st32(tm_o + 32 * c, o);
                        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    }
                }
            }
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 64; ++j) {
                float e = fast_exp2(s[j] - mref);
                if (!warp_full) e = s[j] <= 0.5f * kMaskedScore ? 0.f : e;      // a NaN stays one
                s[j] = e;
                if constexpr (SC) sum += e;
            }
            if constexpr (SC) {
#pragma unroll
                for (int j = 0; j < 64; j += 4) {
                    const float4 v4 = *reinterpret_cast<const float4 *>(my_scales + 64 + j);
                    s[j] *= v4.x; s[j + 1] *= v4.y; s[j + 2] *= v4.z; s[j + 3] *= v4.w;
                }
            }
            float pk[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                const uint32_t w = pack_half2(s[2 * j], s[2 * j + 1]);
                pk[j] = __uint_as_float(w);
                if constexpr (!SC) sum = add_halves(sum, w);
            }
            lrow += sum;
            tmem_st32(tm_s, pk);
            if constexpr (SC) {
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    const uint32_t w = __float_as_uint(pk[j]);
                    const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w));
                    pk[j] = __uint_as_float(pack_half2(s[2 * j] - f.x, s[2 * j + 1] - f.y));
                }
                tmem_st32(tm_s + 32u, pk);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            mbar_arrive(bar(2u + buf));
        }
        if (!ok) s_ctl[1] = 1u;
        bool ran = n_tiles > 0u && ok;
        if (ran && !mbar_wait(bar(4u + ((n_tiles - 1u) & 1u)), ((n_tiles - 1u) >> 1) & 1u)) { s_ctl[1] = 1u; ran = false; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (s_ctl[1] != 0u) ran = false;
        // ---- rows out: each warp stages its 32 rows where Q and the ring were (every product has been
        // through with them), so that a store covers whole rows
        const float unit = SC ? __uint_as_float(vs_ref) * (1.0f / kPUnit) : 1.0f;
        float row_scale, finite = 0.f;             // finite: 0, or NaN if an element is not
        float *row_dst, *piece = nullptr;
        if (op.n_split > 1u) {
            piece = op.scratch + uint64_t(blockIdx.x) * T::PIECE;
            piece[BM * D + tid] = ran ? mref : kMaskedScore;
            piece[BM * D + BM + tid] = ran ? lrow : 0.f;
            row_scale = unit;
            row_dst = r_ok ? piece + tid * D : nullptr;
        } else {
            row_scale = ran && lrow > 0.f ? unit / lrow : 0.f;
            row_dst = r_ok ? p.out + (uint64_t(r / g) * p.n_q_heads + kvh * g + r % g) * D : nullptr;
        }
        constexpr uint32_t ROWB = D * 4, UNITS = D / 4, SW = UNITS < 32 ? UNITS - 1 : 31;
        uint8_t *const stage = sm + warp * 32u * ROWB;
#pragma unroll 1
        for (uint32_t c = 0; c < D / 32; ++c) {
            float v[32];
            if (ran) {
                tmem_ld32(tm_o + 32 * c, v);
            } else {
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = 0.f;
            }
#pragma unroll
            for (int j = 0; j < 32; ++j) { v[j] *= row_scale; finite = fmaf(v[j], 0.f, finite); }
#pragma unroll
            for (uint32_t j = 0; j < 8; ++j)
                *reinterpret_cast<float4 *>(stage + lane * ROWB + (((8u * c + j) ^ (lane & SW)) << 4)) =
                    make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        }
        __syncwarp();
        const unsigned long long mine = reinterpret_cast<unsigned long long>(row_dst);
#pragma unroll 4
        for (uint32_t i = lane; i < 32u * UNITS; i += 32u) {
            const uint32_t rr = i / UNITS, u = i % UNITS;
            const unsigned long long dst = __shfl_sync(0xffffffffu, mine, int(rr));
            const float4 x = *reinterpret_cast<const float4 *>(stage + rr * ROWB + ((u ^ (rr & SW)) << 4));
            if (dst != 0ull) *reinterpret_cast<float4 *>(reinterpret_cast<float *>(dst) + 4u * u) = x;
        }
        const uint32_t cta_end = c_lo + n_tiles * BN;
        for (uint32_t again = __ballot_sync(0xffffffffu, finite != 0.f && r_ok); again != 0u; again &= again - 1u) {
            const int rr = __ffs(int(again)) - 1;
            const uint32_t lo = max(__shfl_sync(0xffffffffu, r_lo, rr), c_lo), hi = min(__shfl_sync(0xffffffffu, r_hi, rr), cta_end);
            float *const dst = reinterpret_cast<float *>(__shfl_sync(0xffffffffu, mine, rr));
            float *const m_out = piece ? piece + BM * D + warp * 32u + uint32_t(rr) : nullptr;
            __syncwarp();
            row_alone<DT, D>(&op.a, row0 + warp * 32u + uint32_t(rr), kvh, lo, hi, dst, m_out, m_out ? m_out + BM : nullptr);
        }
    } else if (warp == 4u) {
        // ================= the MMA thread ===================================================================
        if (lane == 0u && n_tiles > 0u) {
            auto issue_s = [&](uint32_t t) {
                const uint32_t st = t % NK, b0 = ring + st * T::STAGE, d = tmem + (t & 1u) * T::S_COLS;
                for (uint32_t h = 0; h < (SPLITQ ? 2u : 1u); ++h) {
                    const uint32_t a0 = q_sm + h * T::QT;
#pragma unroll
                    for (uint32_t ks = 0; ks < D / 16; ++ks)
                        umma_f16(d + (T::ACC2 ? (ks & 1u) * 64u : 0u), smem_desc(a0 + (ks >> 2) * SLAB_Q + (ks & 3u) * 32u, 16, 1024),
                                 smem_desc(b0 + (ks >> 2) * SLAB_KV + (ks & 3u) * 32u, 16, 1024), idesc_f16(false, BN), T::ACC2 ? h | (ks >> 1) : h | ks);
                }
                umma_commit(bar(t & 1u));
                umma_commit(bar(free0 + st));
            };
            auto issue_pv = [&](uint32_t t) {
                const uint32_t st = NK + t % NV, b0 = ring + st * T::STAGE, a0 = tmem + (t & 1u) * T::S_COLS;
#pragma unroll
                for (uint32_t h = 0; h < (SC ? 2u : 1u); ++h)
#pragma unroll
                    for (uint32_t kk = 0; kk < BN / 16; ++kk)
                        umma_f16_ts(tmem + T::O_COL, a0 + 32u * h + kk * 8u, smem_desc(b0 + kk * 2048u, SLAB_KV, 1024),
                                    idesc_f16(true, D), t | h | kk);
                umma_commit(bar(4u + (t & 1u)));
                umma_commit(bar(free0 + st));
            };
            auto k_full = [&](uint32_t t) { return mbar_test(bar(full0 + t % NK), (t / NK) & 1u); };
            auto v_full = [&](uint32_t t) { return mbar_test(bar(full0 + NK + t % NV), (t / NV) & 1u); };
            uint32_t next_s = 0u, next_pv = 0u, idle = 0u;
            uint64_t t_idle = 0;
            while (next_pv < n_tiles && ok) {
                bool did = false;
                // S(t) goes over P(t - 2), whose product has been issued before (products of a thread run in order)
                if (next_s < n_tiles && next_s < next_pv + 2u && k_full(next_s)) {
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    issue_s(next_s++);
                    did = true;
                }
                if (next_pv < next_s && mbar_test(bar(2u + (next_pv & 1u)), (next_pv >> 1) & 1u) && v_full(next_pv)) {
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    issue_pv(next_pv++);
                    did = true;
                }
                if (did) { idle = 0u; t_idle = 0; }
                else if ((++idle & 1023u) == 0u) {
                    if (t_idle == 0) t_idle = timer_ns();
                    else if (timer_ns() - t_idle > 1000000000ull) ok = false;
                    if (s_ctl[1] != 0u) ok = false;
                }
            }
            if (!ok) s_ctl[1] = 1u;
        }
    } else if constexpr (FP8) {
        // ================= K / V rows: fetch a tile ahead, widen, place ======================================
        for (uint32_t it = 0; it < n_tiles; ++it) {
            uint4 cur[NP];
#pragma unroll
            for (uint32_t i = 0; i < NP; ++i) cur[i] = raw[i];
            if (it + 1u < n_tiles) fetch(it + 1u);
            const uint32_t ns = is_v ? NV : NK, st = (is_v ? NK : 0u) + it % ns;
            if (it >= ns && !mbar_wait(bar(free0 + st), (it / ns - 1u) & 1u)) { ok = false; break; }
            uint8_t *const dst = sm + T::Q + st * T::STAGE;
#pragma unroll
            for (uint32_t i = 0; i < NP; ++i) {
                const uint32_t idx = pt + 96u * i, pos = idx / (D / 16), c = idx % (D / 16);
                if (idx >= PIECES) continue;
                const uint32_t w[4] = {cur[i].x, cur[i].y, cur[i].z, cur[i].w};
                uint32_t h[8];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const __half2 lo = e4m3x2_to_half2(w[j] & 0xffffu), hi = e4m3x2_to_half2(w[j] >> 16);
                    h[2 * j] = *reinterpret_cast<const uint32_t *>(&lo);
                    h[2 * j + 1] = *reinterpret_cast<const uint32_t *>(&hi);
                }
                *reinterpret_cast<uint4 *>(dst + chunk_off(pos, 2u * c, SLAB_KV)) = make_uint4(h[0], h[1], h[2], h[3]);
                *reinterpret_cast<uint4 *>(dst + chunk_off(pos, 2u * c + 1u, SLAB_KV)) = make_uint4(h[4], h[5], h[6], h[7]);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mbar_arrive(bar(full0 + st));
        }
        if (!ok) s_ctl[1] = 1u;
    } else if (tid == 160u || tid == 256u) {
        // ================= K (one thread) and V rows (another) by TMA; positions from n_kv on are outside the
        // map: zeros ==========================================================================================
        const uint32_t ns = is_v ? NV : NK, first = is_v ? NK : 0u;
        const CUtensorMap *const tm = is_v ? &tm_v : &tm_k;
        uint32_t it = 0u;
        for (; it < n_tiles; ++it) {
            const uint32_t st = first + it % ns, dst = ring + st * T::STAGE;
            if (it >= ns && !mbar_wait(bar(free0 + st), (it / ns - 1u) & 1u)) { ok = false; break; }
            mbar_expect_tx(bar(full0 + st), T::STAGE);
#pragma unroll
            for (uint32_t c = 0; c < D / 64; ++c)
                tma_load_2d(dst + c * SLAB_KV, tm, int32_t(kvh * D * ES + c * 128u), int32_t(c_lo + it * BN), bar(full0 + st));
        }
        if (!ok) {                             // leave nothing in flight: the last copies into every stage have landed
            s_ctl[1] = 1u;
            for (uint32_t i = it > ns ? it - ns : 0u; i < it; ++i) mbar_wait(bar(full0 + first + i % ns), (i / ns) & 1u);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (s_ctl[1] != 0u && tid == 0) atomicOr(op.status, 1u);
    if (warp == 4u) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "n"(T::TMEM) : "memory");
}

// The pieces of every row block put together: a warp per row.  grid = (kv-head x 16 row groups, row blocks: at most
// two CTAs an SM are cut).
template <int D>
__global__ void __launch_bounds__(256) prefill_pieces_kernel(const OneTileParams op)
{
    constexpr uint64_t PIECE = OneTile<D, false>::PIECE;
    constexpr uint32_t NV = D < 128 ? 1 : D / 128, LANES = D / 4 < 32 ? D / 4 : 32;
    const PrefillParams &p = op.a;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, n = op.n_split;
    const uint32_t kvh = blockIdx.x / 16u, rl = (blockIdx.x % 16u) * 8u + warp, g = p.group;
    const uint32_t r = (op.n_rb - 1u - blockIdx.y) * uint32_t(BM) + rl;
    pdl_wait();
    if (r >= p.m * g) return;
    const float *const first = op.scratch + (uint64_t(blockIdx.y) * p.n_kv_heads + kvh) * n * PIECE;
    float mx = kMaskedScore;
    for (uint32_t i = lane; i < n; i += 32u) mx = fmaxf(mx, __ldcg(first + i * PIECE + BM * D + rl));
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float l = 0.f;
    float4 acc[NV];
#pragma unroll
    for (uint32_t v = 0; v < NV; ++v) acc[v] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t i0 = 0; i0 < n; i0 += 32u) {
        float w_mine = 0.f;
        if (i0 + lane < n) {
            const float *const pc = first + (i0 + lane) * PIECE + BM * D + rl;
            w_mine = fast_exp2(__ldcg(pc) - mx);
            l += w_mine * __ldcg(pc + BM);
        }
        const uint32_t cnt = min(32u, n - i0);
#pragma unroll 8
        for (uint32_t i = 0; i < cnt; ++i) {
            const float w = __shfl_sync(0xffffffffu, w_mine, int(i));
            if (lane < LANES) {
                const float4 *const src = reinterpret_cast<const float4 *>(first + (i0 + i) * PIECE + rl * D) + lane;
#pragma unroll
                for (uint32_t v = 0; v < NV; ++v) {
                    const float4 x = __ldcg(src + 32u * v);
                    acc[v].x = fmaf(w, x.x, acc[v].x); acc[v].y = fmaf(w, x.y, acc[v].y);
                    acc[v].z = fmaf(w, x.z, acc[v].z); acc[v].w = fmaf(w, x.w, acc[v].w);
                }
            }
        }
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    const float inv = l > 0.f ? 1.0f / l : 0.f;                // an empty range yields zeros
    if (lane < LANES) {
        float4 *const out = reinterpret_cast<float4 *>(p.out + (uint64_t(r / g) * p.n_q_heads + kvh * g + r % g) * D) + lane;
#pragma unroll
        for (uint32_t v = 0; v < NV; ++v) out[32u * v] = make_float4(acc[v].x * inv, acc[v].y * inv, acc[v].z * inv, acc[v].w * inv);
    }
}

// CTAs that the tiles of a row block are cut over, and the time of the launch (us), by a model of it: a CTA
// pays t0 once and t1 a tile (measured, in us: 1.07 for FP8 and 0.87 for F16 rows of 128 dims, 1.31 and, with
// Q in two terms, 1.75 for 256, 1.65 for scaled FP8 of 128), pieces cost a second launch and their traffic.
// CTAs beyond one an SM share its tensor cores and issue slots: the SMs that got one more set the time (700 queries
// at 20 000, F16: 176 CTAs take twice one CTA's time).
struct Cut { uint32_t pieces; double us; };
Cut best_cut(const vfkv_ctx *ctx, uint32_t dtype, bool split_q, const PrefillParams &p)
{
    const uint32_t D = p.head_dim, n_rb = uint32_t((uint64_t(p.m) * p.group + BM - 1) / BM);
    uint32_t longest = 0;
    uint64_t total = 0;
    for (uint32_t rb = 0; rb < n_rb; ++rb) {
        uint32_t r0, cl, nt;
        block_extent(p, n_rb, rb, &r0, &cl, &nt);
        longest = std::max(longest, nt);
        total += uint64_t(nt) * p.n_kv_heads;
    }
    const bool sc = p.k_scales != nullptr;
    const double t1 = (dtype == VFKV_F8 ? (D == 256 ? 1.31 : D == 128 ? 1.07 : 0.95) : 0.87) +
                      (sc ? (D == 256 ? 0.9 : 0.6) : split_q ? (D == 256 ? 0.88 : D == 128 ? 0.2 : 0.0) : 0.0) + (p.softcap > 0.f ? 0.3 : 0.0);
    const double t0 = D == 256 ? 9.0 : 7.0;
    const uint64_t items = uint64_t(n_rb) * p.n_kv_heads, n_sm = uint64_t(ctx->sm_count);
    Cut best{1, 1e30};
    for (uint32_t n = 1; n <= 64 && n <= std::max(longest, 1u); ++n) {
        if (n > 1 && (p.whole || items * n > n_sm * 2)) break;
        const double one_cta = t0 + t1 * double((longest + n - 1) / n);
        double us = one_cta;
        if (items * n > n_sm)
            us = std::max(us, double((items * n + n_sm - 1) / n_sm) * (t0 + t1 * double(total) / double(items * n)));
        if (n > 1) us += 5.0 + 0.3 * n * D / 128.0;
        if (us < best.us * 0.98) best = {n, us};
    }
    return best;
}

template <int DT, int D, bool SPLITQ, bool SC, bool CAP>
int32_t launch_one_tile_t(vfkv_ctx *ctx, OneTileParams op, cudaStream_t st)
{
    using T = OneTile<D, SPLITQ>;
    const PrefillParams &p = op.a;
    auto kern = prefill_one_tile_kernel<DT, D, SPLITQ, SC, CAP>;
    static std::atomic<bool> configured[64];
    if (!configured[ctx->device & 63].load(std::memory_order_acquire)) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, T::SMEM);
        if (e != cudaSuccess) return check_cuda(ctx, e, "cudaFuncSetAttribute(one-tile prefill attention)");
        configured[ctx->device & 63].store(true, std::memory_order_release);
    }
    CUtensorMap tm_k, tm_v;
    memset(&tm_k, 0, sizeof tm_k);
    memset(&tm_v, 0, sizeof tm_v);
    if (DT == VFKV_F16 && p.n_kv != 0u &&
        (!encode_rows_map(ctx, &tm_k, p.k, p.row_bytes, p.n_kv, BN) || !encode_rows_map(ctx, &tm_v, p.v, p.row_bytes, p.n_kv, BN)))
        return set_error(ctx, VFKV_ERR_CUDA, "cuTensorMapEncodeTiled failed");
    op.n_rb = uint32_t((uint64_t(p.m) * p.group + BM - 1) / BM);
    op.n_split = best_cut(ctx, DT, SPLITQ, p).pieces;
    if (op.n_split > 1) {
        uint64_t floats = 0;
        op.scratch = prefill_scratch(ctx, st, &floats);
        const uint64_t most = op.scratch ? floats / T::PIECE / (uint64_t(op.n_rb) * p.n_kv_heads) : 1;
        if (op.n_split > most) op.n_split = most > 1 ? uint32_t(most) : 1u;
    }
    op.status = ctx->d_status;
    cudaError_t e = launch_dependent(ctx, kern, dim3(op.n_split * p.n_kv_heads * op.n_rb), dim3(kThreads), T::SMEM, st, op, tm_k, tm_v);
    ctx->count_launch();
    if (e == cudaSuccess && op.n_split > 1) {
        e = launch_dependent(ctx, prefill_pieces_kernel<D>, dim3(p.n_kv_heads * 16, op.n_rb), dim3(256), 0, st, op);
        ctx->count_launch();
    }
    prefill_scratch_used(ctx, st, op.scratch);
    return check_cuda(ctx, e, "one-tile prefill attention launch");
}

template <int DT, int D, bool SPLITQ, bool SC>
int32_t launch_one_tile_c(vfkv_ctx *ctx, const OneTileParams &op, cudaStream_t st)
{
    return op.a.softcap > 0.f ? launch_one_tile_t<DT, D, SPLITQ, SC, true>(ctx, op, st)
                              : launch_one_tile_t<DT, D, SPLITQ, SC, false>(ctx, op, st);
}

template <int D>
int32_t launch_one_tile_d(vfkv_ctx *ctx, uint32_t dtype, bool split_q, const OneTileParams &op, cudaStream_t st)
{
    if (dtype == VFKV_F8)
        return op.a.k_scales ? launch_one_tile_c<VFKV_F8, D, true, true>(ctx, op, st) : launch_one_tile_c<VFKV_F8, D, false, false>(ctx, op, st);
    if constexpr (D == 128)
        if (!split_q) return launch_one_tile_c<VFKV_F16, D, false, false>(ctx, op, st);
    return launch_one_tile_c<VFKV_F16, D, true, false>(ctx, op, st);
}

}  // namespace

bool prefill_one_tile_supported(const vfkv_ctx *ctx, uint32_t dtype, uint32_t D)
{
    return (D == 64 || D == 128 || D == 256) && (dtype == VFKV_F8 || (dtype == VFKV_F16 && ctx->encode_tiled));
}

double prefill_one_tile_us(const vfkv_ctx *ctx, uint32_t dtype, bool split_q, const PrefillParams &p)
{
    return best_cut(ctx, dtype, split_q || (dtype == VFKV_F16 && p.head_dim != 128), p).us;
}

int32_t launch_prefill_one_tile(vfkv_ctx *ctx, uint32_t dtype, bool split_q, const PrefillParams &p, cudaStream_t st)
{
    OneTileParams op{};
    op.a = p;
    switch (p.head_dim) {
    case 64: return launch_one_tile_d<64>(ctx, dtype, split_q, op, st);
    case 128: return launch_one_tile_d<128>(ctx, dtype, split_q, op, st);
    default: return launch_one_tile_d<256>(ctx, dtype, split_q, op, st);
    }
}

}  // namespace vfkv
