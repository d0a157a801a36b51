// Chunked-prefill causal attention on tcgen05 with one Q tile of 128 rows a CTA: the shapes that the
// two-tile kernel of attn_prefill_tc5.cu does not hold (head_dim 64 and 256, Q as two half-precision
// terms, FP8 rows with a scale per position and head) and chunks with few rows.
//
// CTA = 128 rows (128 / g consecutive queries x the g q-heads of a kv-head) x K/V tiles of 64 positions.
//   warps 0-3, 4-7   softmax of the even and of the odd tiles: thread = row; scores out of tensor memory, P back over them
//   warp  8          issues every MMA, all lanes running through: S(t) = Q K^T, up to four tiles ahead (one or two of 256 dims
//                    in two terms), each behind the O += P V that frees its columns
//   the rest         K and V rows into a ring of stages each: FP8 fetched, widened and placed by three warps
//                    each, two tiles ahead in registers; F16 copied by TMA, the first ones requested before Q is
// What bounds a tile (F16, 128 dims): the exponentials of its 8192 scores, 512 of some 900 cycles.  One group of softmax warps
// took a tile's whole chain of latencies (scores out, maximum, exponentials, P back) for every tile, and one thread
// that issued the products 700 cycles for what a warp with its operands in uniform registers issues in 130: 333 queries of
// 1333 (F16, with the RoPE and append launches) 32.4 -> 24.5 us; 231 of 2589, 64 / 8 heads 51.5 -> 36.0; 1024 of 5120 with 256
// dims, window and soft-cap 66 -> 54; FP8, 484 of 1147 36.3 -> 30.1, 38 of 21 152 62.8 -> 50.
// 64 positions a tile, because Q of 256 dims in two terms takes 128 KB and leaves room for three stages (two
// of K, whose products come a tile earlier, and one of V).
// A row's exponents refer to a maximum that is moved, and O rescaled, only when the true one has outgrown
// it by 2^14, which half precision holds.  The two groups share O, and so the reference: a tile that leaves it alone says so
// as soon as its maximum is known and goes on with the reference as far as its group knows it; before P is handed over it
// looks at what the tile before left, and starts again from the scores if that is another (in a row's first tiles).  A tile
// that moves the reference waits for the product of the tile before.  (Handed from tile to tile instead, it cost 300 cycles
// a tile; moved from 2^8 on, FP8 calls with outliers took up to 15 % longer: 30 queries of 35 666 49.2 against 56.2 us.)
// The largest p is then any number up to 2^14 and not 1, so a row's sum is taken of the
// p as they go into the product, rounded to half precision: a row that one position dominates is that position's V
// whatever its p was rounded to (with the sum of the unrounded p: off by up to 2^-12).
//
// SPLITQ: Q = high + low half-precision term, scaled per row by a power of two (two products for S).
// SC: the scales of K multiply the scores, those of V multiply P, in f32; P is then also fed as two terms,
// relative to the largest power of two among the V scales so far (exact but for 2^-22 of it, or for the last bit of the second
// term: 2^-34 of the row's largest p x the largest V scale), which makes the result as accurate as f32 tiles on the CUDA cores.
// So the reference lags by 2^4 at most here: room for a lag of 2^9 in the first term would take five bits from the second
// (V scales 2^12 apart, 256 dims x 500 positions: 1.2e-5 off against 64 bits where this is 2.3e-6; no faster).
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
// 8 softmax warps, the MMA warp, and for K and for V three warps each (FP8: widening) or one (F16: a thread that issues TMA)
template <int DT> constexpr uint32_t kThreads = DT == VFKV_F8 ? 480 : 352;
constexpr uint32_t SLAB_Q = 128 * 128, SLAB_KV = 64 * 128;      // [rows][64 halves], 128-byte swizzle
constexpr uint32_t kSmall = 3072;                               // barriers, row multipliers, tile scales
constexpr float kPUnit = 1024.0f;                               // SC: P terms are fed as p * v_scale / reference * 2^10 <= 2^15

struct OneTileParams {
    PrefillParams a;
    uint32_t n_split, n_rb;
    float *scratch;                    // pieces {O [128][D], reference maxima [128], sums [128]} of n_split > 1
    uint32_t *status;
};

template <int D, bool SPLITQ> struct OneTile {
    // Q of up to 128 dims lies in tensor memory (an MMA with both operands in shared memory takes as long as the reads
    // of 128 rows of Q and 64 of K, twice the products' own time), of 256 in shared memory.
    static constexpr bool QTM = D <= 128;
    static constexpr uint32_t QT = BM * D * 2, Q = QT * (SPLITQ ? 2 : 1), STAGE = BN * D * 2;
    static constexpr uint32_t ROOM = 227 * 1024 - kSmall - Q, NST = ROOM / STAGE < 8 ? ROOM / STAGE : 8;
    static constexpr uint32_t NK = (NST + 1) / 2, NV = NST / 2;  // stages of K, stages of V behind them
    static constexpr uint32_t SMEM = Q + NST * STAGE + kSmall;
    // Columns of tensor memory: S of even and odd tiles, then O.  With 32 products a tile (256 dims, Q in two
    // terms) those of S go to two accumulators in turn, which the softmax adds: MMAs into one wait for each
    // other (1.85 -> 1.73 us a tile; with 16 products the addition costs as much as it saves).
    static constexpr bool ACC2 = D > 128 && SPLITQ;
    static constexpr uint32_t S_COLS = ACC2 ? 128 : 64, NSB = ACC2 ? 2 : 4, O_COL = NSB * S_COLS, Q_COL = O_COL + D, TMEM = 512;
    static_assert(Q_COL + (QTM ? (SPLITQ ? D : D / 2) : 0) <= TMEM, "columns");
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

// What a group tells the other of a row: the reference, and the number of its tiles that it is of.  Who finds the tile that it
// waits for, or a later one (at most a second), has the reference of that tile or a later one: they only rise.  One word of
// 64 bits, stored and loaded whole; with scales, where shared memory has no room for those and the exponent goes along, the
// references and a count behind them for each warp (28 against 29.5 us a call of 98 queries at 2616, but 25.0 against 24.2 for
// 333 of 1333, F16).  The count in the reference's own low bits would move it by up to 15 units in its last place, which from
// scores of 2^24 on is more binary orders than half precision has.
__device__ __forceinline__ void word_set(uint32_t at, uint32_t value)
{
    asm volatile("st.volatile.shared::cta.u32 [%0], %1;" :: "r"(at), "r"(value) : "memory");
}
__device__ __forceinline__ uint32_t word_get(uint32_t at)
{
    uint32_t value;
    asm volatile("ld.volatile.shared::cta.u32 %0, [%1];" : "=r"(value) : "r"(at) : "memory");
    return value;
}
__device__ __forceinline__ void pair_set(uint32_t at, float value, uint32_t count)
{
    asm volatile("st.volatile.shared::cta.u64 [%0], %1;" :: "r"(at), "l"(uint64_t(count) << 32 | __float_as_uint(value)) : "memory");
}
__device__ __forceinline__ void count_set(uint32_t at, uint32_t count)      // by one lane, behind __syncwarp()
{
    asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" :: "r"(at), "r"(count) : "memory");
}
template <typename Look> __device__ __forceinline__ bool wait_until(Look look)
{
    uint64_t t0 = 0;
    for (uint32_t it = 0;; ++it) {
        if (look()) return true;
        if ((it & 1023u) == 1023u) {
            if (t0 == 0) t0 = timer_ns();
            else if (timer_ns() - t0 > 1000000000ull) return false;
        }
    }
}
__device__ __forceinline__ bool pair_wait(uint32_t at, uint32_t count, float *value)
{
    return wait_until([&]() {
        uint64_t w;
        asm volatile("ld.volatile.shared::cta.u64 %0, [%1];" : "=l"(w) : "r"(at) : "memory");
        *value = __uint_as_float(uint32_t(w));
        return uint32_t(w >> 32) >= count;
    });
}
__device__ __forceinline__ bool count_wait(uint32_t at, uint32_t count)
{
    return wait_until([&]() {
        uint32_t n;
        asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(n) : "r"(at) : "memory");
        return n >= count;
    });
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
__global__ void __launch_bounds__(kThreads<DT>, 1)
prefill_one_tile_kernel(const __grid_constant__ OneTileParams op, const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v)
{
    using T = OneTile<D, SPLITQ>;
    static_assert(!SC || (SPLITQ && DT == VFKV_F8), "scales belong to FP8 caches and keep f32 accuracy");
    constexpr bool FP8 = DT == VFKV_F8;
    constexpr uint32_t NST = T::NST, NK = T::NK, NV = T::NV, NSB = T::NSB, ES = FP8 ? 1 : 2, NW = kThreads<DT> / 32;
    const PrefillParams &p = op.a;
    extern __shared__ __align__(1024) uint8_t sm[];
    const uint32_t base = smem_addr(sm), q_sm = base, ring = base + T::Q, small = ring + NST * T::STAGE;
    uint8_t *const sm_small = sm + T::Q + NST * T::STAGE;
    // 0: barriers   352: tensor memory address, abort flag   384: row multipliers [128]
    // 896: the reference maximum of a row as a group knows it and the number of the group's tiles that it is of [group][128]
    // SC: 896: the reference [group][128]   1920: the exponent of the largest V scale [group][quarter of the rows]   1952: the
    // number of tiles that these are of [group][quarter]   2048: a tile's scales [group][64 of K, 64 of V]
    volatile uint32_t *const s_ctl = reinterpret_cast<uint32_t *>(sm_small + 352);
    float *const s_mult = reinterpret_cast<float *>(sm_small + 384);
    const uint32_t refs = small + 896u, vrefs = small + 1920u, counts = small + 1952u;
    float *const s_scales = reinterpret_cast<float *>(sm_small + 2048);
    const uint32_t tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31u;
    const uint32_t g = p.group, n_rows = p.m * g;
    // barriers: S ready [buffer] (commit)   P ready [buffer] (128)   P V done [buffer] (commit)   all products done (commit)
    // stage full   stage free (commit).  A wait on a phase parity must not be more than one phase away from the barrier's
    // state.  For P V done: S(t) goes behind P V(t - NSB), so who has seen S(t) may wait for the products of up to t - 1,
    // whose barriers were last completed by t - NSB - 1 or earlier, and are next by a product behind P V(t).
    auto bar = [&](uint32_t i) { return small + 8u * i; };
    constexpr uint32_t s0 = 0u, p0 = NSB, o0 = 2u * NSB, done = 3u * NSB, full0 = done + 1u, free0 = full0 + NST;
    static_assert(8u * (free0 + NST) <= 352u, "barriers");
    if ((base & 1023u) != 0u) {                // the swizzle counts on it; the array's alignment provides it
        if (tid == 0) atomicOr(op.status, 1u);
        return;
    }
    if (tid == 0) {
        for (uint32_t i = 0; i < NSB; ++i) { mbar_init(bar(s0 + i), 1); mbar_init(bar(p0 + i), BM); }
        for (uint32_t i = o0; i < full0; ++i) mbar_init(bar(i), 1);
        for (uint32_t i = 0; i < NST; ++i) { mbar_init(bar(full0 + i), FP8 ? 3u : 1u); mbar_init(bar(free0 + i), 1); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_ctl[1] = 0u;
    }
    if constexpr (SC) {
        if (tid < 16u) word_set(vrefs + 4u * tid, 0u);     // the counts as well
    } else {
        if (tid < 256u) pair_set(refs + 8u * tid, 0.f, 0u);
    }
    if (warp == 8) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(small + 352u), "n"(T::TMEM) : "memory");
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
    __syncthreads();                           // the barriers are there
    pdl_wait();

    // ---- K/V rows of FP8 caches: 96 threads for K, 96 for V, the first tiles requested before Q is -----
    constexpr uint32_t PIECES = BN * D / 16;                    // 16-code pieces of a stage
    constexpr uint32_t NP = (PIECES + 95) / 96;
    const bool is_v = FP8 ? warp >= 12u : warp >= 10u;
    const uint32_t pt = tid - (is_v ? 384u : 288u);
    // two tiles in flight: a thread's pieces of tile t are in buffer t & 1, which t + 2's are fetched into as soon as
    // they are placed
    uint4 raw[FP8 ? 2 : 1][FP8 ? NP : 1];
    constexpr uint32_t UNITS_ROW = D / 16, STEP = 96 / UNITS_ROW;      // a thread's pieces lie STEP rows apart in one column
    const uint32_t pr = pt / UNITS_ROW, pc = pt % UNITS_ROW;
    const uint8_t *const rows = (is_v ? p.v : p.k) + uint64_t(kvh) * D + pc * 16u + uint64_t(c_lo + pr) * p.row_bytes;
    auto fetch = [&](uint32_t it, uint4 (&to)[FP8 ? NP : 1]) {
        const uint8_t *src = rows + uint64_t(it) * BN * p.row_bytes;
        const uint32_t t0 = c_lo + it * BN, left = it < n_tiles && t0 < p.n_kv ? min(p.n_kv - t0, uint32_t(BN)) : 0u;
#pragma unroll
        for (uint32_t i = 0; i < NP; ++i)
            to[i] = pr + STEP * i < left ? *reinterpret_cast<const uint4 *>(src + i * (STEP * p.row_bytes)) : make_uint4(0u, 0u, 0u, 0u);
    };
    if constexpr (FP8)
        if (warp >= 9u) {
            fetch(0u, raw[0]);
            if constexpr (D < 256) fetch(1u, raw[1]);           // of 256 dims, behind Q: registers
        }
    // F16 rows by TMA, one thread for K and one for V; positions from n_kv on are outside the map: zeros
    const uint32_t ns_tma = is_v ? NV : NK, first_tma = is_v ? NK : 0u;
    auto copy_rows = [&](uint32_t it) {
        const uint32_t st = first_tma + it % ns_tma, dst = ring + st * T::STAGE;
        const CUtensorMap *const tm = is_v ? &tm_v : &tm_k;
        mbar_expect_tx(bar(full0 + st), T::STAGE);
#pragma unroll
        for (uint32_t c = 0; c < D / 64; ++c)
            tma_load_2d(dst + c * SLAB_KV, tm, int32_t(kvh * D * ES + c * 128u), int32_t(c_lo + it * BN), bar(full0 + st));
    };
    if constexpr (!FP8)
        if (tid == 288u || tid == 320u) {
            for (uint32_t it = 0; it < ns_tma && it < n_tiles; ++it) copy_rows(it);
        }

    // ---- Q -> shared memory, all warps: D / 8 neighbouring lanes hold a row --------------------------
    {
        constexpr uint32_t CHUNKS = BM * D / 8 / 32, QB = D == 256 ? 6 : (CHUNKS + NW - 1) / NW;      // of up to 128 dims in one go
        const float q_mult = p.scale * (CAP ? 1.0f : kLog2e);
        const uint32_t g_shift = 31u - __clz(g);
        const bool g_pow2 = (g & (g - 1u)) == 0u;
        for (uint32_t c0 = warp; c0 < CHUNKS; c0 += NW * QB) {
            float4 a[QB], b[QB];
#pragma unroll
            for (uint32_t u = 0; u < QB; ++u) {
                const uint32_t idx = (c0 + NW * u) * 32u + lane, r = row0 + idx / (D / 8), c = idx % (D / 8);
                const bool in = c0 + NW * u < CHUNKS && r < n_rows;
                const uint32_t qi = g_pow2 ? r >> g_shift : r / g;
                const float4 *src = reinterpret_cast<const float4 *>(p.q + (uint64_t(qi) * p.n_q_heads + kvh * g + (r - qi * g)) * D + 8 * c);
                a[u] = in ? *src : make_float4(0.f, 0.f, 0.f, 0.f);
                b[u] = in ? src[1] : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (uint32_t u = 0; u < QB; ++u) {
                if (c0 + NW * u >= CHUNKS) break;
                const uint32_t idx = (c0 + NW * u) * 32u + lane, r = idx / (D / 8), c = idx % (D / 8);
                float x[8] = {a[u].x * q_mult, a[u].y * q_mult, a[u].z * q_mult, a[u].w * q_mult,
                              b[u].x * q_mult, b[u].y * q_mult, b[u].z * q_mult, b[u].w * q_mult};
                if constexpr (SPLITQ) {
                    // rows scaled by a power of two into [128, 256); its inverse goes to the scores
                    float top = 0.f;
#pragma unroll
                    for (int j = 0; j < 8; ++j) top = fmaxf(top, fabsf(x[j]));
#pragma unroll
                    for (int o = 1; o < D / 8; o <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
                    int e = int((__float_as_uint(top) >> 23) & 0xFF) - 127;
                    e = top > 0.f ? max(-100, min(100, e)) : 7;
                    const float qs = __uint_as_float(uint32_t(7 - e + 127) << 23);
#pragma unroll
                    for (int j = 0; j < 8; ++j) x[j] *= qs;
                    if (c == 0u) s_mult[r] = __uint_as_float(uint32_t(e - 7 + 127) << 23);
                }
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

    if (warp < 8u) {
        // ================= softmax: threads rt and 128 + rt own row rt, of the even and of the odd tiles ==========
        const uint32_t grp = warp >> 2, quarter = warp & 3u, rt = tid & 127u;
        const uint32_t r = row0 + rt;
        const bool r_ok = r < n_rows;
        uint32_t r_lo = 0u, r_hi = 0xffffffffu;    // rows past the end: nothing to mask, they are not written
        if (r_ok) query_range(p, r / g, &r_lo, &r_hi);
        const uint32_t t_lane = (quarter * 32u) << 16, tm_o = tmem + T::O_COL + t_lane;
        if constexpr (T::QTM) {                    // Q on to tensor memory: half of the row's dims by each of its threads
            constexpr uint32_t HC = D / 16;        // 16-byte chunks of a half
#pragma unroll
            for (uint32_t h = 0; h < (SPLITQ ? 2u : 1u); ++h) {
                float w[4 * HC];
#pragma unroll
                for (uint32_t c = 0; c < HC; ++c) {
                    const float4 x = *reinterpret_cast<const float4 *>(sm + h * T::QT + chunk_off(rt, grp * HC + c, SLAB_Q));
                    w[4 * c] = x.x; w[4 * c + 1] = x.y; w[4 * c + 2] = x.z; w[4 * c + 3] = x.w;
                }
                const uint32_t to = tmem + T::Q_COL + h * (D / 2) + grp * (D / 4) + t_lane;
                if constexpr (HC == 8) tmem_st32(to, w); else tmem_st16(to, w);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            asm volatile("bar.arrive 4, 288;" ::: "memory");
        }
        const float mult = SPLITQ ? s_mult[rt] : 1.0f, inv_cap = CAP ? 1.0f / p.softcap : 0.f;
        // what is left to multiply the scores by when they are exponentiated
        const float late = CAP ? kLog2e : SC ? 1.0f : mult;
        constexpr float GROW = SC ? 4.0f : 14.0f;            // half precision holds p up to 2^16
        float mref = kMaskedScore, lrow = 0.f;      // the row's reference as this group knows it, and its sum of p in terms of it
        uint32_t vs_ref = 0u;                      // SC: exponent bits of the largest V scale so far
        float *const my_scales = s_scales + grp * 128u;
        float sc_next = 0.f;                       // SC: this thread's one of the next tile's 64 + 64 scales
        auto load_scales = [&](uint32_t it) {
            const uint32_t pos = c_lo + it * BN + (rt & 63u);
            const bool in = it < n_tiles && pos < p.n_kv;
            sc_next = in ? (rt < 64u ? p.k_scales : p.v_scales)[uint64_t(pos) * p.n_kv_heads + kvh] : rt < 64u ? 1.f : 0.f;
        };
        if constexpr (SC) load_scales(grp);
        for (uint32_t it = grp; it < n_tiles; it += 2u) {
            if constexpr (SC) {
                asm volatile("bar.sync %0, 128;" :: "r"(1u + grp) : "memory");         // the group's previous tile has been read
                my_scales[rt] = sc_next;
                asm volatile("bar.sync %0, 128;" :: "r"(1u + grp) : "memory");
                load_scales(it + 2u);
            }
            if (!ok) continue;                     // a wait ran out: only the barriers of the group are left to keep
            const uint32_t buf = it % NSB, tm_s = tmem + buf * T::S_COLS + t_lane, t0 = c_lo + it * BN;
            // full: every row of the warp sees the whole tile
            const bool full = __all_sync(0xffffffffu, t0 >= r_lo && t0 + BN <= r_hi);
            // the reference that the other group's tile before left, once it is settled; `moved`: not the one known here.  (A
            // tile that leaves the reference alone is settled as soon as its maximum is known, whatever the tile before did.)
            bool moved = false;
            auto their_ref = [&]() -> bool {
                bool there;
                float theirs;                                    // references only rise: the later one is the larger
                uint32_t v = 0u;
                if constexpr (SC) {
                    there = count_wait(counts + 4u * ((grp ^ 1u) * 4u + quarter), (it + 1u) / 2u);
                    theirs = __uint_as_float(word_get(refs + 4u * ((grp ^ 1u) * 128u + rt)));
                    v = word_get(vrefs + 4u * ((grp ^ 1u) * 4u + quarter));
                } else {
                    there = pair_wait(refs + 8u * ((grp ^ 1u) * 128u + rt), (it + 1u) / 2u, &theirs);
                }
                moved = theirs > mref;
                if (moved) {
                    lrow *= fast_exp2(mref - theirs);
                    mref = theirs;
                }
                if (SC && v > vs_ref) vs_ref = v;
                return __all_sync(0xffffffffu, there);
            };
            // asked first in this group's first tile (no use guessing) and by SC (whose P is two registers a score: no room
            // to wait with it)
            const bool ask_first = SC ? it > 0u : it == 1u;
            if (ask_first && !their_ref()) { ok = false; continue; }
            if (!__all_sync(0xffffffffu, mbar_wait(bar(s0 + buf), (it / NSB) & 1u))) { ok = false; continue; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float pk[32], sum[4], s[64];
            for (uint32_t pass = 0;; ++pass) {     // twice at most
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
                } else if constexpr (SPLITQ && CAP) {
#pragma unroll
                    for (int j = 0; j < 64; ++j) s[j] *= mult;
                }
                if constexpr (CAP) softcap_all(s, p.softcap, inv_cap);
                // a position that the row does not see is -infinity, of which exp2 makes 0 (a NaN stays one)
                if (!full) {
#pragma unroll
                    for (int j = 0; j < 64; ++j)
                        if (t0 + j < r_lo || t0 + j >= r_hi) s[j] = -INFINITY;
                }
                const float mx = max_of(s) * late;
                uint32_t top = 0u;
                if constexpr (SC) top = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(my_scales[64u + lane], my_scales[96u + lane]))) & 0x7f800000u;
                bool asked = it == 0u || ask_first || pass != 0u;
                if (__any_sync(0xffffffffu, mx > mref + GROW) || (SC && top > vs_ref) || it == 0u) {
                    // ---- the reference moves, and O with it, behind the product of the tile before
                    if (it > 0u) {
                        if (!__all_sync(0xffffffffu, mbar_wait(bar(o0 + (it - 1u) % NSB), ((it - 1u) / NSB) & 1u))) { ok = false; break; }
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        if (!their_ref()) { ok = false; break; }
                    }
                    asked = true;
                    const float mnew = mx > mref + GROW ? mx : mref;
                    float f = fast_exp2(mref - mnew);
                    lrow *= f;
                    mref = mnew;
                    if constexpr (SC)
                        if (top > vs_ref) {
                            f *= vs_ref != 0u && top - vs_ref < (127u << 23) ? __uint_as_float((127u << 23) - (top - vs_ref)) : 0.f;
                            vs_ref = top;
                        }
                    if (it > 0u && __any_sync(0xffffffffu, f != 1.f)) {
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
                if (pass == 0u) {                  // what this tile does to the reference is done, or nothing
                    if constexpr (SC) {
                        word_set(refs + 4u * (grp * 128u + rt), __float_as_uint(mref));
                        if (lane == 0u) word_set(vrefs + 4u * (grp * 4u + quarter), vs_ref);
                        __syncwarp();
                        if (lane == 0u) count_set(counts + 4u * (grp * 4u + quarter), it / 2u + 1u);
                    } else {
                        pair_set(refs + 8u * (grp * 128u + rt), mref, it / 2u + 1u);
                    }
                }
                // a row that has seen nothing yet refers to a finite value, from where exp2 gives 0 for it
                const float from = fmaxf(mref, 0.5f * kMaskedScore);
#pragma unroll
                for (int i = 0; i < 4; ++i) sum[i] = 0.f;
                if constexpr (SC) {
                    const float to_ref = __uint_as_float((254u << 23) - vs_ref) * kPUnit;
#pragma unroll
                    for (int j = 0; j < 64; j += 4) {
                        const float4 v4 = *reinterpret_cast<const float4 *>(my_scales + 64 + j);
                        const float v[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float e = fast_exp2(fmaf(s[j + i], late, -from));
                            sum[i] += e;
                            s[j + i] = e * (v[i] * to_ref);
                        }
                    }
#pragma unroll
                    for (int j = 0; j < 32; ++j) pk[j] = __uint_as_float(pack_half2(s[2 * j], s[2 * j + 1]));
                } else {
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const uint32_t w = pack_half2(fast_exp2(fmaf(s[2 * j], late, -from)), fast_exp2(fmaf(s[2 * j + 1], late, -from)));
                        pk[j] = __uint_as_float(w);
                        sum[j & 3] = add_halves(sum[j & 3], w);
                    }
                }
                if (asked) break;
                // was that the reference that the tile before left?  If not (it moves a few times in a row's first tiles),
                // once more: S is still there
                if (!their_ref()) { ok = false; break; }
                if (!__any_sync(0xffffffffu, moved)) break;
            }
            if (!ok) continue;
            lrow += (sum[0] + sum[1]) + (sum[2] + sum[3]);
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
            mbar_arrive(bar(p0 + buf));
        }
        if (!ok) s_ctl[1] = 1u;
        bool ran = n_tiles > 0u && ok;
        // the last product, on a barrier of its own: the last phase of the others may come and go before it is looked at
        if (ran && !mbar_wait(bar(done), 0u)) { s_ctl[1] = 1u; ran = false; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // ---- rows out: each warp stages its half of 32 rows where Q and the ring were (every product has been
        // through with them), so that a store covers whole sectors; behind the rows what the two groups tell each other
        float *const s_end = reinterpret_cast<float *>(sm + T::Q + NST * T::STAGE) - 6 * BM;
        asm volatile("bar.sync 3, 256;" ::: "memory");
        s_end[(2u * grp) * BM + rt] = lrow;
        s_end[(2u * grp + 1u) * BM + rt] = mref;
        asm volatile("bar.sync 3, 256;" ::: "memory");
        if (s_ctl[1] != 0u) ran = false;
        // the later reference is the one that O is at, the sums of before are brought to it
        mref = fmaxf(s_end[BM + rt], s_end[3u * BM + rt]);
        lrow = s_end[rt] * fast_exp2(s_end[BM + rt] - mref) + s_end[2u * BM + rt] * fast_exp2(s_end[3u * BM + rt] - mref);
        if constexpr (SC) vs_ref = max(vs_ref, word_get(vrefs + 4u * ((grp ^ 1u) * 4u + quarter)));        // both groups are through
        const float unit = SC ? __uint_as_float(vs_ref) * (1.0f / kPUnit) : 1.0f;
        float row_scale, finite = 0.f;             // finite: 0, or NaN if an element is not
        float *row_dst, *piece = nullptr;
        if (op.n_split > 1u) {
            piece = op.scratch + uint64_t(blockIdx.x) * T::PIECE;
            if (grp == 0u) {
                piece[BM * D + rt] = ran ? mref : kMaskedScore;
                piece[BM * D + BM + rt] = ran ? lrow : 0.f;
            }
            row_scale = unit;
            row_dst = r_ok ? piece + rt * D : nullptr;
        } else {
            row_scale = ran && lrow > 0.f ? unit / lrow : 0.f;
            row_dst = r_ok ? p.out + (uint64_t(r / g) * p.n_q_heads + kvh * g + r % g) * D : nullptr;
        }
        constexpr uint32_t HALF = D / 2, ROWB = HALF * 4, UNITS = HALF / 4, SW = UNITS < 32 ? UNITS - 1 : 31;
        uint8_t *const stage = sm + warp * 32u * ROWB;
#pragma unroll 1
        for (uint32_t c = 0; c < HALF / 32; ++c) {
            float v[32];
            if (ran) {
                tmem_ld32(tm_o + grp * HALF + 32 * c, v);
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
            if (dst != 0ull) *reinterpret_cast<float4 *>(reinterpret_cast<float *>(dst) + grp * HALF + 4u * u) = x;
        }
        s_end[(4u + grp) * BM + rt] = finite;
        asm volatile("bar.sync 3, 256;" ::: "memory");
        finite = s_end[4u * BM + rt] + s_end[5u * BM + rt];
        const uint32_t cta_end = c_lo + n_tiles * BN;
        // rows with an element that is not finite are done again alone, by the warp of the even tiles
        for (uint32_t again = __ballot_sync(0xffffffffu, grp == 0u && finite != 0.f && r_ok); again != 0u; again &= again - 1u) {
            const int rr = __ffs(int(again)) - 1;
            const uint32_t lo = max(__shfl_sync(0xffffffffu, r_lo, rr), c_lo), hi = min(__shfl_sync(0xffffffffu, r_hi, rr), cta_end);
            float *const dst = reinterpret_cast<float *>(__shfl_sync(0xffffffffu, mine, rr));
            float *const m_out = piece ? piece + BM * D + warp * 32u + uint32_t(rr) : nullptr;
            __syncwarp();
            row_alone<DT, D>(&op.a, row0 + warp * 32u + uint32_t(rr), kvh, lo, hi, dst, m_out, m_out ? m_out + BM : nullptr);
        }
    } else if (warp == 8u) {
        // ================= the MMA warp =====================================================================
        if constexpr (T::QTM) {
            asm volatile("bar.sync 4, 288;" ::: "memory");
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
        const uint32_t leader = mma_leader(), n = __shfl_sync(0xffffffffu, n_tiles, 0), tm = __shfl_sync(0xffffffffu, tmem, 0);
        auto issue_s = [&](uint32_t t) {
            const uint32_t st = t % NK, b0 = ring + st * T::STAGE, d = tm + (t % NSB) * T::S_COLS;
            if (!__all_sync(0xffffffffu, mbar_wait(bar(full0 + st), (t / NK) & 1u))) { ok = false; return; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (uint32_t h = 0; h < (SPLITQ ? 2u : 1u); ++h)
#pragma unroll
                for (uint32_t ks = 0; ks < D / 16; ++ks) {
                    const uint64_t kd = smem_desc(b0 + (ks >> 2) * SLAB_KV + (ks & 3u) * 32u, 16, 1024);
                    if constexpr (T::QTM)
                        umma_f16_ts_by(leader, d, tm + T::Q_COL + h * (D / 2) + ks * 8u, kd, idesc_f16(false, BN), h | ks);
                    else
                        umma_f16_by(leader, d + (T::ACC2 ? (ks & 1u) * 64u : 0u), smem_desc(q_sm + h * T::QT + (ks >> 2) * SLAB_Q + (ks & 3u) * 32u, 16, 1024),
                                    kd, idesc_f16(false, BN), T::ACC2 ? h | (ks >> 1) : h | ks);
                }
            umma_commit_by(leader, bar(s0 + t % NSB));
            umma_commit_by(leader, bar(free0 + st));
        };
        auto issue_pv = [&](uint32_t t) {
            const uint32_t st = NK + t % NV, b0 = ring + st * T::STAGE, a0 = tm + (t % NSB) * T::S_COLS;
            if (!__all_sync(0xffffffffu, mbar_wait(bar(full0 + st), (t / NV) & 1u) && mbar_wait(bar(p0 + t % NSB), (t / NSB) & 1u))) { ok = false; return; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (uint32_t h = 0; h < (SC ? 2u : 1u); ++h)
#pragma unroll
                for (uint32_t kk = 0; kk < BN / 16; ++kk)
                    umma_f16_ts_by(leader, tm + T::O_COL, a0 + 32u * h + kk * 8u, smem_desc(b0 + kk * 2048u, SLAB_KV, 1024),
                                   idesc_f16(true, D), t | h | kk);
            umma_commit_by(leader, bar(o0 + t % NSB));
            umma_commit_by(leader, bar(free0 + st));
        };
        // S(t + NSB) goes over P(t), right behind the product that reads it (products are carried out in order)
        for (uint32_t t = 0; t < NSB && t < n && ok; ++t) issue_s(t);
        for (uint32_t t = 0; t < n && ok; ++t) {
            issue_pv(t);
            if (ok && t + NSB < n) issue_s(t + NSB);
        }
        umma_commit_by(leader, bar(done));
        if (!ok) s_ctl[1] = 1u;
    } else if constexpr (FP8) {
        // ================= K / V rows: widen, place, fetch the tile after next ===============================
        auto place = [&](uint32_t it, uint4 (&from)[NP]) {
            const uint32_t ns = is_v ? NV : NK, st = (is_v ? NK : 0u) + it % ns;
            if (it >= ns && !__all_sync(0xffffffffu, mbar_wait(bar(free0 + st), (it / ns - 1u) & 1u))) { ok = false; return; }
            uint8_t *const dst = sm + T::Q + st * T::STAGE + (pc >> 2) * SLAB_KV + pr * 128u;
#pragma unroll
            for (uint32_t i = 0; i < NP; ++i) {
                if (pr + STEP * i >= uint32_t(BN)) continue;
                const uint32_t w[4] = {from[i].x, from[i].y, from[i].z, from[i].w};
                uint32_t h[8];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const __half2 lo = e4m3x2_to_half2(w[j] & 0xffffu), hi = e4m3x2_to_half2(w[j] >> 16);
                    h[2 * j] = *reinterpret_cast<const uint32_t *>(&lo);
                    h[2 * j + 1] = *reinterpret_cast<const uint32_t *>(&hi);
                }
                // 16-byte chunks 2 pc and 2 pc + 1 of the row (chunk_off)
                const uint32_t at = ((2u * pc) & 7u) ^ ((pr + STEP * i) & 7u);
                uint8_t *const d = dst + i * STEP * 128u;
                *reinterpret_cast<uint4 *>(d + (at << 4)) = make_uint4(h[0], h[1], h[2], h[3]);
                *reinterpret_cast<uint4 *>(d + ((at ^ 1u) << 4)) = make_uint4(h[4], h[5], h[6], h[7]);
            }
            fetch(it + 2u, from);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0u) mbar_arrive(bar(full0 + st));
        };
        if constexpr (D == 256) fetch(1u, raw[1]);
        for (uint32_t it = 0; it < n_tiles && ok; it += 2u) {
            place(it, raw[0]);
            if (ok && it + 1u < n_tiles) place(it + 1u, raw[1]);
        }
        if (!ok) s_ctl[1] = 1u;
    } else if (tid == 288u || tid == 320u) {
        // ================= K (one thread) and V rows (another) by TMA, behind the stages filled above ==========
        uint32_t it = ns_tma;
        for (; it < n_tiles; ++it) {
            if (!mbar_wait(bar(free0 + first_tma + it % ns_tma), (it / ns_tma - 1u) & 1u)) { ok = false; break; }
            copy_rows(it);
        }
        if (!ok) {                             // leave nothing in flight: the last copies into every stage have landed
            s_ctl[1] = 1u;
            for (uint32_t i = it - ns_tma; i < it; ++i) mbar_wait(bar(full0 + first_tma + i % ns_tma), (i / ns_tma) & 1u);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (s_ctl[1] != 0u && tid == 0) atomicOr(op.status, 1u);
    if (warp == 8u) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "n"(T::TMEM) : "memory");
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
// pays t0 once and t1 a tile (measured, in us: F16 rows of 64 / 128 / 256 dims 0.45 / 0.55 / 1.2, the last with Q in two terms;
// FP8 0.65 / 0.85 / 1.05, scaled FP8 1.3 of 128), pieces cost a second launch and their traffic.
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
    const double t1 = (dtype == VFKV_F8 ? (D == 256 ? 1.05 : D == 128 ? 0.85 : 0.65) : (D == 256 ? 1.2 : D == 128 ? 0.55 : 0.45)) +
                      (sc ? (D == 256 ? 0.9 : 0.45) : split_q && D == 128 ? 0.06 : 0.0) + (p.softcap > 0.f ? 0.25 : 0.0);
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
    cudaError_t e = launch_dependent(ctx, kern, dim3(op.n_split * p.n_kv_heads * op.n_rb), dim3(kThreads<DT>), T::SMEM, st, op, tm_k, tm_v);
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
