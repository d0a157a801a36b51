// Chunked-prefill causal attention with f32 operands and accumulation on CUDA cores: F32 caches, FP8
// caches with a scale per (position, kv-head), head_dim 512 and group sizes that the tensor-core
// kernels do not tile.  (Those feed Q and P as half-precision values; these callers have f32 results.)
//
// Work split: CTA = 64 rows = (64 / g) consecutive queries x the g q-heads of one kv-head, so a K/V
// tile of 64 positions is fetched and widened to f32 once per 64 rows.  A warp owns 8 rows from the
// scores to the output: scores, maxima, P and O never leave it, and the only CTA-wide step is the
// hand-over of the next 16 KB piece of K or V (double-buffered in shared memory, the piece after it
// in flight in registers).
//   S: thread = 4 rows x 4 positions; 8 16-byte shared loads for 64 FMAs.
//   PV: thread = 8 rows x 4 dims; 3 16-byte shared loads for 32 FMAs.
// No pipe is full (shared-memory wavefronts 48 %, FMA pipe 46 %, issue slots 61 %); a 16-byte load of a warp takes four
// shared-memory cycles whoever shares an address, so the thread's tile of S is square: 2 x 8, with ten loads for the
// same FMAs, took 90.5 us where this took 84.6 (200 queries at 700 positions, F32).
//
// A score's products are summed two at a time (fma.rn.f32x2: the even and the odd dims) in chains of sixteen.  In one chain
// of head_dim products (85.5 us) a result was 4.8e-7 off against 64 bits, and 2.4e-6 with scores of 100; in chains of sixteen 3.1e-7
// and 8.4e-7 (88.4 us, one product an instruction; 84.2 with two), in chains of four 3.5e-7 and 1.3e-6 (91.7).  The same for P V,
// which has to pair values up first, gained nothing (84.6).
//
// Row blocks are few and uneven (200 queries x 4 heads x 8 kv-heads: 104 blocks of 8 to 11 tiles), and an SM is
// at its rate only with two CTAs on it, so the tiles of all (row block, kv-head) items form one line of which every
// resident CTA takes an even share.  An item that a share ends in goes to scratch in pieces, which a second kernel
// puts together.  200 queries at 700 positions, F32: 119 us with a CTA or a cluster of two an item, whose second
// CTAs sat on 60 of 148 SMs; 85 in even shares (in one chain a score).  Sixteen rows a warp, four warps a CTA (fewer shared loads a product)
// were faster only from about 1000 positions on (200 at 1500: 153 against 160; 368 at 368: 84 against 76).
#include "fp8_codec.cuh"
#include "prefill_params.cuh"
#include "softcap.cuh"

#include <atomic>

namespace vfkv {
namespace {

constexpr float kLog2e = 1.4426950408889634f;
constexpr int BM = 64, BN = 64;           // rows per CTA, positions per tile
constexpr int kWarps = 8, kThreads = kWarps * 32;
constexpr int WR = BM / kWarps, HR = 4;           // rows of a warp, and of a thread in S
constexpr int LR = 32 / (WR / HR), HP = BN / LR;  // lanes that share a row of S, and positions of each
constexpr int CHAIN = 32;                 // products of a score in two chains before they go onto its sum
constexpr int kPiece = 4096;              // elements of a piece of K ([64 positions][64 dims]) or V ([VP][CW])
constexpr int kPitchK = 68;               // floats per K row: 16-byte units of consecutive rows fall into different banks

template <int D> struct F32Shape {
    static constexpr int CW = D < 128 ? D : 128;     // dims of a V piece
    static constexpr int VP = kPiece / CW;           // positions of a V piece
    static constexpr int NK = D / 64;                // K pieces per tile; as many V pieces
    static constexpr int CB = D / CW;                // column blocks of O
    static constexpr int LC = CW / 32;               // dims of a column block per lane
    static constexpr int PITCH_Q = D + 4;
    static constexpr int Q_BYTES = BM * PITCH_Q * 4;
    static constexpr int BUF_BYTES = BN * kPitchK * 4;
    static constexpr int P_BYTES = BM * BN * 4;
    static constexpr int SMEM = Q_BYTES + 2 * BUF_BYTES + P_BYTES;
    static constexpr int PIECE = BM * (D + 2);       // floats of a piece: O, then the rows' maxima, then their sums
};

__device__ __forceinline__ float fast_exp2(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Two f32 in one register pair, an operation on both at a time.
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b)
{
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ float lo2(uint64_t a) { return __uint_as_float(uint32_t(a)); }
__device__ __forceinline__ float hi2(uint64_t a) { return __uint_as_float(uint32_t(a >> 32)); }

// One thread's share of a piece as it lies in the cache.
template <int DT> struct Raw { uint4 w[kPiece / kThreads / (DT == VFKV_F32 ? 4 : DT == VFKV_F16 ? 8 : 16)]; };

// Unit u of a piece with `cols` elements a row: a unit is 16 bytes of one row.
template <int DT> struct Unit { static constexpr int ELEMS = DT == VFKV_F32 ? 4 : DT == VFKV_F16 ? 8 : 16; };

template <int DT>
__device__ __forceinline__ void widen(const uint4 &w, float scale, float *x)
{
    const uint32_t r[4] = {w.x, w.y, w.z, w.w};
    if constexpr (DT == VFKV_F32) {
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = __uint_as_float(r[i]);
    } else if constexpr (DT == VFKV_F16) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&r[i]));
            x[2 * i] = f.x; x[2 * i + 1] = f.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 a = e4m3x2_to_float2(r[i] & 0xffffu), b = e4m3x2_to_float2(r[i] >> 16);
            x[4 * i] = a.x * scale; x[4 * i + 1] = a.y * scale; x[4 * i + 2] = b.x * scale; x[4 * i + 3] = b.y * scale;
        }
    }
}

// The line of tiles: items in the order (row block, kv-head); CTA c takes tiles [share(c), share(c + 1)).
struct F32Params {
    PrefillParams a;
    uint32_t n_rb, n_cta, each, rest;         // CTAs below `rest` take each + 1 tiles, the others `each`
    float *scratch;                   // [n_cta][2] pieces: an item begun by an earlier CTA, an item left to the next;
                                      // null: a CTA for each item
};
__device__ __forceinline__ uint32_t share(const F32Params &p, uint32_t c) { return c * p.each + min(c, p.rest); }
__device__ __forceinline__ uint32_t owner(const F32Params &p, uint32_t tile)
{
    const uint32_t longer = p.rest * (p.each + 1u);
    return tile < longer ? tile / (p.each + 1u) : p.rest + (tile - longer) / p.each;
}
// Positions row block rb sees, [*lo, *hi), and its tiles: at least one, so that rows without a position are written.
__host__ __device__ __forceinline__ uint32_t block_tiles(const PrefillParams &p, uint32_t rb, uint32_t *lo, uint32_t *hi)
{
    uint32_t qb = (rb * BM + BM - 1) / p.group, lo_b, hi_a;
    if (qb >= p.m) qb = p.m - 1;
    query_range(p, rb * BM / p.group, lo, &hi_a);                  // ranges are monotone in the query index
    query_range(p, qb, &lo_b, hi);
    return *hi > *lo ? (*hi + BN - 1) / BN - *lo / BN : 1u;
}

template <int DT, int D>
__global__ void __launch_bounds__(kThreads, D <= 128 ? 2 : 1) prefill_f32_kernel(const F32Params fp)
{
    const PrefillParams &p = fp.a;
    using S = F32Shape<D>;
    constexpr int UE = Unit<DT>::ELEMS, NU = kPiece / kThreads / UE, ES = DT == VFKV_F32 ? 4 : DT == VFKV_F16 ? 2 : 1;
    extern __shared__ __align__(16) float sm[];
    float *const sq = sm;                                          // [64][PITCH_Q]
    float *const sbuf = sq + BM * S::PITCH_Q;                      // [2][64 * 68]
    float *const sp = sbuf + 2 * BN * kPitchK;                     // [warp][position][8 rows]
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t g = p.group, n_rows = p.m * g;
    const uint32_t rp = lane / LR * HR, cl = lane % LR;            // first of the thread's HR rows of the warp, first position
    const float q_mult = p.scale * (p.softcap > 0.f ? 1.0f : kLog2e);      // into the log2 domain; after a soft-cap if there is one
    float *const my_p = sp + warp * BN * WR;
    uint32_t line = fp.scratch ? share(fp, blockIdx.x) : 0u;
    const uint32_t line_end = fp.scratch ? share(fp, blockIdx.x + 1u) : 1u;
    pdl_wait();

    while (line < line_end) {
    // ---- the item that tile `line` belongs to, and how much of it is this CTA's ----
    uint32_t rb = blockIdx.x / p.n_kv_heads, kvh = blockIdx.x % p.n_kv_heads, n_item = 0u, off = 0u, c_lo, c_hi;
    for (uint32_t base = 0, before = 0; fp.scratch != nullptr; base += 32) {
        uint32_t lo, hi;
        const uint32_t n = base + lane < fp.n_rb ? block_tiles(p, base + lane, &lo, &hi) : 0u;
        uint32_t x = n * p.n_kv_heads;
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        const uint32_t here = __ballot_sync(0xffffffffu, before + x > line);
        if (here != 0u || base + 32 >= fp.n_rb) {
            const int k = here != 0u ? __ffs(here) - 1 : 0;
            n_item = __shfl_sync(0xffffffffu, n, k);
            const uint32_t rel = line - before - (__shfl_sync(0xffffffffu, x, k) - n_item * p.n_kv_heads);
            rb = base + uint32_t(k); kvh = rel / n_item; off = rel % n_item;
            break;
        }
        before += __shfl_sync(0xffffffffu, x, 31);
    }
    const uint32_t n_all = block_tiles(p, rb, &c_lo, &c_hi);
    if (fp.scratch == nullptr) n_item = n_all;
    const uint32_t row0 = rb * BM, n_mine = fp.scratch ? min(n_item - off, line_end - line) : n_item;
    const uint32_t t_begin = c_lo / BN + off, t_end = t_begin + n_mine;

    // this thread's rows in S
    uint32_t r_lo[HR], r_hi[HR], w_lo, w_hi, full_lo, full_hi;
    {
        uint32_t mx_lo = 0u, mn_hi = 0xffffffffu, mn_lo = 0xffffffffu, mx_hi = 0u;
#pragma unroll
        for (int h = 0; h < HR; ++h) {
            const uint32_t row = row0 + warp * WR + rp + h;
            r_lo[h] = r_hi[h] = 0u;
            if (row < n_rows) {
                query_range(p, row / g, &r_lo[h], &r_hi[h]);
                mn_lo = min(mn_lo, r_lo[h]); mx_hi = max(mx_hi, r_hi[h]);
                mx_lo = max(mx_lo, r_lo[h]); mn_hi = min(mn_hi, r_hi[h]);
            }                                                      // rows past the end: whatever, they are not written
        }
        w_lo = __reduce_min_sync(0xffffffffu, mn_lo); w_hi = __reduce_max_sync(0xffffffffu, mx_hi);
        full_lo = __reduce_max_sync(0xffffffffu, mx_lo); full_hi = __reduce_min_sync(0xffffffffu, mn_hi);
    }

    const uint8_t *const kg = p.k + uint64_t(kvh) * D * ES, *const vg = p.v + uint64_t(kvh) * D * ES;
    Raw<DT> raw;
    float raw_scale[NU];
    // piece c of tile t into registers: K pieces 0 .. NK-1 (64 dims each), then V pieces (position block, column block)
    auto fetch = [&](uint32_t t, int c) {
        const bool is_v = c >= S::NK;
        const int cols = is_v ? S::CW : 64, vi = c - S::NK;
        const uint32_t first_pos = t * BN + (is_v ? uint32_t(vi / S::CB) * S::VP : 0u);
        const uint32_t first_col = is_v ? uint32_t(vi % S::CB) * S::CW : uint32_t(c) * 64u;
#pragma unroll
        for (int i = 0; i < NU; ++i) {
            const uint32_t u = threadIdx.x + i * kThreads, r = u / (cols / UE), e = (u % (cols / UE)) * UE;
            const uint32_t pos = first_pos + r;
            const bool ok = pos >= c_lo && pos < c_hi;             // nothing outside the block's range is read
            raw.w[i] = ok ? *reinterpret_cast<const uint4 *>((is_v ? vg : kg) + uint64_t(pos) * p.row_bytes + uint64_t(first_col + e) * ES)
                          : make_uint4(0u, 0u, 0u, 0u);
            raw_scale[i] = 1.f;
            if constexpr (DT == VFKV_F8) {
                const float *sc = is_v ? p.v_scales : p.k_scales;
                if (sc && ok) raw_scale[i] = sc[uint64_t(pos) * p.n_kv_heads + kvh];
            }
        }
    };
    auto place = [&](int c) {
        const bool is_v = c >= S::NK;
        const int cols = is_v ? S::CW : 64, pitch = is_v ? S::CW : kPitchK;
        float *const dst = sbuf + (c & 1) * BN * kPitchK;
#pragma unroll
        for (int i = 0; i < NU; ++i) {
            const uint32_t u = threadIdx.x + i * kThreads, r = u / (cols / UE), e = (u % (cols / UE)) * UE;
            float x[UE];
            widen<DT>(raw.w[i], raw_scale[i], x);
#pragma unroll
            for (int j = 0; j < UE; j += 4)
                *reinterpret_cast<float4 *>(dst + r * pitch + e + j) = make_float4(x[j], x[j + 1], x[j + 2], x[j + 3]);
        }
    };

    float acc[S::CB][WR][S::LC];
#pragma unroll
    for (int b = 0; b < S::CB; ++b)
#pragma unroll
        for (int r = 0; r < WR; ++r)
#pragma unroll
            for (int j = 0; j < S::LC; ++j) acc[b][r][j] = 0.f;
    float m_run[HR], l_run[HR];
#pragma unroll
    for (int h = 0; h < HR; ++h) { m_run[h] = kMaskedScore; l_run[h] = 0.f; }
    fetch(t_begin, 0);
    // Q rows, scaled
    __syncthreads();                                               // the item before is done with its own
    for (uint32_t i = threadIdx.x; i < uint32_t(BM * D / 4); i += kThreads) {
        const uint32_t r = i / (D / 4), c = i % (D / 4), row = row0 + r;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row < n_rows)
            x = *reinterpret_cast<const float4 *>(p.q + (uint64_t(row / g) * p.n_q_heads + kvh * g + row % g) * D + 4 * c);
        *reinterpret_cast<float4 *>(sq + r * S::PITCH_Q + 4 * c) = make_float4(x.x * q_mult, x.y * q_mult, x.z * q_mult, x.w * q_mult);
    }
    for (uint32_t t = t_begin; t < t_end; ++t) {
        const uint32_t t0 = t * BN;
        const bool live = t0 < w_hi && t0 + BN > w_lo;             // some row of this warp sees some of the tile
        const bool full = t0 >= full_lo && t0 + BN <= full_hi;
        float s[HR][HP];
#pragma unroll
        for (int h = 0; h < HR; ++h)
#pragma unroll
            for (int j = 0; j < HP; ++j) s[h][j] = 0.f;
#pragma unroll
        for (int c = 0; c < S::NK; ++c) {                          // S = Q K^T, 64 dims at a time
            place(c);
            __syncthreads();
            fetch(t, c + 1);
            if (live) {
                const float *const qa = sq + (warp * WR + rp) * S::PITCH_Q + c * 64, *const ka = sbuf + (c & 1) * BN * kPitchK + cl * kPitchK;
#pragma unroll 1
                for (int k0 = 0; k0 < 64; k0 += CHAIN) {           // two chains of CHAIN / 2 products each: a shorter one loses less
                    uint64_t part[HR][HP];
#pragma unroll
                    for (int k = k0; k < k0 + CHAIN; k += 4) {
                        ulonglong2 qv[HR];
#pragma unroll
                        for (int h = 0; h < HR; ++h) qv[h] = *reinterpret_cast<const ulonglong2 *>(qa + h * S::PITCH_Q + k);
#pragma unroll
                        for (int j = 0; j < HP; ++j) {
                            const ulonglong2 kv = *reinterpret_cast<const ulonglong2 *>(ka + j * LR * kPitchK + k);
#pragma unroll
                            for (int h = 0; h < HR; ++h) {
                                part[h][j] = k == k0 ? mul2(qv[h].x, kv.x) : fma2(qv[h].x, kv.x, part[h][j]);
                                part[h][j] = fma2(qv[h].y, kv.y, part[h][j]);
                            }
                        }
                    }
#pragma unroll
                    for (int h = 0; h < HR; ++h)
#pragma unroll
                        for (int j = 0; j < HP; ++j) s[h][j] += lo2(part[h][j]) + hi2(part[h][j]);
                }
            }
        }
        if (live) {                                                // masks, online softmax, P to the warp's buffer
            float corr[HR];
            bool moved = false;
#pragma unroll
            for (int h = 0; h < HR; ++h) {
                float mx = kMaskedScore;
                if (p.softcap > 0.f) {
                    softcap_all(s[h], p.softcap, 1.0f / p.softcap);
#pragma unroll
                    for (int j = 0; j < HP; ++j) s[h][j] *= kLog2e;
                }
#pragma unroll
                for (int j = 0; j < HP; ++j) {
                    float x = s[h][j];
                    const uint32_t pos = t0 + cl + LR * j;
                    if (!full && (pos < r_lo[h] || pos >= r_hi[h])) x = kMaskedScore;
                    s[h][j] = x;
                    mx = fmaxf(mx, x);
                }
#pragma unroll
                for (int o = 1; o < LR; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                const float mn = fmaxf(m_run[h], mx);
                corr[h] = fast_exp2(m_run[h] - mn);
                moved |= corr[h] != 1.f;
                m_run[h] = mn;
                float sum = 0.f;
#pragma unroll
                for (int j = 0; j < HP; ++j) {
                    // a masked position contributes nothing, also while the row's maximum is still the sentinel; a NaN stays one
                    const float e = (full || !(s[h][j] <= 0.5f * kMaskedScore)) ? fast_exp2(s[h][j] - mn) : 0.f;
                    s[h][j] = e;
                    sum += e;
                }
                l_run[h] = l_run[h] * corr[h] + sum;               // this lane's positions; summed over lanes at the end
            }
#pragma unroll
            for (int j = 0; j < HP; ++j) {
                float *const d = my_p + (cl + LR * j) * WR + rp;
                *reinterpret_cast<float4 *>(d) = make_float4(s[0][j], s[1][j], s[2][j], s[3][j]);
            }
            if (__any_sync(0xffffffffu, moved)) {
#pragma unroll
                for (int r = 0; r < WR; ++r) {
                    const float f = __shfl_sync(0xffffffffu, corr[r % HR], r / HR * LR);
#pragma unroll
                    for (int b = 0; b < S::CB; ++b)
#pragma unroll
                        for (int j = 0; j < S::LC; ++j) acc[b][r][j] *= f;
                }
            }
            __syncwarp();
        }
#pragma unroll
        for (int vi = 0; vi < S::NK; ++vi) {                       // O += P V, one piece at a time
            const int c = S::NK + vi, pb = vi / S::CB, cb = vi % S::CB;
            place(c);
            __syncthreads();
            if (vi + 1 < S::NK) fetch(t, c + 1);
            else if (t + 1 < t_end) fetch(t + 1, 0);
            if (live) {
                const float *const va = sbuf + (c & 1) * BN * kPitchK + lane * S::LC, *const pa = my_p + pb * S::VP * WR;
                auto step = [&](int i, bool masked) {
                    float v[S::LC];
                    if constexpr (S::LC == 4) {
                        const float4 x = *reinterpret_cast<const float4 *>(va + i * S::CW);
                        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
                    } else {
                        const float2 x = *reinterpret_cast<const float2 *>(va + i * S::CW);
                        v[0] = x.x; v[1] = x.y;
                    }
                    float pr[WR];
#pragma unroll
                    for (int r = 0; r < WR; r += 4) {
                        const float4 x = *reinterpret_cast<const float4 *>(pa + i * WR + r);
                        pr[r] = x.x; pr[r + 1] = x.y; pr[r + 2] = x.z; pr[r + 3] = x.w;
                    }
#pragma unroll
                    for (int r = 0; r < WR; ++r)
#pragma unroll
                        for (int j = 0; j < S::LC; ++j)
                            // a row that does not see a position takes nothing from it, not even 0 x infinity
                            acc[cb][r][j] = masked && pr[r] == 0.f ? acc[cb][r][j] : fmaf(pr[r], v[j], acc[cb][r][j]);
                };
                // the piece's positions that some row of the warp sees, and those that all of them see
                const int first = int(t0) + pb * S::VP;
                const int lo = max(int(w_lo) - first, 0), hi = min(int(w_hi) - first, S::VP);
                const int all_lo = min(max(int(full_lo) - first, lo), hi), all_hi = max(min(int(full_hi) - first, hi), all_lo);
                if (lo == 0 && all_lo == 0 && all_hi == S::VP) {
#pragma unroll 8
                    for (int i = 0; i < S::VP; ++i) step(i, false);
                } else {
#pragma unroll 1
                    for (int i = lo; i < all_lo; ++i) step(i, true);
#pragma unroll 1
                    for (int i = all_lo; i < all_hi; ++i) step(i, false);
#pragma unroll 1
                    for (int i = all_hi; i < hi; ++i) step(i, true);
                }
            }
        }
        __syncwarp();                                              // P is read before the next tile's is written
    }

    // row sums over the eight lanes that share a row
#pragma unroll
    for (int h = 0; h < HR; ++h)
#pragma unroll
        for (int o = 1; o < LR; o <<= 1) l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], o);

    if (n_mine == n_item) {
#pragma unroll
        for (int r = 0; r < WR; ++r) {
            const float l = __shfl_sync(0xffffffffu, l_run[r % HR], r / HR * LR);
            const uint32_t row = row0 + warp * WR + r;
            if (row >= n_rows) continue;
            const float inv = l > 0.f ? 1.0f / l : 0.f;            // an empty range yields zeros
            float *o = p.out + (uint64_t(row / g) * p.n_q_heads + kvh * g + row % g) * D + lane * S::LC;
#pragma unroll
            for (int b = 0; b < S::CB; ++b) {
                if constexpr (S::LC == 4)
                    *reinterpret_cast<float4 *>(o + b * S::CW) = make_float4(acc[b][r][0] * inv, acc[b][r][1] * inv, acc[b][r][2] * inv, acc[b][r][3] * inv);
                else
                    *reinterpret_cast<float2 *>(o + b * S::CW) = make_float2(acc[b][r][0] * inv, acc[b][r][1] * inv);
            }
        }
    } else {
        float *const o = fp.scratch + (uint64_t(blockIdx.x) * 2 + (off == 0u ? 1 : 0)) * S::PIECE;
#pragma unroll
        for (int r = 0; r < WR; ++r)
#pragma unroll
            for (int b = 0; b < S::CB; ++b) {
                float *const d = o + (warp * WR + r) * D + b * S::CW + lane * S::LC;
                if constexpr (S::LC == 4) *reinterpret_cast<float4 *>(d) = make_float4(acc[b][r][0], acc[b][r][1], acc[b][r][2], acc[b][r][3]);
                else *reinterpret_cast<float2 *>(d) = make_float2(acc[b][r][0], acc[b][r][1]);
            }
        if (cl == 0u) {
#pragma unroll
            for (int h = 0; h < HR; ++h) {
                o[BM * D + warp * WR + rp + h] = m_run[h];
                o[BM * D + BM + warp * WR + rp + h] = l_run[h];
            }
        }
    }
    line += n_mine;
    }
}

// The items that were cut, put together: a warp per row, four pieces at a time.  grid = (items, groups of eight rows).
template <int D>
__global__ void __launch_bounds__(kThreads) prefill_f32_merge_kernel(const F32Params fp)
{
    using S = F32Shape<D>;
    constexpr int NV = D < 128 ? 1 : D / 128, LANES = D / 4 < 32 ? D / 4 : 32, U = 4;
    const PrefillParams &p = fp.a;
    pdl_wait();
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = p.group;
    const uint32_t rb = blockIdx.x / p.n_kv_heads, kvh = blockIdx.x % p.n_kv_heads;
    uint32_t before = 0, lo, hi;
    for (uint32_t r = lane; r < rb; r += 32) before += block_tiles(p, r, &lo, &hi);
    before = __reduce_add_sync(0xffffffffu, before);
    const uint32_t n = block_tiles(p, rb, &lo, &hi), begin = before * p.n_kv_heads + kvh * n;
    const uint32_t c0 = owner(fp, begin), n_pieces = owner(fp, begin + n - 1u) - c0 + 1u;
    if (n_pieces == 1u) return;                                    // one CTA had all of it
    auto piece = [&](uint32_t i) {                                 // the first piece lies in its CTA's second place
        i = min(i, n_pieces - 1u);
        return fp.scratch + (uint64_t(c0 + i) * 2 + (i == 0u ? 1 : 0)) * S::PIECE;
    };
    const uint32_t rl = blockIdx.y * (kThreads / 32) + warp, row = rb * BM + rl;
    if (row >= p.m * g) return;
    float M = kMaskedScore;
    for (uint32_t i = lane; i < n_pieces; i += 32) M = fmaxf(M, __ldcg(piece(i) + BM * D + rl));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
    float L = 0.f;
    float4 acc[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[v] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t i0 = 0; i0 < n_pieces; i0 += U) {
        float4 x[U][NV];
        float f[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const float *const o = piece(i0 + u);
            f[u] = i0 + u < n_pieces ? fast_exp2(__ldcg(o + BM * D + rl) - M) : 0.f;
            L = fmaf(f[u], __ldcg(o + BM * D + BM + rl), L);
#pragma unroll
            for (int v = 0; v < NV; ++v) x[u][v] = __ldcg(reinterpret_cast<const float4 *>(o + rl * D) + lane % LANES + 32 * v);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                acc[v].x = fmaf(f[u], x[u][v].x, acc[v].x); acc[v].y = fmaf(f[u], x[u][v].y, acc[v].y);
                acc[v].z = fmaf(f[u], x[u][v].z, acc[v].z); acc[v].w = fmaf(f[u], x[u][v].w, acc[v].w);
            }
    }
    const float inv = L > 0.f ? 1.0f / L : 0.f;                // an empty range yields zeros
    if (lane < uint32_t(LANES)) {
        float4 *const out = reinterpret_cast<float4 *>(p.out + (uint64_t(row / g) * p.n_q_heads + kvh * g + row % g) * D) + lane;
#pragma unroll
        for (int v = 0; v < NV; ++v) out[32 * v] = make_float4(acc[v].x * inv, acc[v].y * inv, acc[v].z * inv, acc[v].w * inv);
    }
}

template <int DT, int D>
int32_t launch_t(vfkv_ctx *ctx, const PrefillParams &p, cudaStream_t st)
{
    using S = F32Shape<D>;
    auto kern = prefill_f32_kernel<DT, D>;
    static std::atomic<bool> configured[64];
    if (!configured[ctx->device & 63].load(std::memory_order_acquire)) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM);
        if (e != cudaSuccess) return check_cuda(ctx, e, "cudaFuncSetAttribute(f32 prefill attention)");
        configured[ctx->device & 63].store(true, std::memory_order_release);
    }
    F32Params fp{};
    fp.a = p;
    fp.n_rb = uint32_t((uint64_t(p.m) * p.group + BM - 1) / BM);
    uint64_t total = 0;
    for (uint32_t rb = 0; rb < fp.n_rb; ++rb) {
        uint32_t lo, hi;
        total += uint64_t(block_tiles(p, rb, &lo, &hi)) * p.n_kv_heads;
    }
    if (total >= (1ull << 31)) return set_error(ctx, VFKV_ERR_UNSUPPORTED, "f32 prefill attention: too many tiles in a call");
    const uint64_t items = uint64_t(fp.n_rb) * p.n_kv_heads, slots = uint64_t(ctx->sm_count) * (D <= 128 ? 2 : 1);
    fp.n_cta = uint32_t(total < slots ? total : slots);
    fp.each = uint32_t(total) / fp.n_cta;
    fp.rest = uint32_t(total) % fp.n_cta;
    uint64_t floats = 0;
    fp.scratch = prefill_scratch(ctx, st, &floats);
    if (floats < uint64_t(fp.n_cta) * 2 * S::PIECE) fp.scratch = nullptr;
    cudaError_t e = launch_dependent(ctx, kern, dim3(fp.scratch ? fp.n_cta : uint32_t(items)), dim3(kThreads), S::SMEM, st, fp);
    ctx->count_launch();
    if (e == cudaSuccess && fp.scratch && fp.n_cta > 1) {
        e = launch_dependent(ctx, prefill_f32_merge_kernel<D>, dim3(uint32_t(items), BM / (kThreads / 32)), dim3(kThreads), 0, st, fp);
        ctx->count_launch();
    }
    prefill_scratch_used(ctx, st, fp.scratch);
    return check_cuda(ctx, e, "f32 prefill attention launch");
}

template <int DT>
int32_t launch_d(vfkv_ctx *ctx, const PrefillParams &p, cudaStream_t st)
{
    switch (p.head_dim) {
    case 64: return launch_t<DT, 64>(ctx, p, st);
    case 128: return launch_t<DT, 128>(ctx, p, st);
    case 256: return launch_t<DT, 256>(ctx, p, st);
    default: return launch_t<DT, 512>(ctx, p, st);
    }
}

}  // namespace

bool prefill_f32_supported(uint32_t D) { return D == 64 || D == 128 || D == 256 || D == 512; }

int32_t launch_prefill_f32(vfkv_ctx *ctx, uint32_t dtype, const PrefillParams &p, cudaStream_t st)
{
    switch (dtype) {
    case VFKV_F32: return launch_d<VFKV_F32>(ctx, p, st);
    case VFKV_F16: return launch_d<VFKV_F16>(ctx, p, st);
    default: return launch_d<VFKV_F8>(ctx, p, st);
    }
}

}  // namespace vfkv
