// Chunked-prefill causal attention with f32 operands and accumulation on CUDA cores: F32 caches, FP8
// caches with a scale per (position, kv-head), head_dim 512 and group sizes that the tensor-core
// kernels do not tile.  (Those feed Q and P as half-precision values; these callers have f32 results.)
//
// Work split: CTA = 64 rows = (64 / g) consecutive queries x the g q-heads of one kv-head, so a K/V
// tile of 64 positions is fetched and widened to f32 once per 64 rows.  A warp owns 8 rows from the
// scores to the output: scores, maxima, P and O never leave it, and the only CTA-wide step is the
// hand-over of the next 16 KB piece of K or V (double-buffered in shared memory, the piece after it
// in flight in registers).
//   S: thread = 2 rows x 8 positions; 10 16-byte shared loads for 64 FMAs.
//   PV: thread = 8 rows x 4 dims; 3 16-byte shared loads for 32 FMAs.
// Both keep the FMA pipe, not shared memory, as the bound (74 TFLOP/s at 1.96 GHz).
//
// A chunk of a short prompt has few row blocks (200 queries x 4 heads x 8 kv-heads: 104), so the K/V
// tiles of a block may be cut over a cluster of 2, 4 or 8 CTAs, which merge their (m, l, O) through
// distributed shared memory: no scratch, no second launch.
#include "fp8_codec.cuh"
#include "prefill_params.cuh"
#include "softcap.cuh"

#include <atomic>

namespace vfkv {
namespace {

constexpr float kLog2e = 1.4426950408889634f;
constexpr int BM = 64, BN = 64;           // rows per CTA, positions per tile
constexpr int kWarps = 8, kThreads = kWarps * 32;
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
    static constexpr int P_BYTES = kWarps * BN * 8 * 4;
    static constexpr int SMEM = Q_BYTES + 2 * BUF_BYTES + P_BYTES;
};

__device__ __forceinline__ float fast_exp2(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// One thread's share of a piece as it lies in the cache: 16 elements.
template <int DT> struct Raw { uint4 w[DT == VFKV_F32 ? 4 : DT == VFKV_F16 ? 2 : 1]; };

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

template <int DT, int D>
__global__ void __launch_bounds__(kThreads, D <= 128 ? 2 : 1) prefill_f32_kernel(const PrefillParams p)
{
    using S = F32Shape<D>;
    constexpr int UE = Unit<DT>::ELEMS, NU = 16 / UE, ES = DT == VFKV_F32 ? 4 : DT == VFKV_F16 ? 2 : 1;
    extern __shared__ __align__(16) float sm[];
    float *const sq = sm;                                          // [64][PITCH_Q]
    float *const sbuf = sq + BM * S::PITCH_Q;                      // [2][64 * 68]
    float *const sp = sbuf + 2 * BN * kPitchK;                     // [warp][position][8 rows]
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t split = blockIdx.x, n_splits = gridDim.x, kvh = blockIdx.z, g = p.group;
    const uint32_t row0 = (gridDim.y - 1u - blockIdx.y) * BM;      // heaviest row blocks (latest queries) first
    const uint32_t n_rows = p.m * g;

    // tiles of this row block, and this CTA's share of them
    uint32_t c_lo, c_hi, t_begin, t_end;
    {
        uint32_t qb = (row0 + BM - 1) / g, lo_b, hi_a;
        if (qb >= p.m) qb = p.m - 1;
        query_range(p, row0 / g, &c_lo, &hi_a);                    // ranges are monotone in the query index
        query_range(p, qb, &lo_b, &c_hi);
        const uint32_t first = c_lo / BN, n = c_hi > c_lo ? (c_hi + BN - 1) / BN - first : 0u;
        t_begin = first + uint32_t(uint64_t(n) * split / n_splits);
        t_end = first + uint32_t(uint64_t(n) * (split + 1) / n_splits);
    }
    pdl_wait();
    // Q rows, scaled into the log2 domain (with a soft-cap the factor is applied after it)
    const float q_mult = p.scale * (p.softcap > 0.f ? 1.0f : kLog2e);
    for (uint32_t i = threadIdx.x; i < uint32_t(BM * D / 4); i += kThreads) {
        const uint32_t r = i / (D / 4), c = i % (D / 4), row = row0 + r;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row < n_rows)
            x = *reinterpret_cast<const float4 *>(p.q + (uint64_t(row / g) * p.n_q_heads + kvh * g + row % g) * D + 4 * c);
        *reinterpret_cast<float4 *>(sq + r * S::PITCH_Q + 4 * c) = make_float4(x.x * q_mult, x.y * q_mult, x.z * q_mult, x.w * q_mult);
    }
    // this thread's two rows in S
    const uint32_t rp = (lane >> 3) * 2, cl = lane & 7;            // row pair of the warp's 8 rows, first position
    uint32_t r_lo[2], r_hi[2], w_lo, w_hi, full_lo, full_hi;
    {
        uint32_t mx_lo = 0u, mn_hi = 0xffffffffu, mn_lo = 0xffffffffu, mx_hi = 0u;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t row = row0 + warp * 8 + rp + h;
            r_lo[h] = r_hi[h] = 0u;
            if (row < n_rows) {
                query_range(p, row / g, &r_lo[h], &r_hi[h]);
                mn_lo = min(mn_lo, r_lo[h]); mx_hi = max(mx_hi, r_hi[h]);
                mx_lo = max(mx_lo, r_lo[h]); mn_hi = min(mn_hi, r_hi[h]);
            } else {
                mn_hi = 0u;                                        // rows past the end: always masked
            }
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

    float acc[S::CB][8][S::LC];
#pragma unroll
    for (int b = 0; b < S::CB; ++b)
#pragma unroll
        for (int r = 0; r < 8; ++r)
#pragma unroll
            for (int j = 0; j < S::LC; ++j) acc[b][r][j] = 0.f;
    float m_run[2] = {kMaskedScore, kMaskedScore}, l_run[2] = {0.f, 0.f};
    float *const my_p = sp + warp * BN * 8;

    if (t_begin < t_end) fetch(t_begin, 0);
    for (uint32_t t = t_begin; t < t_end; ++t) {
        const uint32_t t0 = t * BN;
        const bool live = t0 < w_hi && t0 + BN > w_lo;             // some row of this warp sees some of the tile
        const bool full = t0 >= full_lo && t0 + BN <= full_hi;
        float s[2][8];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int j = 0; j < 8; ++j) s[h][j] = 0.f;
#pragma unroll
        for (int c = 0; c < S::NK; ++c) {                          // S = Q K^T, 64 dims at a time
            place(c);
            __syncthreads();
            fetch(t, c + 1);
            if (live) {
                const float *const qa = sq + (warp * 8 + rp) * S::PITCH_Q + c * 64, *const ka = sbuf + (c & 1) * BN * kPitchK + cl * kPitchK;
#pragma unroll 4
                for (int k = 0; k < 64; k += 4) {
                    const float4 q0 = *reinterpret_cast<const float4 *>(qa + k), q1 = *reinterpret_cast<const float4 *>(qa + S::PITCH_Q + k);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float4 kv = *reinterpret_cast<const float4 *>(ka + j * 8 * kPitchK + k);
                        s[0][j] = fmaf(q0.x, kv.x, s[0][j]); s[1][j] = fmaf(q1.x, kv.x, s[1][j]);
                        s[0][j] = fmaf(q0.y, kv.y, s[0][j]); s[1][j] = fmaf(q1.y, kv.y, s[1][j]);
                        s[0][j] = fmaf(q0.z, kv.z, s[0][j]); s[1][j] = fmaf(q1.z, kv.z, s[1][j]);
                        s[0][j] = fmaf(q0.w, kv.w, s[0][j]); s[1][j] = fmaf(q1.w, kv.w, s[1][j]);
                    }
                }
            }
        }
        if (live) {                                                // masks, online softmax, P to the warp's buffer
            float corr[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float mx = kMaskedScore;
                if (p.softcap > 0.f) {
                    softcap_all(s[h], p.softcap, 1.0f / p.softcap);
#pragma unroll
                    for (int j = 0; j < 8; ++j) s[h][j] *= kLog2e;
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    float x = s[h][j];
                    const uint32_t pos = t0 + cl + 8 * j;
                    if (!full && (pos < r_lo[h] || pos >= r_hi[h])) x = kMaskedScore;
                    s[h][j] = x;
                    mx = fmaxf(mx, x);
                }
#pragma unroll
                for (int o = 1; o < 8; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                const float mn = fmaxf(m_run[h], mx);
                corr[h] = fast_exp2(m_run[h] - mn);
                m_run[h] = mn;
                float sum = 0.f;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    // a masked position contributes nothing, also while the row's maximum is still the sentinel
                    const float e = (full || s[h][j] > 0.5f * kMaskedScore) ? fast_exp2(s[h][j] - mn) : 0.f;
                    s[h][j] = e;
                    sum += e;
                }
                l_run[h] = l_run[h] * corr[h] + sum;               // this lane's positions; summed over lanes at the end
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) *reinterpret_cast<float2 *>(my_p + (cl + 8 * j) * 8 + rp) = make_float2(s[0][j], s[1][j]);
            if (__any_sync(0xffffffffu, corr[0] != 1.f || corr[1] != 1.f)) {
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    const float f = __shfl_sync(0xffffffffu, corr[r & 1], (r >> 1) << 3);
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
                const float *const va = sbuf + (c & 1) * BN * kPitchK + lane * S::LC, *const pa = my_p + pb * S::VP * 8;
                auto step = [&](int i, bool masked) {
                    float v[S::LC];
                    if constexpr (S::LC == 4) {
                        const float4 x = *reinterpret_cast<const float4 *>(va + i * S::CW);
                        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
                    } else {
                        const float2 x = *reinterpret_cast<const float2 *>(va + i * S::CW);
                        v[0] = x.x; v[1] = x.y;
                    }
                    const float4 pl = *reinterpret_cast<const float4 *>(pa + i * 8), ph = *reinterpret_cast<const float4 *>(pa + i * 8 + 4);
                    const float pr[8] = {pl.x, pl.y, pl.z, pl.w, ph.x, ph.y, ph.z, ph.w};
#pragma unroll
                    for (int r = 0; r < 8; ++r)
#pragma unroll
                        for (int j = 0; j < S::LC; ++j)
                            // a row that does not see a position takes nothing from it, not even 0 x infinity
                            acc[cb][r][j] = masked && pr[r] == 0.f ? acc[cb][r][j] : fmaf(pr[r], v[j], acc[cb][r][j]);
                };
                if (full) {
#pragma unroll 8
                    for (int i = 0; i < S::VP; ++i) step(i, false);
                } else {
#pragma unroll 2
                    for (int i = 0; i < S::VP; ++i) step(i, true);
                }
            }
        }
        __syncwarp();                                              // P is read before the next tile's is written
    }

    // row sums over the eight lanes that share a row
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], o);

    if (n_splits == 1u) {
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const float l = __shfl_sync(0xffffffffu, l_run[r & 1], (r >> 1) << 3);
            const uint32_t row = row0 + warp * 8 + r;
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
        return;
    }

    // ---- the cluster's CTAs merge: O over Q's place, m and l over P's; CTA r writes the r-th rows ----
    __syncthreads();                                               // Q, K/V pieces and P are dead
    float *const so = sq, *const s_m = sp, *const s_l = sp + BM;
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int b = 0; b < S::CB; ++b)
#pragma unroll
            for (int j = 0; j < S::LC; ++j) so[(warp * 8 + r) * D + b * S::CW + lane * S::LC + j] = acc[b][r][j];
    if (cl == 0u) {
#pragma unroll
        for (int h = 0; h < 2; ++h) { s_m[warp * 8 + rp + h] = m_run[h]; s_l[warp * 8 + rp + h] = l_run[h]; }
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    const uint32_t rows_each = BM / n_splits;
    auto peer = [&](const float *a, uint32_t rank) {
        uint32_t addr;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(uint32_t(__cvta_generic_to_shared(a))), "r"(rank));
        return addr;
    };
    auto peer_f = [&](const float *a, uint32_t rank) {
        float x;
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(peer(a, rank)) : "memory");
        return x;
    };
    for (uint32_t i = threadIdx.x; i < rows_each * (D / 4); i += kThreads) {
        const uint32_t r = split * rows_each + i / (D / 4), c = 4 * (i % (D / 4)), row = row0 + r;
        if (row >= n_rows) continue;
        float M = kMaskedScore, L = 0.f;
        for (uint32_t k = 0; k < n_splits; ++k) M = fmaxf(M, peer_f(s_m + r, k));
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
        for (uint32_t k = 0; k < n_splits; ++k) {
            const float f = fast_exp2(peer_f(s_m + r, k) - M);
            L = fmaf(peer_f(s_l + r, k), f, L);
            float4 x;
            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                         : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w) : "r"(peer(so + r * D + c, k)) : "memory");
            o.x = fmaf(x.x, f, o.x); o.y = fmaf(x.y, f, o.y); o.z = fmaf(x.z, f, o.z); o.w = fmaf(x.w, f, o.w);
        }
        const float inv = L > 0.f ? 1.0f / L : 0.f;
        *reinterpret_cast<float4 *>(p.out + (uint64_t(row / g) * p.n_q_heads + kvh * g + row % g) * D + c) =
            make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv);
    }
    __syncthreads();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");      // a peer may still be reading this CTA's memory
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
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
    const uint32_t row_blocks = uint32_t((uint64_t(p.m) * p.group + BM - 1) / BM);
    // Cut a block's K/V tiles while that still adds CTAs to idle SMs and leaves each at least two
    // tiles: 104 blocks of up to 11 tiles take two CTAs per SM of a D <= 128 kernel in clusters of two.
    const uint64_t blocks = uint64_t(row_blocks) * p.n_kv_heads, slots = uint64_t(ctx->sm_count) * (D <= 128 ? 2 : 1);
    const uint32_t visible = p.window && p.window < p.n_kv ? p.window + BM / p.group : p.n_kv - (p.kv_start < p.n_kv ? p.kv_start : p.n_kv);
    const uint32_t tiles = (visible + BN - 1) / BN;
    uint32_t n_splits = 1;
    while (n_splits < 8 && blocks * n_splits * 2 <= slots + slots / 4 && tiles >= n_splits * 4) n_splits *= 2;
    const cudaError_t e = launch_clusters(ctx, kern, dim3(n_splits, row_blocks, p.n_kv_heads), dim3(kThreads), S::SMEM, st, n_splits, p);
    ctx->count_launch();
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
