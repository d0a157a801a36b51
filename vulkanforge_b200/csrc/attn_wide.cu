// Split-K GQA decode attention on mma.sync for the FP8 / F16 shapes whose rows the TMA-fed kernel in attn_mma.cu
// has no tiles for: head_dim 512, and 64-dim FP8 rows.  Same math as attn_generic.cu and the same partials.
//
// What bounds it is the stream of K and V.  On CUDA cores these shapes took five shuffles and D / 32 multiply-adds
// a position, head and lane: 16 q / 2 kv heads of 512, 3 sequences x 20 000 positions x 4 layers, FP8, 557 us
// (10 000, F16: 326) where the rows stream in 76; 8 / 8 heads of 64, FP8, 288 us against 38.
//
//   CTA   = (split, kv-head x block of eight q-heads, unit), eight warps, one tile of T positions at a time.
//   S^T   = K Q^T, M = 16 positions, N = 8 heads.  A K row goes from global memory straight into A fragments: the
//           contraction does not care about the order of the dims, so lane tig of a row takes 16 consecutive bytes
//           and Q is laid out in shared memory as the matching B fragments, in a high and a low half-precision term.
//   softmax: warp h does head h: scores from shared memory, running maximum and sum in its registers, P back as the
//           B fragments (high + low term) of the second product.
//   O^T   = V^T P^T, M = 16 dims, N = 8 heads, for 64 dims of the tile's positions a warp (all warps along the
//           dims of a 512-dim head, along the positions of a 64-dim one).  Lane tig takes positions 4 tig .. 4 tig + 3
//           of a block of 16, lane gid 8 consecutive dims of each; a byte permute pairs positions.
//   The next tile's K rows are loaded behind the first product, its V rows behind the second, so one of the two is
//   always in flight: 32 registers a lane each, two CTAs an SM (short rows: two tiles of each instead).
#include "attn_params.cuh"
#include "mma_sync.cuh"
#include "softcap.cuh"

namespace vfkv {

namespace {

constexpr int kWarps = 8;

template <int DT, int D> struct Wide {
    static constexpr int ES = DT == VFKV_F8 ? 1 : 2;
    static constexpr int ROW = D * ES;                       // bytes of a head's row
    static constexpr int T = ROW > 512 ? 32 : ROW > 256 ? 64 : 128;     // positions of a tile: 32 KB of rows or less
    static constexpr int NBUF = ROW > 256 ? 1 : 2;           // tiles of K and of V in registers or on their way there
    static constexpr int DP = kWarps / (T / 16);             // warps along the dims in the first product
    static constexpr int E = 16 / ES;                        // dims of a lane's 16 bytes
    static constexpr int NU = ROW / 64 / DP;                 // 64-byte units of a row a warp contracts over
    static constexpr int NDG = D / 64, PH = kWarps / NDG;    // warps along the dims / positions in the second product
    static constexpr int PB = T / 16 / PH;                   // blocks of 16 positions a warp takes there
    static constexpr int VW = 2 * ES;                        // words of 8 dims
    // shared memory, bytes
    static constexpr int Q_AT = 0, Q_BYTES = D / 16 * 32 * 16;
    static constexpr int S_AT = Q_AT + Q_BYTES, S_PITCH = T + 4, S_BYTES = DP * 8 * S_PITCH * 4;
    static constexpr int P_AT = S_AT + S_BYTES, P_BYTES = T / 16 * 32 * 16;
    static constexpr int C_AT = P_AT + P_BYTES, C_BYTES = 3 * 8 * 4;    // factor of the accumulators, maximum, sum
    static constexpr int O_PITCH = 64 + 4, O_BYTES = PH > 1 ? kWarps * 8 * O_PITCH * 4 : 0;
    static constexpr int SMEM = (C_AT + C_BYTES > O_BYTES ? C_AT + C_BYTES : O_BYTES) + (PH > 1 ? C_BYTES : 0);
};

// words -> the A fragment of 16 rows x 4 dims a lane
template <int DT> __device__ __forceinline__ void k_fragment(const uint4 &lo, const uint4 &hi, int j, uint32_t (&a)[4])
{
    const uint32_t l[4] = {lo.x, lo.y, lo.z, lo.w}, h[4] = {hi.x, hi.y, hi.z, hi.w};
    if constexpr (DT == VFKV_F8) {
        e4m3x4_to_half2x2(l[j], a[0], a[2]);
        e4m3x4_to_half2x2(h[j], a[1], a[3]);
    } else {
        a[0] = l[2 * j]; a[2] = l[2 * j + 1];
        a[1] = h[2 * j]; a[3] = h[2 * j + 1];
    }
}
// dims 2i, 2i + 1 of four positions -> the A fragment of V^T
template <int DT, int VW> __device__ __forceinline__ void v_fragment(const uint32_t (&v)[4][VW], int i, uint32_t (&a)[4])
{
    if constexpr (DT == VFKV_F8) {
        const uint32_t sel = (i & 1) ? 0x7362u : 0x5140u;       // {p0.d, p1.d, p0.d+1, p1.d+1}
        e4m3x4_to_half2x2(prmt(v[0][i / 2], v[1][i / 2], sel), a[0], a[1]);
        e4m3x4_to_half2x2(prmt(v[2][i / 2], v[3][i / 2], sel), a[2], a[3]);
    } else {
        a[0] = prmt(v[0][i], v[1][i], 0x5410u); a[1] = prmt(v[0][i], v[1][i], 0x7632u);
        a[2] = prmt(v[2][i], v[3][i], 0x5410u); a[3] = prmt(v[2][i], v[3][i], 0x7632u);
    }
}

template <int DT, int D>
__global__ void __launch_bounds__(kWarps * 32, 2)
attn_wide_kernel(const AttnParams p)
{
    using W = Wide<DT, D>;
    extern __shared__ __align__(16) uint8_t sm[];
    uint4 *const sq = reinterpret_cast<uint4 *>(sm + W::Q_AT);        // [16 dims][lane]
    float *const ss = reinterpret_cast<float *>(sm + W::S_AT);        // [dim part][head][position]
    uint4 *const sp = reinterpret_cast<uint4 *>(sm + W::P_AT);        // [16 positions][lane]
    float *const sc_corr = reinterpret_cast<float *>(sm + W::SMEM - W::C_BYTES), *const sc_m = sc_corr + 8, *const sc_l = sc_m + 8;

    const uint32_t head_blocks = (p.group + 7u) / 8u;
    const uint32_t split = blockIdx.x, kvh = blockIdx.y / head_blocks, hb = blockIdx.y % head_blocks;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gid = lane >> 2, tig = lane & 3;
    const UnitOf unit = unit_of(p, blockIdx.z);
    const uint32_t h0 = kvh * p.group + hb * 8u, nh = min(8u, p.group - hb * 8u);

    pdl_wait();
    uint32_t slot, start, len, begin, end;
    seq_range(p, unit, &slot, &start, &len);
    split_range(start, len, p.n_splits, split, 32, &begin, &end);
    const uint32_t n_tiles = (end - begin + W::T - 1) / W::T;

    const uint64_t row_bytes = uint64_t(p.n_kv_heads) * W::ROW;
    const uint64_t head_at = uint64_t(slot) * p.slot_stride_bytes + uint64_t(kvh) * W::ROW;
    const uint32_t pg = warp % (W::T / 16), dp = warp / (W::T / 16);
    const uint32_t dg = warp % W::NDG, ph = warp / W::NDG;
    const uint8_t *const kb = p.k + head_at + dp * (W::NU * 64) + tig * 16;
    const uint8_t *const vb = p.v + head_at + (dg * 64 + gid * 8) * W::ES;

    // rows past the range are read as its last one; their P is zero
    uint4 kr[W::NBUF][W::NU][2];
    auto load_k = [&](uint32_t t, uint4 (&kr)[W::NU][2]) {
        const uint32_t t0 = begin + t * W::T + pg * 16 + gid;
        const uint8_t *const r0 = kb + uint64_t(min(t0, end - 1)) * row_bytes, *const r1 = kb + uint64_t(min(t0 + 8, end - 1)) * row_bytes;
#pragma unroll
        for (int u = 0; u < W::NU; ++u) {
            kr[u][0] = *reinterpret_cast<const uint4 *>(r0 + u * 64);
            kr[u][1] = *reinterpret_cast<const uint4 *>(r1 + u * 64);
        }
    };
    uint32_t vr[W::NBUF][W::PB][4][W::VW];
    auto load_v = [&](uint32_t t, uint32_t (&vr)[W::PB][4][W::VW]) {
#pragma unroll
        for (int b = 0; b < W::PB; ++b)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t pos = min(begin + t * W::T + (ph * W::PB + b) * 16 + 4 * tig + i, end - 1);
                const uint8_t *const r = vb + uint64_t(pos) * row_bytes;
                if constexpr (W::VW == 2) {
                    const uint2 x = *reinterpret_cast<const uint2 *>(r);
                    vr[b][i][0] = x.x; vr[b][i][1] = x.y;
                } else {
                    const uint4 x = *reinterpret_cast<const uint4 *>(r);
                    vr[b][i][0] = x.x; vr[b][i][1] = x.y; vr[b][i][2] = x.z; vr[b][i][3] = x.w;
                }
            }
    };
    const float *const ksc = p.k_scales ? p.k_scales + uint64_t(slot) * p.slot_stride_scales + kvh : nullptr;
    const float *const vsc = p.v_scales ? p.v_scales + uint64_t(slot) * p.slot_stride_scales + kvh : nullptr;
    float ks_next[4], vs_next[4];            // scales of the next tile's positions 4 lane .. 4 lane + 3
    auto load_scales = [&](uint32_t t) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t pos = begin + t * W::T + 4 * lane + i;
            const bool ok = lane < uint32_t(W::T / 4) && pos < end;
            ks_next[i] = ok ? ksc[uint64_t(pos) * p.n_kv_heads] : 1.f;
            vs_next[i] = ok ? vsc[uint64_t(pos) * p.n_kv_heads] : 0.f;
        }
    };
#pragma unroll
    for (int i = 0; i < W::NBUF; ++i)
        if (uint32_t(i) < n_tiles) { load_k(i, kr[i]); load_v(i, vr[i]); }
    const bool scaled = DT == VFKV_F8 && ksc != nullptr;
    if (scaled && n_tiles) load_scales(0);

    // Q: head `warp`, scaled by a power of two (largest element in [128, 256)), as B fragments
    float mult;
    {
        const bool hv = warp < nh;
        const float *const q = p.q + (uint64_t(unit.row) * p.n_q_heads + h0 + (hv ? warp : 0)) * D;
        constexpr int NQ = (D + 127) / 128;
        float4 x[NQ];
        float amax = 0.f;
#pragma unroll
        for (int i = 0; i < NQ; ++i) {
            const uint32_t d = 4 * (lane + 32 * i);
            x[i] = hv && d < uint32_t(D) ? *reinterpret_cast<const float4 *>(q + d) : make_float4(0.f, 0.f, 0.f, 0.f);
            amax = fmaxf(amax, fmaxf(fmaxf(fabsf(x[i].x), fabsf(x[i].y)), fmaxf(fabsf(x[i].z), fabsf(x[i].w))));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        int e = int((__float_as_uint(amax) >> 23) & 0xFF) - 127;
        e = amax > 0.f ? max(-100, min(100, e)) : 7;
        const float qs = __uint_as_float(uint32_t(7 - e + 127) << 23);
        mult = p.scale * __uint_as_float(uint32_t(e - 7 + 127) << 23) * (p.softcap > 0.f ? 1.0f : kLog2e);
#pragma unroll
        for (int i = 0; i < NQ; ++i) {
            const uint32_t d = 4 * (lane + 32 * i);
            if (d < uint32_t(D)) {
                const uint32_t un = d / (4 * W::E), r = d % (4 * W::E);
                uint4 f;
                split_f16x2(x[i].x * qs, x[i].y * qs, f.x, f.z);
                split_f16x2(x[i].z * qs, x[i].w * qs, f.y, f.w);
                sq[(un * (W::E / 4) + r % W::E / 4) * 32 + warp * 4 + r / W::E] = f;
            }
        }
    }
    __syncthreads();

    const float inv_cap = p.softcap > 0.f ? 1.0f / p.softcap : 0.f;
    float m = kMaskedScore, l = 0.f;         // head `warp`
    uint32_t vs_ref = 0u;                    // exponent that the V scales of the accumulators are relative to
    float acc[4][4];                         // summed in f32 tile by tile, see below
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;

    auto tile = [&](uint32_t t, uint4 (&kr)[W::NU][2], uint32_t (&vr)[W::PB][4][W::VW]) {
        const uint32_t t0 = begin + t * W::T;
        // ---- S^T = K Q^T for 16 positions; four chains of products ----
        {
            float s[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f;
            const uint4 *const qf = sq + dp * (W::NU * (W::E / 4) * 32) + lane;
#pragma unroll
            for (int u = 0; u < W::NU; ++u)
#pragma unroll
                for (int j = 0; j < W::E / 4; ++j) {
                    uint32_t a[4];
                    k_fragment<DT>(kr[u][0], kr[u][1], j, a);
                    const uint4 b = qf[(u * (W::E / 4) + j) * 32];
                    mma_f16(s[2 * (j & 1)], a, b.x, b.y);
                    mma_f16(s[2 * (j & 1) + 1], a, b.z, b.w);
                }
            float *const out = ss + (dp * 8 + 2 * tig) * W::S_PITCH + pg * 16 + gid;
#pragma unroll
            for (int i = 0; i < 4; ++i) out[(i & 1) * W::S_PITCH + (i >> 1) * 8] = (s[0][i] + s[2][i]) + (s[1][i] + s[3][i]);
        }
        if (t + W::NBUF < n_tiles) load_k(t + W::NBUF, kr);
        __syncthreads();

        // ---- softmax of head `warp`; lane: positions 4 lane .. 4 lane + 3 ----
        {
            const bool mine = lane < uint32_t(W::T / 4);
            const uint32_t pos = t0 + 4 * lane;
            float x[4];
            if (mine) {
                const float4 a = *reinterpret_cast<const float4 *>(ss + warp * W::S_PITCH + 4 * lane);
                x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
#pragma unroll
                for (int i = 1; i < W::DP; ++i) {
                    const float4 b = *reinterpret_cast<const float4 *>(ss + (8 * i + warp) * W::S_PITCH + 4 * lane);
                    x[0] += b.x; x[1] += b.y; x[2] += b.z; x[3] += b.w;
                }
            } else {
                x[0] = x[1] = x[2] = x[3] = 0.f;
            }
            float vs[4] = {kPScale, kPScale, kPScale, kPScale}, vs_corr = 1.f;
            if (scaled) {
                float top = 0.f;
#pragma unroll
                for (int i = 0; i < 4; ++i) { x[i] *= ks_next[i]; vs[i] = vs_next[i]; top = fmaxf(top, vs[i]); }
                if (t + 1 < n_tiles) load_scales(t + 1);
                // powers of two relative to the largest scale so far; scales are at least 1e-12 and at most 2^119
                const uint32_t top_e = __reduce_max_sync(0xffffffffu, __float_as_uint(top)) & 0x7f800000u;
                if (top_e > vs_ref) {
                    vs_corr = vs_ref != 0u && top_e - vs_ref < (127u << 23) ? __uint_as_float((127u << 23) - (top_e - vs_ref)) : 0.f;
                    vs_ref = top_e;
                }
                const float f = __uint_as_float((254u << 23) - vs_ref) * kPScale;
#pragma unroll
                for (int i = 0; i < 4; ++i) vs[i] *= f;
            }
            float mn = m;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                x[i] *= mult;
                if (p.softcap > 0.f) x[i] = softcap_any(x[i], p.softcap, inv_cap) * kLog2e;
                x[i] = mine && pos + i < end ? x[i] : kMaskedScore;
                mn = fmaxf(mn, x[i]);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
            const float corr = fast_exp2(m - mn);
            m = mn;
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float e = fast_exp2(x[i] - mn);
                sum += e;
                x[i] = e * vs[i];
            }
            l = fmaf(l, corr, sum);          // this lane's share of the sum
            if (mine) {
                uint4 f;
                split_f16x2(x[0], x[1], f.x, f.z);
                split_f16x2(x[2], x[3], f.y, f.w);
                sp[(lane >> 2) * 32 + warp * 4 + (lane & 3)] = f;
            }
            if (lane == 0) sc_corr[warp] = corr * vs_corr;
        }
        __syncthreads();

        // ---- O^T += V^T P^T ----
        {
            // The tensor cores cut off towards zero what an accumulator does not hold, so a tile's products start
            // from zero and are added to the others in f32 (F16, 20 000 positions x 4 layers: results 3.1e-6 off in one
            // chain, 3.1e-7 so; 95.6 -> 100.2 us).
            const float2 c = *reinterpret_cast<const float2 *>(sc_corr + 2 * tig);
            float o[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
#pragma unroll
            for (int b = 0; b < W::PB; ++b) {
                const uint4 f = sp[(ph * W::PB + b) * 32 + lane];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    uint32_t a[4];
                    v_fragment<DT, W::VW>(vr[b], i, a);
                    mma_f16(o[i], a, f.x, f.y);
                    mma_f16(o[i], a, f.z, f.w);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                acc[i][0] = fmaf(acc[i][0], c.x, o[i][0]); acc[i][1] = fmaf(acc[i][1], c.y, o[i][1]);
                acc[i][2] = fmaf(acc[i][2], c.x, o[i][2]); acc[i][3] = fmaf(acc[i][3], c.y, o[i][3]);
            }
        }
        if (t + W::NBUF < n_tiles) load_v(t + W::NBUF, vr);
    };
    for (uint32_t t = 0; t < n_tiles; t += W::NBUF) {
#pragma unroll
        for (int i = 0; i < W::NBUF; ++i)
            if (t + i < n_tiles) tile(t + i, kr[i], vr[i]);
    }

    // ---- epilogue: maxima and sums by head, then this warp's 64 dims (after a sum over the warps of a 64-dim head) ----
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    __syncthreads();
    if (lane == 0) { sc_m[warp] = m; sc_l[warp] = l; sc_corr[warp] = kInvPScale * (vs_ref ? __uint_as_float(vs_ref) : 1.f); }
    if constexpr (W::PH > 1) {
        float *const so = reinterpret_cast<float *>(sm) + warp * (8 * W::O_PITCH);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) so[(2 * tig + (j & 1)) * W::O_PITCH + gid * 8 + 2 * i + (j >> 1)] = acc[i][j];
    }
    __syncthreads();
    auto store = [&](uint32_t h, uint32_t d, float4 o) {
        const float M = sc_m[h], L = sc_l[h], f = sc_corr[h];
        o = make_float4(o.x * f, o.y * f, o.z * f, o.w * f);
        const uint64_t row = uint64_t(unit.row) * p.n_q_heads + h0 + h;
        // a range without positions: maximum kMaskedScore, sum 0
        const float mm = n_tiles ? M * kLn2 : kMaskedScore;
        if (p.n_splits == 1) {
            const float inv = L > 0.f ? 1.0f / L : 0.f;
            if (p.out) *reinterpret_cast<float4 *>(p.out + row * D + d) = make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv);
            if (p.out_o) {
                *reinterpret_cast<float4 *>(p.out_o + row * D + d) = o;
                if (d == 0) { p.out_m[row] = mm; p.out_l[row] = L; }
            }
        } else {
            const uint64_t pi = (uint64_t(blockIdx.z) * p.n_q_heads + h0 + h) * p.n_splits + split;
            *reinterpret_cast<float4 *>(p.part_o + pi * D + d) = o;
            if (d == 0) { p.part_m[pi] = mm; p.part_l[pi] = L; }
        }
    };
    if constexpr (W::PH > 1) {
        for (uint32_t i = threadIdx.x; i < nh * (D / 4); i += kWarps * 32) {
            const uint32_t h = i / (D / 4), d = 4 * (i % (D / 4));
            float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int w = 0; w < kWarps; ++w) {
                const float4 a = *reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(sm) + (w * 8 + h) * W::O_PITCH + d);
                o.x += a.x; o.y += a.y; o.z += a.z; o.w += a.w;
            }
            store(h, d, o);
        }
    } else {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const uint32_t h = 2 * tig + j, d = dg * 64 + gid * 8;
            if (h < nh) {
                store(h, d, make_float4(acc[0][j], acc[0][2 + j], acc[1][j], acc[1][2 + j]));
                store(h, d + 4, make_float4(acc[2][j], acc[2][2 + j], acc[3][j], acc[3][2 + j]));
            }
        }
    }
}

template <int DT, int D> int32_t launch_wide_t(vfkv_ctx *ctx, const AttnParams &p, cudaStream_t st)
{
    static_assert(Wide<DT, D>::SMEM <= 48 * 1024, "no attribute needed");
    const dim3 grid(p.n_splits, p.n_kv_heads * ((p.group + 7) / 8), p.n_seqs * p.n_layers);
    {
        ProfScope ps(ctx, VFKV_PROF_FA_SPLIT, st);
        if (cudaError_t e = launch_dependent(ctx, attn_wide_kernel<DT, D>, grid, dim3(kWarps * 32), Wide<DT, D>::SMEM, st, p))
            return check_cuda(ctx, e, "wide attention launch");
    }
    ctx->count_launch(p.n_layers);
    return check_cuda(ctx, cudaGetLastError(), "wide attention launch");
}

}  // namespace

bool attn_wide_supported(const AttnArgs &a)
{
    const uint32_t D = a.kv.head_dim;
    const uintptr_t at = reinterpret_cast<uintptr_t>(a.kv.k) | reinterpret_cast<uintptr_t>(a.kv.v) | reinterpret_cast<uintptr_t>(a.q) |
                         reinterpret_cast<uintptr_t>(a.out) | reinterpret_cast<uintptr_t>(a.out_o);
    if (at % 16 != 0 || a.kv.slot_stride_bytes % 16 != 0) return false;
    if ((a.kv.k_scales != nullptr) != (a.kv.v_scales != nullptr)) return false;
    return (a.kv.dtype == VFKV_F8 && (D == 64 || D == 512)) || (a.kv.dtype == VFKV_F16 && D == 512 && !a.kv.k_scales);
}

int32_t launch_attn_wide(vfkv_ctx *ctx, vfkv_workspace *ws, const AttnArgs &a, uint32_t n_splits, cudaStream_t st)
{
    const AttnParams p = make_params(ctx, ws, a, n_splits);
    if (a.kv.dtype == VFKV_F16) return launch_wide_t<VFKV_F16, 512>(ctx, p, st);
    return a.kv.head_dim == 64 ? launch_wide_t<VFKV_F8, 64>(ctx, p, st) : launch_wide_t<VFKV_F8, 512>(ctx, p, st);
}

}  // namespace vfkv
