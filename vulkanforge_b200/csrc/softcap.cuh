// Score soft-cap: cap * tanh(s / cap), the formula the reference applies to final logits
// (src/backend/vulkan/forward/arch/gemma4.rs:85-94).
//
// tanhf costs some 25 instructions and a branch for every score, which made the softmax of a capped
// prefill tile several times as long as the rest of the tile (282 queries with a window of 1024 on the
// tcgen05 kernel: 50 us without a cap, 294 with it).  Scores lie well inside the cap, where an odd
// polynomial is all that is needed: with y = s / cap, cap * tanh(y) = s * P(y^2), P the degree-6
// Chebyshev interpolant of tanh(sqrt(u)) / sqrt(u) on [0, 0.64] (largest relative error 1e-7 in f32;
// tanhf allows itself 2 ulp).  Beyond |y| = 0.8, tanh(y) = 1 - 2 / (1 + e^(2y)): nothing cancels there.
#pragma once

#include <cuda_runtime.h>

namespace vfkv {

constexpr float kSoftcapSmall = 0.8f;      // |s / cap| up to which the polynomial holds

__device__ __forceinline__ float softcap_small(float s, float inv_cap)
{
    const float y = s * inv_cap, u = y * y;
    float r = 0.0015708811f;
    r = fmaf(r, u, -0.0073803058f);
    r = fmaf(r, u, 0.021279233f);
    r = fmaf(r, u, -0.053843055f);
    r = fmaf(r, u, 0.13332045f);
    r = fmaf(r, u, -0.33333284f);
    return fmaf(s * u, r, s);
}
__device__ __forceinline__ float softcap_any(float s, float cap, float inv_cap)
{
    const float y = s * inv_cap;
    float e, r;
    asm("ex2.approx.f32 %0, %1;" : "=f"(e) : "f"(y * 2.8853900818f));      // e^(2y)
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(e + 1.0f));
    const float big = fmaf(-2.0f * cap, r, cap);
    return fabsf(y) > kSoftcapSmall ? big : softcap_small(s, inv_cap);
}
// N scores of a thread; all 32 lanes of the warp take part.
template <int N> __device__ __forceinline__ void softcap_all(float (&s)[N], float cap, float inv_cap)
{
    float top = 0.f;
#pragma unroll
    for (int i = 0; i < N; ++i) top = fmaxf(top, fabsf(s[i]));
    if (__any_sync(0xffffffffu, top * inv_cap > kSoftcapSmall)) {
#pragma unroll
        for (int i = 0; i < N; ++i) s[i] = softcap_any(s[i], cap, inv_cap);
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) s[i] = softcap_small(s[i], inv_cap);
    }
}

}  // namespace vfkv
