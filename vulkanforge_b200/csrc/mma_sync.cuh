// What the mma.sync decode kernels share: the f16 product, the split of a value into two half-precision terms,
// and the constants of the log2-domain softmax.
#pragma once

#include "fp8_codec.cuh"

namespace vfkv {

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;
// P goes into the tensor cores as half-precision terms.  With tens of thousands of positions most
// p = 2^(x - m) lie below the smallest normal half (6.1e-5), where the terms keep few or no bits
// (measured: 6.5e-5 absolute error at 40 000 positions).  So P is fed as p * 2^14 (still at most
// 16 384) and the accumulators are scaled back when the warp's partial is written; both scalings
// are exact, and l is summed from the unscaled p.
constexpr float kPScale = 16384.0f, kInvPScale = 1.0f / 16384.0f;

__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel)
{
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}
__device__ __forceinline__ float fast_exp2(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// Two values -> (hi, lo) half2 pairs with hi + lo == value to about 2^-22.
__device__ __forceinline__ void split_f16x2(float x0, float x1, uint32_t &hi, uint32_t &lo)
{
    __half2 h = __floats2half2_rn(x0, x1);
    float2 hf = __half22float2(h);
    hi = *reinterpret_cast<uint32_t *>(&h);
    lo = f32x2_to_f16x2(x0 - hf.x, x1 - hf.y);
}

// Four E4M3 codes -> two half2: bytes 0,1 and bytes 2,3 (exact).
__device__ __forceinline__ void e4m3x4_to_half2x2(uint32_t w, uint32_t &lo, uint32_t &hi)
{
    asm("{\n\t.reg .b16 a, b;\n\t"
        "mov.b32 {a, b}, %2;\n\t"
        "cvt.rn.f16x2.e4m3x2 %0, a;\n\t"
        "cvt.rn.f16x2.e4m3x2 %1, b;\n\t}"
        : "=r"(lo), "=r"(hi)
        : "r"(w));
}

}  // namespace vfkv
