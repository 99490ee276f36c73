// GELU and its derivative, rounded to BF16, for the surrogate's layers.
//
// The reference evaluations gelu() and gelu_grad() use CUDA's erff (about 25
// instructions a value, which bound the inference kernel: tensor pipe 12 %,
// issue 59 %).  What the layers keep is the value rounded to BF16, so a
// cheaper approximation whose error interval rounds to one BF16 number gives
// the same bits; where the two ends differ (about one value in a thousand of
// normally distributed ones) the reference decides.  The approximation is
//   Phi(x) = 1/2 + s (1/2 - Q),  s = sign of x,  Q = erfc(|x| / sqrt 2) / 2,
//   Q = 2^-P(|x|),  P a degree-8 polynomial with P(0) = 1 (a weighted minimax
// fit of -log2 Q by Lawson's iteration, error of Q below 1e-8), evaluated two
// values at a time with packed FP32 multiply-adds.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace anacor {
namespace gelu {

// the reference evaluations
__device__ __forceinline__ float value(float x)
{
    return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f));
}

__device__ __forceinline__ float grad(float x)
{
    const float cdf = 0.5f * (1.0f + erff(x * 0.70710678118654752f));
    const float pdf = 0.3989422804014327f * expf(-0.5f * x * x);
    return cdf + x * pdf;
}

// ---- two floats in a 64-bit register
using F2 = unsigned long long;

__device__ __forceinline__ F2 f2(float a, float b)
{
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}

__device__ __forceinline__ void split(F2 v, float &a, float &b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}

__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c)
{
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

__device__ __forceinline__ F2 add2(F2 a, F2 b)
{
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__device__ __forceinline__ F2 mul2(F2 a, F2 b)
{
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__device__ __forceinline__ float ex2(float x)
{
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// (lower half from a, upper half from b)
__device__ __forceinline__ uint32_t bf16x2(float a, float b)
{
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
    return r;
}

// Phi(x) of two values
__device__ __forceinline__ F2 phi(F2 x)
{
    const F2 a = x & 0x7fffffff7fffffffull;
    F2 p = fma2(a, f2(-2.83490704e-06f, -2.83490704e-06f), f2(3.93776281e-05f, 3.93776281e-05f));
    p = fma2(a, p, f2(-0.000186179954f, -0.000186179954f));
    p = fma2(a, p, f2(-0.000136937015f, -0.000136937015f));
    p = fma2(a, p, f2(0.00706342096f, 0.00706342096f));
    p = fma2(a, p, f2(-0.0524961799f, -0.0524961799f));
    p = fma2(a, p, f2(-0.45920819f, -0.45920819f));
    p = fma2(a, p, f2(-1.15110517f, -1.15110517f));
    p = fma2(a, p, f2(-1.0f, -1.0f));
    float p0, p1;
    split(p, p0, p1);
    const F2 h = add2(f2(0.5f, 0.5f), f2(-ex2(p0), -ex2(p1)));
    const F2 s = (x & 0x8000000080000000ull) | 0x3f8000003f800000ull;
    return fma2(s, h, f2(0.5f, 0.5f));
}

// An interval around phi(x) that holds the reference's (1 + erff) / 2 and
// makes up for the rounding of the products after it: erff near 1 is a
// multiple of 2^-24 off by up to two of them, so the absolute part matters on
// the negative side, the relative one on the positive side.  (Checked over
// all 2^32 floats: no value rounds differently.)
__device__ __forceinline__ void widen(F2 u, F2 &lo, F2 &hi)
{
    constexpr float kAbs = 7.5e-8f, kLess = 1.0f - 0x1.8p-23f, kMore = 1.0f + 0x1p-22f;
    lo = fma2(u, f2(kLess, kLess), f2(-kAbs, -kAbs));
    hi = fma2(u, f2(kMore, kMore), f2(kAbs, kAbs));
}

// BF16 of gelu at two values (a in the lower half); `open` is nonzero in the
// half whose rounding the approximation leaves open.
__device__ __forceinline__ uint32_t value_bf16x2(float a, float b, uint32_t &open)
{
    const F2 x = f2(a, b);
    F2 lo, hi;
    widen(phi(x), lo, hi);
    float l0, l1, h0, h1;
    split(mul2(x, lo), l0, l1);
    split(mul2(x, hi), h0, h1);
    const uint32_t r = bf16x2(l0, l1);
    open = r ^ bf16x2(h0, h1);
    return r;
}

// the halves left open, from the reference evaluation
__device__ __noinline__ uint32_t value_decide(float a, float b, uint32_t r, uint32_t open)
{
    if (open & 0xffffu)
        r = (r & 0xffff0000u) | (bf16x2(value(a), 0.0f) & 0xffffu);
    if (open >> 16)
        r = (r & 0xffffu) | bf16x2(0.0f, value(b));
    return r;
}

// BF16 of gelu at 2 * n values, bit for bit the reference's
template <int n>
__device__ __forceinline__ void values_bf16(const float *v, uint32_t *r)
{
    uint32_t open[n], any = 0u;
#pragma unroll
    for (int j = 0; j < n; j++) {
        r[j] = value_bf16x2(v[2 * j], v[2 * j + 1], open[j]);
        any |= open[j];
    }
    if (any) {
#pragma unroll
        for (int j = 0; j < n; j++)
            if (open[j])
                r[j] = value_decide(v[2 * j], v[2 * j + 1], r[j], open[j]);
    }
}

}  // namespace gelu
}  // namespace anacor
