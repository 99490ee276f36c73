// GELU and its derivative, rounded to BF16, for the surrogate's layers.
//
// The reference evaluations gelu() and gelu_grad() use CUDA's erff (about 25
// instructions a value, which bound the inference kernel: tensor pipe 12 %,
// issue 59 %).  What the layers keep is the value rounded to BF16, so a
// cheaper approximation whose error interval rounds to one BF16 number gives
// the same bits; where the two ends differ (about four values in 10,000 of
// normally distributed ones) the reference decides.  The approximation is
//   Phi(x) = 1 / (1 + 2^-G(x)),  G(x) = log2(Phi(x) / Phi(-x)) = x W(x^2),
// W a degree-6 polynomial (a minimax fit weighted by Phi's sensitivity, by
// Lawson's iteration: Phi within 3e-8; its leading coefficient is positive, so
// the ends need no clamp), evaluated two values at a time with packed FP32
// multiply-adds.  (Phi from erfc(|x|) = 2^-P(|x|) with the sign put back took a
// degree-8 polynomial and four bit operations a value more: 3.60 ms for a
// million rows x 4 members.)
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

// 1 / x of a positive float, within one ulp
__device__ __forceinline__ float rcp(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Phi(x) of two values
__device__ __forceinline__ F2 phi(F2 x)
{
    const F2 y = mul2(x, x);
    F2 p = fma2(y, f2(-5.06723685e-09f, -5.06723685e-09f), f2(3.8163131e-07f, 3.8163131e-07f));
    p = fma2(y, p, f2(-1.14398335e-05f, -1.14398335e-05f));
    p = fma2(y, p, f2(0.00015957994f, 0.00015957994f));
    p = fma2(y, p, f2(9.40492246e-05f, 9.40492246e-05f));
    p = fma2(y, p, f2(-0.104835123f, -0.104835123f));
    p = fma2(y, p, f2(-2.30220938f, -2.30220938f));
    float p0, p1;
    split(mul2(x, p), p0, p1);
    split(add2(f2(ex2(p0), ex2(p1)), f2(1.0f, 1.0f)), p0, p1);
    return f2(rcp(p0), rcp(p1));
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

// BF16 of gelu at two values (the first in the lower half) from the two ends
// of the interval; they differ in a half whose rounding is left open
__device__ __forceinline__ uint32_t value_bf16x2(F2 x, uint32_t &other)
{
    F2 lo, hi;
    widen(phi(x), lo, hi);
    float l0, l1, h0, h1;
    split(mul2(x, lo), l0, l1);
    split(mul2(x, hi), h0, h1);
    other = bf16x2(h0, h1);
    return bf16x2(l0, l1);
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

// BF16 of gelu at the 2 * n values v + bias, bit for bit the reference's
template <int n>
__device__ __forceinline__ void values_bf16(float *v, const float *bias, uint32_t *r)
{
    uint32_t other[n], any = 0u;   // the roundings of the intervals' other ends
#pragma unroll
    for (int j = 0; j < n; j++) {
        const F2 x = bias ? add2(f2(v[2 * j], v[2 * j + 1]), f2(bias[2 * j], bias[2 * j + 1]))
                          : f2(v[2 * j], v[2 * j + 1]);
        split(x, v[2 * j], v[2 * j + 1]);
        r[j] = value_bf16x2(x, other[j]);
        any |= r[j] ^ other[j];
    }
    if (any) {
#pragma unroll
        for (int j = 0; j < n; j++)
            if (r[j] != other[j])
                r[j] = value_decide(v[2 * j], v[2 * j + 1], r[j], r[j] ^ other[j]);
    }
}

// ---- the derivative, Phi(x) + x phi(x)

// two values below and above grad(x) (checked for every float)
constexpr float kGradMargin = 4e-7f;

__device__ __forceinline__ void grad_bounds(F2 x, F2 &lo, F2 &hi)
{
    // the density as a power of two: 2^(-x^2 / (2 ln 2) + log2(1 / sqrt(2 pi)))
    float d0, d1;
    split(fma2(mul2(x, x), f2(-0.72134752f, -0.72134752f), f2(-1.32574806f, -1.32574806f)), d0, d1);
    const F2 g = fma2(x, f2(ex2(d0), ex2(d1)), phi(x));
    lo = add2(g, f2(-kGradMargin, -kGradMargin));
    hi = add2(g, f2(kGradMargin, kGradMargin));
}

__device__ __noinline__ uint32_t grad_decide(float v0, float v1, float x0, float x1, uint32_t r, uint32_t open)
{
    if (open & 0xffffu)
        r = (r & 0xffff0000u) | (bf16x2(v0 * grad(x0), 0.0f) & 0xffffu);
    if (open >> 16)
        r = (r & 0xffffu) | bf16x2(0.0f, v1 * grad(x1));
    return r;
}

// BF16 of v * grad(x) at 2 * n values, bit for bit the reference's: the
// products with both bounds lie on both sides of the reference's product
template <int n>
__device__ __forceinline__ void grads_bf16(const float *v, const float *x, uint32_t *r)
{
    uint32_t other[n], any = 0u;
#pragma unroll
    for (int j = 0; j < n; j++) {
        const F2 w = f2(v[2 * j], v[2 * j + 1]);
        F2 lo, hi;
        grad_bounds(f2(x[2 * j], x[2 * j + 1]), lo, hi);
        float l0, l1, h0, h1;
        split(mul2(w, lo), l0, l1);
        split(mul2(w, hi), h0, h1);
        r[j] = bf16x2(l0, l1);
        other[j] = bf16x2(h0, h1);
        any |= r[j] ^ other[j];
    }
    if (any) {
#pragma unroll
        for (int j = 0; j < n; j++)
            if (r[j] != other[j])
                r[j] = grad_decide(v[2 * j], v[2 * j + 1], x[2 * j], x[2 * j + 1], r[j], r[j] ^ other[j]);
    }
}

}  // namespace gelu
}  // namespace anacor
