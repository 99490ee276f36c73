// Small device helpers shared by the absorption, gridding and interpolation
// kernels.
#pragma once
#include <cuda_runtime.h>
#include <math.h>

namespace anacor {

// x within [-b, b], undefined where x is
__device__ __forceinline__ float clamp_nan(float x, float b)
{
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(x), "f"(b));
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(r), "f"(-b));
    return r;
}

// exp(-x) = 2^-k exp(-r) with the additive range reduction of exp by
// multiples of ln 2 (Cody and Waite, "Software Manual for the Elementary
// Functions", 1980, the exp chapter): k = rint(x / ln2), r = x - k ln2 in FP64
// (one FP64 constant instead of their two-part split: the rounding of k ln2,
// ~1e-16 k, is far below FP32's resolution), then CUDA's expf on the FP32 r,
// |r| <= ln2/2, and an exact scaling by 2^-k.
// Where k ln2 no longer holds x's last bits (from about 1e17 on) r lies far
// outside that range; clamped, its expf stays near one, and the scaling gives
// the 0 or infinity that exp is there.  (A branch for such exponents instead
// left the four voxels of a load one after another: 9,727 bilinear lookups of
// 960 voxels, a block each, 115 us, 100 so.)
__device__ __forceinline__ float exp_neg(double x)
{
    const double kd = rint(__dmul_rn(x, 1.4426950408889634));
    const double r = __fma_rn(-kd, 0.6931471805599453, x);
    const float e = expf(-clamp_nan((float)r, 0.5f));
    const int k = (int)fmaxf(fminf((float)kd, 400.0f), -400.0f);
    return ldexpf(e, -k);
}

// Knuth's TwoSum: s + e == a + b exactly
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e)
{
    s = a + b;
    const float bp = s - a;
    e = (a - (s - bp)) + (b - bp);
}

// A sum of floats as three: each holds what the ones before it round away
// (72 bits), so it is exact while the terms lie within about 2^40 of each other
// and the order of the terms does not matter.
struct FloatSum {
    float s, c, d;
};

__device__ __forceinline__ void sum_add(FloatSum &a, float x)
{
    float s, c, e, f;
    two_sum(a.s, x, s, e);
    two_sum(a.c, e, c, f);
    a.s = s;
    a.c = c;
    a.d += f;
}

__device__ __forceinline__ void sum_merge(FloatSum &a, float s, float c, float d)
{
    sum_add(a, s);
    float h, f;
    two_sum(a.c, c, h, f);
    a.c = h;
    a.d += d + f;
}

// the same in FP64, s + e exactly a + b
__device__ __forceinline__ void two_sum(double a, double b, double &s, double &e)
{
    s = __dadd_rn(a, b);
    const double bp = __dadd_rn(s, -a);
    e = __dadd_rn(__dadd_rn(a, -__dadd_rn(s, -bp)), __dadd_rn(b, -bp));
}

// ---- pairs of floats (h + l, |l| <= ulp(h) / 2) ----------------------------
//
// About 46 significant bits from FP32 instructions (Dekker, "A floating-point
// technique for extending the available precision", Numer. Math. 18, 1971),
// where GB300's FP64 pipe would bind a kernel: an FP64 instruction takes a
// warp 16 cycles there, an FP32 one a quarter of a cycle.

struct FloatPair {
    float h, l;
};

__device__ __forceinline__ FloatPair pair_of(double x)
{
    const float h = (float)x;
    return {h, (float)(x - (double)h)};
}

// h + l with |l| <= |h| renormalised (Fast2Sum)
__device__ __forceinline__ FloatPair pair_norm(float h, float l)
{
    const float s = __fadd_rn(h, l);
    return {s, __fadd_rn(l, -__fadd_rn(s, -h))};
}

__device__ __forceinline__ FloatPair pair_add(FloatPair a, FloatPair b)
{
    const float s = __fadd_rn(a.h, b.h);
    const float t = __fadd_rn(s, -a.h);
    const float e = __fadd_rn(__fadd_rn(a.h, -__fadd_rn(s, -t)), __fadd_rn(b.h, -t));
    return pair_norm(s, __fadd_rn(e, __fadd_rn(a.l, b.l)));
}

__device__ __forceinline__ FloatPair pair_neg(FloatPair a) { return {-a.h, -a.l}; }

// a * b for a float b
__device__ __forceinline__ FloatPair pair_mul(FloatPair a, float b)
{
    const float p = __fmul_rn(a.h, b);
    return pair_norm(p, __fmaf_rn(a.l, b, __fmaf_rn(a.h, b, -p)));
}

__device__ __forceinline__ FloatPair pair_mul(FloatPair a, FloatPair b)
{
    const float p = __fmul_rn(a.h, b.h);
    return pair_norm(p, __fmaf_rn(a.h, b.l, __fmaf_rn(a.l, b.h, __fmaf_rn(a.h, b.h, -p))));
}

// x * x, exact: a whole number of more than 12 bits has a square that a float
// does not hold
__device__ __forceinline__ FloatPair pair_square(float x)
{
    const float h = __fmul_rn(x, x);
    return {h, __fmaf_rn(x, x, -h)};
}

// square root: one Newton step on the FP32 root
__device__ __forceinline__ FloatPair pair_sqrt(FloatPair a)
{
    if (!(a.h > 0.0f))
        return {0.0f, 0.0f};
    const float s = __fsqrt_rn(a.h);
    const float r = __fadd_rn(__fmaf_rn(-s, s, a.h), a.l);   // a - s^2 (exact but for a.l's place)
    return pair_norm(s, __fdividef(r, __fadd_rn(s, s)));
}

// exp(-x) as exp_neg, from a pair: the same k and the same FP32 r but where
// r's rounding is a near tie.  ln 2 as the sum of three floats, each the
// rounding of what the ones before leave, the first cut to 12 bits so that
// its product with k is exact.
__device__ __forceinline__ float exp_neg(FloatPair x)
{
    const float k = clamp_nan(rintf(__fmul_rn(x.h, 1.44269504f)), 6000.0f);   // 2^-6000 is far below a float
    const float c1 = 2839.0f / 4096.0f;
    const float c2 = 0x1.0bfbe80000000p-15f;
    const float c3 = 0x1.cf79ac0000000p-40f;
    const float t = __fmaf_rn(-k, c1, x.h);   // exact
    const float p = __fmul_rn(-k, c2);
    const float pe = __fmaf_rn(-k, c2, -p);
    const FloatPair r = pair_add({t, 0.0f}, pair_add({p, pe}, {x.l, -k * c3}));
    const float e = expf(-clamp_nan(__fadd_rn(r.h, r.l), 0.5f));
    return ldexpf(e, -(int)k);
}

}  // namespace anacor
