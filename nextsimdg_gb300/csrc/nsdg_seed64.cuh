// nsdg_seed64.cuh — FP64 reciprocals and square roots from FP32 arithmetic.
//
// GB300 issues FP64 at about 1/60 of its FP32 rate, and CUDA's double
// division, sqrt and rsqrt take 10 to 20 FP64 instructions in one dependent
// chain.  Here the argument's significand is taken as a pair of floats, the
// FP32 approximation of 1/m or 1/sqrt(m) gets one step of the series in its
// residual, formed with error-free FP32 products (the FMA-based TwoProduct),
// and seed and correction are added on the integer pipe: 46 correct bits.  One
// Newton step in FP64 then gives the result, within 0.51 ulp for a square root
// and 0.51 for a reciprocal:
//   1/d      = r + r e,    e = 1 - d r                  (2 FP64 instructions)
//   sqrt t   = h + (t - h^2) y / 2,    h = t y          (3)
//   p/sqrt t = z + z e,    z = p y, e = 1/2 - h (y/2)   (4)
// Against the cubic series from the FP32 seed alone (3, 5 and 6 instructions):
// update of 100 iterations, 256 x 256 rectangles 4.21 -> 3.88 ms, 201 x 143
// quadrilaterals 2.84 -> 2.55, 96 x 80 BBM 3.01 -> 2.90.
// Arguments outside [2^-120, 2^120], negative or NaN take CUDA's own functions.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#define NSDG_SEED_HD __host__ __device__ __forceinline__
#else
#define NSDG_SEED_HD inline
#endif

namespace nsdg {
namespace sf {

namespace seed {
NSDG_SEED_HD uint64_t bitsOf(double d)
{
#if defined(__CUDA_ARCH__)
    return static_cast<uint64_t>(__double_as_longlong(d));
#else
    uint64_t u;
    std::memcpy(&u, &d, sizeof u);
    return u;
#endif
}
NSDG_SEED_HD double doubleOf(uint64_t u)
{
#if defined(__CUDA_ARCH__)
    return __longlong_as_double(static_cast<long long>(u));
#else
    double d;
    std::memcpy(&d, &u, sizeof d);
    return d;
#endif
}
NSDG_SEED_HD uint32_t bitsOf(float f)
{
#if defined(__CUDA_ARCH__)
    return __float_as_uint(f);
#else
    uint32_t u;
    std::memcpy(&u, &f, sizeof u);
    return u;
#endif
}
NSDG_SEED_HD float floatOf(uint32_t u)
{
#if defined(__CUDA_ARCH__)
    return __uint_as_float(u);
#else
    float f;
    std::memcpy(&f, &u, sizeof f);
    return f;
#endif
}
// FP32 operations rounded one by one
NSDG_SEED_HD float mulF(float a, float b)
{
#if defined(__CUDA_ARCH__)
    return __fmul_rn(a, b);
#else
    return a * b;
#endif
}
NSDG_SEED_HD float subF(float a, float b)
{
#if defined(__CUDA_ARCH__)
    return __fsub_rn(a, b);
#else
    return a - b;
#endif
}
NSDG_SEED_HD int roundF(float a)
{
#if defined(__CUDA_ARCH__)
    return __float2int_rn(a);
#else
    return static_cast<int>(std::lrintf(a));
#endif
}

// the significand of t in [1, 2) (odd: [2, 4)) as floats hi + lo
NSDG_SEED_HD float high(uint64_t t, unsigned odd)
{
    return floatOf((static_cast<uint32_t>(t >> 29) & 0x7fffffu) | ((127u + odd) << 23));
}
NSDG_SEED_HD float low(uint64_t t, unsigned odd)
{
    return mulF(static_cast<float>(static_cast<int>(t & 0x1fffffffu)), odd ? 0x1p-51f : 0x1p-52f);
}
// the approximation, held in [1/2, 1] (one binade of the sum below)
NSDG_SEED_HD float heldIn(float s) { return fminf(fmaxf(s, 0.5f), 1.f); }
// seed + correction, seed in [1/2, 1], |correction| < 2^-21, times 2^-k
NSDG_SEED_HD double join(float s, float c, int k)
{
    const int64_t v = static_cast<int64_t>((static_cast<uint64_t>(bitsOf(s)) << 29) + (896ull << 52))
        + 2 * static_cast<int64_t>(roundF(mulF(c, 0x1p52f)));
    return doubleOf(static_cast<uint64_t>(v) - (static_cast<uint64_t>(static_cast<int64_t>(k)) << 52));
}
// 1/d to 46 bits from s ~ 1/m, m the significand of d
NSDG_SEED_HD double reciprocal(uint64_t d, float hi, float s)
{
    s = heldIn(s);
    const float q = mulF(hi, s), qe = fmaf(hi, s, -q);
    const float e = fmaf(-low(d, 0), s, subF(subF(1.f, q), qe));
    const float c = mulF(s, e);
    return join(s, fmaf(c, e, c), static_cast<int>(d >> 52) - 1023);
}
// 1/sqrt(t) to 46 bits from s ~ 1/sqrt(m), m the significand in [1, 4)
NSDG_SEED_HD double rsqrt(uint64_t t, float hi, unsigned odd, float s)
{
    s = heldIn(s);
    const float p = mulF(s, s), pe = fmaf(s, s, -p);
    const float q = mulF(hi, p), qe = fmaf(hi, p, -q);
    const float e = fmaf(-low(t, odd), p, fmaf(-hi, pe, subF(subF(1.f, q), qe)));
    const int k = (static_cast<int>(t >> 52) - 1023 - static_cast<int>(odd)) / 2;
    return join(s, mulF(mulF(s, e), fmaf(0.375f, e, 0.5f)), k);
}
NSDG_SEED_HD unsigned oddOf(uint64_t t) { return (static_cast<unsigned>(t >> 52) & 1u) ^ 1u; }
// the FP64 steps
NSDG_SEED_HD double finishReciprocal(double d, double r) { return fma(r, fma(-d, r, 1.0), r); }
NSDG_SEED_HD double halfOf(double y) { return doubleOf(bitsOf(y) - (1ull << 52)); }
NSDG_SEED_HD double finishSqrt(double t, double y)
{
    const double h = t * y;
    return fma(fma(-h, h, t), halfOf(y), h);
}
NSDG_SEED_HD double finishTimesRsqrt(double p, double t, double y)
{
    const double h = t * y, z = p * y;
    return fma(z, fma(-h, halfOf(y), 0.5), z);
}
} // namespace seed

#if defined(__CUDACC__)
// t in [2^-120, 2^120]
__device__ __forceinline__ bool seedRange(double t)
{
    const unsigned h = static_cast<unsigned>(__double2hiint(t));
    return h - ((1023u - 120u) << 20) < (240u << 20);
}

static __device__ __noinline__ double recipSlow(double d) { return 1.0 / d; }
static __device__ __noinline__ double sqrtSlow(double t) { return sqrt(t); }
static __device__ __noinline__ double rsqrtSlow(double t) { return rsqrt(t); }

__device__ __forceinline__ double rsqrtSeed(double t)
{
    const uint64_t b = seed::bitsOf(t);
    const unsigned odd = seed::oddOf(b);
    const float hi = seed::high(b, odd);
    return seed::rsqrt(b, hi, odd, rsqrtf(hi));
}
__device__ __forceinline__ double recip64(double d)
{
    if (!seedRange(d))
        return recipSlow(d);
    const uint64_t b = seed::bitsOf(d);
    const float hi = seed::high(b, 0);
    return seed::finishReciprocal(d, seed::reciprocal(b, hi, __fdividef(1.f, hi)));
}
__device__ __forceinline__ double sqrt64(double t)
{
    return seedRange(t) ? seed::finishSqrt(t, rsqrtSeed(t)) : sqrtSlow(t);
}
// p / sqrt(t)
__device__ __forceinline__ double timesRsqrt64(double p, double t)
{
    return seedRange(t) ? seed::finishTimesRsqrt(p, t, rsqrtSeed(t)) : p * rsqrtSlow(t);
}
#endif

} // namespace sf
} // namespace nsdg
