// nsdg_seed64.cuh — FP64 reciprocals and square roots from FP32 seeds.
//
// GB300 issues FP64 at about 1/60 of its FP32 rate, and CUDA's double
// division, sqrt and rsqrt take 10 to 20 FP64 instructions in one dependent
// chain.  Here the seed is the FP32 approximation of the truncated argument
// (relative error below 2^-21) and one step of the convergent series in the
// residual e follows, cut off below 2^-60:
//   1/d      = r (1 + e + e^2 + ...),         e = 1 - d r
//   1/sqrt t = y (1 + e/2 + 3/8 e^2 + ...),   e = 1 - t y^2
// three FP64 instructions for a reciprocal, five for a square root.  The
// conversions rebias exponents on the integer pipe.  Arguments that a normal
// float seed does not cover (outside [2^-120, 2^120], negative, NaN) take
// CUDA's own functions.
#pragma once

namespace nsdg {
namespace sf {

__device__ __forceinline__ double widenSeed(float f)
{
    return __longlong_as_double(
        static_cast<long long>((static_cast<unsigned long long>(__float_as_uint(f)) << 29) + (896ull << 52)));
}
// the float at or below t, for 2^-120 <= t <= 2^120
__device__ __forceinline__ float narrowSeed(double t)
{
    const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(t));
    return __uint_as_float(static_cast<unsigned>((b - (896ull << 52)) >> 29));
}
// t in [2^-120, 2^120]
__device__ __forceinline__ bool seedRange(double t)
{
    const unsigned h = static_cast<unsigned>(__double2hiint(t));
    return h - ((1023u - 120u) << 20) < (240u << 20);
}

static __device__ __noinline__ double recipSlow(double d) { return 1.0 / d; }
static __device__ __noinline__ double sqrtSlow(double t) { return sqrt(t); }
static __device__ __noinline__ double rsqrtSlow(double t) { return rsqrt(t); }

__device__ __forceinline__ double recip64(double d)
{
    if (!seedRange(d))
        return recipSlow(d);
    const double r = widenSeed(__fdividef(1.f, narrowSeed(d)));
    const double e = fma(-d, r, 1.0);
    return fma(r, fma(e, e, e), r);
}
__device__ __forceinline__ double sqrt64(double t)
{
    if (!seedRange(t))
        return sqrtSlow(t);
    const double y = widenSeed(rsqrtf(narrowSeed(t)));
    const double h = t * y;
    const double e = fma(-h, y, 1.0);
    return fma(h, e * fma(0.375, e, 0.5), h);
}
// p / sqrt(t)
__device__ __forceinline__ double timesRsqrt64(double p, double t)
{
    if (!seedRange(t))
        return p * rsqrtSlow(t);
    const double y = widenSeed(rsqrtf(narrowSeed(t)));
    const double h = t * y;
    const double e = fma(-h, y, 1.0);
    const double z = p * y;
    return fma(z, e * fma(0.375, e, 0.5), z);
}

} // namespace sf
} // namespace nsdg
