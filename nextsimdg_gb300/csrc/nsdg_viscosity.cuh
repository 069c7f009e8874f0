// nsdg_viscosity.cuh — P/(8 alpha Delta) of the mixed-precision mEVP kernels.
#pragma once

#include "nsdg_visc_ff.hpp"

namespace nsdg {
namespace {

// float <-> double by exponent rebiasing on the integer pipe (GB300 executes
// FP64 at about 1/60 of its FP32 rate): exact for positive normal
// floats; a value below the smallest normal float maps to zero.
__device__ __forceinline__ double widenPos(float f)
{
    const unsigned long long b = (static_cast<unsigned long long>(__float_as_uint(f)) << 29) + (896ull << 52);
    return __longlong_as_double(static_cast<long long>(b));
}
// f / 2 for a positive normal float f (exact)
__device__ __forceinline__ double widenHalfPos(float f)
{
    const unsigned long long b = (static_cast<unsigned long long>(__float_as_uint(f)) << 29) + (895ull << 52);
    return __longlong_as_double(static_cast<long long>(b));
}
__device__ __forceinline__ double widenNonneg(float f)
{
    return __float_as_uint(f) >= 0x00800000u ? widenPos(f) : 0.0;
}
// d >= 0 and below 2^128: nearest float (ties away from zero); 0 below the
// smallest normal float
__device__ __forceinline__ float narrowPos(double d)
{
    const long long b = __double_as_longlong(d);
    const long long r = (b - (896ll << 52) + (1ll << 28)) >> 29;
    return b >= (897ll << 52) ? __uint_as_float(static_cast<unsigned>(r)) : 0.f;
}
// P/(8 alpha Delta) with Delta = sqrt(t), t = inv + DeltaMin^2 formed in FP64
// with one rounding (FMA), evaluated in FP64.  VM 0: CUDA's rsqrt(double).
// VM 1 and 2: one Newton-Raphson step for the reciprocal square root,
// y1 = y0 + y0 (1 - t y0^2) / 2, in FP64 from the FP32 seed
// y0 = rsqrtf(inv + DeltaMin^2) (relative error of y1: 1.5 e0^2 + FP64
// rounding, e0 <= 2^-21 for the seed and its FP32 argument, i.e. below
// 1e-12); VM 2 converts between float and double on the integer pipe (y0/2
// by the exponent bias).  Five FP64 instructions per Gauss point in VM 2.
// VM 3: the same Newton step from the same seed with float pairs on the FP32
// pipe (nsdg_visc_ff.hpp: one FP64 subtraction per Gauss point; dmin2lo is
// the low part of DeltaMin^2).  VM 4: VM 3's float pairs with the check of
// nsdg_ff::viscFloatFloatChecked, and VM 2's FP64 operations from the same
// seed wherever the check cannot prove the pair's rounding equal to theirs
// (near a float rounding boundary: about 1e-4 of the Gauss points): bitwise
// VM 2's result with one FP64 subtraction per Gauss point instead of five
// FP64 instructions.
//
// The sum-factorised kernels' default is VM 3 with the numerator given as a
// pair of floats (nsdg_ff::viscPair: no FP64 instruction).  Against extended
// precision its RMS error is VM 2's to nine digits (0.2887 ulp, both round an
// approximation far below the float's last place; they differ in 1e-7 of the
// cases).  512 x 512 parallelograms, launch included: 12.3 us (one thread
// per element), VM 4 26.7 us, VM 2 39.0 us (FP64 issue, the pair's sum included), VM
// 0 and 1 57.4 us (three threads).
__device__ __forceinline__ float viscNewton64(float inv, double Pa, double dmin, float y0)
{
    const double t = fma(dmin, dmin, widenNonneg(inv));
    const double yd = widenPos(y0);
    const double h = t * yd;
    const double e2 = fma(-h, widenHalfPos(y0), 0.5); // (1 - t y0^2) / 2
    const double z = Pa * yd;
    return narrowPos(fma(z, e2, z));
}

template <int VM>
__device__ __forceinline__ float viscosity8(float inv, double Pa, double dmin, float dmin2f, float dmin2lo)
{
    if constexpr (VM == 3) {
        return nsdg_ff::viscFloatFloat(inv, Pa, dmin2f, dmin2lo, rsqrtf(inv + dmin2f));
    } else if constexpr (VM == 4) {
        const float y0 = rsqrtf(inv + dmin2f);
        bool exact;
        const float z = nsdg_ff::viscFloatFloatChecked(inv, Pa, dmin2f, dmin2lo, y0, exact);
        return exact ? z : viscNewton64(inv, Pa, dmin, y0);
    } else {
        const double td = VM == 2 ? widenNonneg(inv) : static_cast<double>(inv);
        const double t = fma(dmin, dmin, td);
        if constexpr (VM == 0) {
            return static_cast<float>(Pa * rsqrt(t));
        } else {
            const float y0 = rsqrtf(inv + dmin2f);
            const double yd = VM == 1 ? static_cast<double>(y0) : widenPos(y0);
            const double yh = VM == 1 ? 0.5 * yd : widenHalfPos(y0);
            const double h = t * yd;
            const double e2 = fma(-h, yh, 0.5); // (1 - t y0^2) / 2
            const double z = Pa * yd;
            const double z8 = fma(z, e2, z);
            return VM == 1 ? static_cast<float>(z8) : narrowPos(z8);
        }
    }
}

} // namespace
} // namespace nsdg
