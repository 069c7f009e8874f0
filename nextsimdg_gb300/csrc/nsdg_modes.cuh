// nsdg_modes.cuh — FP64 values of a DG expansion at tensor points, and back,
// by 1-D factors: Legendre modes 1, x, x^2 - 1/12 per direction (x from the
// cell's centre), the DG modes (dgVector.hpp, basisfunctions.py:33-52) their
// products 1, x, y, L2(x), L2(y), xy, L2(x) y, x L2(y).  18 FP64 instructions
// for nine values of a DG2 field where the dense product takes 54.
#pragma once

namespace nsdg {
namespace sf {

constexpr double kGauss3 = 0.38729833462074168852; // sqrt(3/20)

// values at the points -+h and 0 of each direction; L2H = h^2 - 1/12
template <int DG, bool LAGRANGE> __device__ __forceinline__ void valuesAt(const double (&c)[DG], double (&v)[9])
{
    constexpr double h = LAGRANGE ? 0.5 : kGauss3;
    constexpr double l2 = LAGRANGE ? 1. / 6. : 0.15 - 1. / 12.;
    constexpr double l0 = -1. / 12.;
    auto along = [&](double c0, double c1, double c2, double (&o)[3]) {
        const double m = fma(l2, c2, c0);
        o[0] = fma(-h, c1, m);
        o[1] = fma(l0, c2, c0);
        o[2] = fma(h, c1, m);
    };
    if constexpr (DG == 1) {
#pragma unroll
        for (int q = 0; q < 9; ++q)
            v[q] = c[0];
    } else if constexpr (DG == 3) {
        const double r[3] = { fma(-h, c[2], c[0]), c[0], fma(h, c[2], c[0]) };
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            v[3 * k] = fma(-h, c[1], r[k]);
            v[3 * k + 1] = r[k];
            v[3 * k + 2] = fma(h, c[1], r[k]);
        }
    } else {
        double c0[3], c1[3], c2[3];
        along(c[0], c[2], c[4], c0);
        if constexpr (DG == 8) {
            along(c[1], c[5], c[7], c1);
            c2[0] = fma(-h, c[6], c[3]);
            c2[1] = c[3];
            c2[2] = fma(h, c[6], c[3]);
        } else {
            c1[0] = fma(-h, c[5], c[1]);
            c1[1] = c[1];
            c1[2] = fma(h, c[5], c[1]);
            c2[0] = c2[1] = c2[2] = c[3];
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            double o[3];
            along(c0[k], c1[k], c2[k], o);
#pragma unroll
            for (int i = 0; i < 3; ++i)
                v[3 * k + i] = o[i];
        }
    }
}
template <int DG> __device__ __forceinline__ void gaussValues(const double (&c)[DG], double (&v)[9])
{
    valuesAt<DG, false>(c, v);
}
template <int DG> __device__ __forceinline__ void lagrangeValues(const double (&c)[DG], double (&v)[9])
{
    valuesAt<DG, true>(c, v);
}

// the first DG modes of the biquadratic through nine Gauss-point values
template <int DG> __device__ __forceinline__ void modesOf(const double (&v)[9], double (&c)[DG])
{
    auto along = [&](double v0, double v1, double v2, double (&o)[3]) {
        const double t = fma(-2.0, v1, v0 + v2);
        o[0] = fma(5. / 18., t, v1);
        o[1] = (0.5 / kGauss3) * (v2 - v0);
        o[2] = (0.5 / (kGauss3 * kGauss3)) * t;
    };
    double r[3][3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
        along(v[3 * k], v[3 * k + 1], v[3 * k + 2], r[k]);
    double a[3];
    along(r[0][0], r[1][0], r[2][0], a);
    c[0] = a[0];
    if constexpr (DG >= 3)
        c[2] = a[1];
    if constexpr (DG >= 6)
        c[4] = a[2];
    if constexpr (DG >= 3) {
        along(r[0][1], r[1][1], r[2][1], a);
        c[1] = a[0];
        if constexpr (DG >= 6)
            c[5] = a[1];
        if constexpr (DG == 8)
            c[7] = a[2];
    }
    if constexpr (DG >= 6) {
        along(r[0][2], r[1][2], r[2][2], a);
        c[3] = a[0];
        if constexpr (DG == 8)
            c[6] = a[1];
    }
}

// clamps by the bit pattern (an FP64 minimum or maximum issues at the FP64
// rate); NaN gives the bound that fmax(x, lo) or fmin(x, hi) would
__device__ __forceinline__ bool isNan64(double x)
{
    return (__double_as_longlong(x) & 0x7fffffffffffffffll) > 0x7ff0000000000000ll;
}
__device__ __forceinline__ double atLeast(double x, double lo) // lo >= 0
{
    return isNan64(x) || __double_as_longlong(x) < __double_as_longlong(lo) ? lo : x;
}
__device__ __forceinline__ double atMost(double x, double hi) // x >= 0
{
    return static_cast<unsigned long long>(__double_as_longlong(x))
            > static_cast<unsigned long long>(__double_as_longlong(hi))
        ? hi
        : x;
}

} // namespace sf
} // namespace nsdg
