// nsdg_sumfact.cuh — the mEVP element update by sum factorisation.
//
// The strain at the 3 x 3 Gauss points is the gradient of the element's
// biquadratic velocity, projected onto the 8 stress modes.  Its tensor
// structure makes every directional derivative a chain of 1-D operators on
// lines of three nodes, and the stress divergence the transposed chain, so an
// element needs the map's derivatives at the Gauss points instead of two
// 9 x 9 operators per direction and phase:
//
//   de/dx at point q     = (K u)(q) with K = (dxi/dx d_xi + deta/dx d_eta)
//   projected strain     = P K u,   P = Psi^T M8^{-1} Psi W  (W = w J [cos lat])
//   divergence share     = K^T P^T (w J f)
//
// The 8 modes leave out one of the 9 point values' degrees of freedom, so P
// differs from the identity by one rank: with nu = (1,-2,1) x (1,-2,1) (the
// point functional that vanishes on all 8 modes) and n = W^{-1} nu / (nu W^{-1} nu),
//   P g = g - n (nu . g),     P^T h = h - nu (n . h).
// On rectangles K u and K v lie in the 8 modes' span and P drops out of both
// phases (P is self-adjoint in W).  On a sphere x = lon, y = lat: K carries
// 1 / (R cos lat) and 1 / R, and the metric terms of the strain and of the
// divergence are point multiplications by m = tan(lat) / R.
//
// The 1-D maps are written for a type T.  FP64 issue bounds the FP64 kernels
// (GB300 issues FP64 at about 1/60 of its FP32 rate), so what counts there is
// the number of FP64 instructions: about 480 per element and iteration on
// rectangles and 720 on general quadrilaterals, against 850 with the 9 x 9
// operators.
//
// Half strains are used throughout: a = e11 / 2, b = e22 / 2, s = e12.
#pragma once

#include <cstddef>
#include <cstdint>

#include "nsdg_kernels.hpp"
#include "nsdg_seed64.cuh"

namespace nsdg {
namespace sf {

// Gauss points 1/2 -+ kG on a line of nodes 0, 1/2, 1: with d = a2 - a0 and
// e = a0 + a2 - 2 a1 the quadratic through the nodes is
// a1 + d x + 2 e x^2 (x from the centre): values a1 + 0.3 e -+ kG d,
// derivatives d -+ 4 kG e.
template <typename T> struct Line {
    static constexpr T g = T(0.38729833462074168852); // sqrt(3/20)
    static constexpr T g4 = T(1.54919333848296675407);
    static constexpr T c3 = T(0.3), c4 = T(0.4);
};

__device__ __forceinline__ double fmaT(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float fmaT(float a, float b, float c) { return fmaf(a, b, c); }

// values at the three Gauss points of a line from its nodes
template <typename T> __device__ __forceinline__ void interp(const T (&n)[3], T (&o)[3])
{
    const T d = n[2] - n[0];
    const T e = fmaT(T(-2), n[1], n[2] + n[0]);
    const T m = fmaT(Line<T>::c3, e, n[1]);
    o[0] = fmaT(-Line<T>::g, d, m);
    o[1] = n[1];
    o[2] = fmaT(Line<T>::g, d, m);
}
// derivatives
template <typename T> __device__ __forceinline__ void deriv(const T (&n)[3], T (&o)[3])
{
    const T d = n[2] - n[0];
    const T e = fmaT(T(-2), n[1], n[2] + n[0]);
    o[0] = fmaT(-Line<T>::g4, e, d);
    o[1] = d;
    o[2] = fmaT(Line<T>::g4, e, d);
}
// both
template <typename T> __device__ __forceinline__ void interpDeriv(const T (&n)[3], T (&v)[3], T (&dv)[3])
{
    const T d = n[2] - n[0];
    const T e = fmaT(T(-2), n[1], n[2] + n[0]);
    const T m = fmaT(Line<T>::c3, e, n[1]);
    v[0] = fmaT(-Line<T>::g, d, m);
    v[1] = n[1];
    v[2] = fmaT(Line<T>::g, d, m);
    dv[0] = fmaT(-Line<T>::g4, e, d);
    dv[1] = d;
    dv[2] = fmaT(Line<T>::g4, e, d);
}
// the transposed maps: three point values to three nodes
template <typename T> __device__ __forceinline__ void interpT(const T (&t)[3], T (&o)[3])
{
    const T s = t[0] + t[2], d = t[2] - t[0];
    const T m = Line<T>::c3 * s;
    o[0] = fmaT(-Line<T>::g, d, m);
    o[1] = fmaT(Line<T>::c4, s, t[1]);
    o[2] = fmaT(Line<T>::g, d, m);
}
template <typename T> __device__ __forceinline__ void derivT(const T (&t)[3], T (&o)[3])
{
    const T s = t[0] + t[1] + t[2];
    const T k = Line<T>::g4 * (t[2] - t[0]);
    o[0] = k - s;
    o[1] = T(-2) * k;
    o[2] = k + s;
}
// interp and interpT times a factor r, with r g, 0.3 r and 0.4 r given
template <typename T> struct Scaled {
    T r, g, c3, c4;
    __device__ __forceinline__ explicit Scaled(T f) : r(f), g(Line<T>::g * f), c3(Line<T>::c3 * f), c4(Line<T>::c4 * f) { }
    __device__ __forceinline__ void interp(const T (&n)[3], T (&o)[3]) const
    {
        const T d = n[2] - n[0];
        const T e = fmaT(T(-2), n[1], n[2] + n[0]);
        o[1] = r * n[1];
        const T m = fmaT(c3, e, o[1]);
        o[0] = fmaT(-g, d, m);
        o[2] = fmaT(g, d, m);
    }
    __device__ __forceinline__ void interpT(const T (&t)[3], T (&o)[3]) const
    {
        const T s = t[0] + t[2], d = t[2] - t[0];
        const T m = c3 * s;
        o[0] = fmaT(-g, d, m);
        o[1] = fmaT(c4, s, r * t[1]);
        o[2] = fmaT(g, d, m);
    }
};

// The transposed eta maps of one column of nodes: x[r] (to the transposed
// interpolation) and y[r] (to the transposed derivative) from the Gauss rows
// r = 0, 1, 2; o[r] is the node in row r.
template <typename T> __device__ __forceinline__ void columnT(const T (&x)[3], const T (&y)[3], T (&o)[3])
{
    const T sx = x[2] + x[0], dx = x[2] - x[0];
    const T sy = y[2] + y[0], k = Line<T>::g4 * (y[2] - y[0]);
    const T p = fmaT(Line<T>::c3, sx, k);
    const T q = fmaT(Line<T>::g, dx, sy + y[1]);
    o[0] = p - q;
    o[1] = fmaT(T(-2), k, fmaT(Line<T>::c4, sx, x[1]));
    o[2] = p + q;
}

// -x / 2 for x >= 0 (subnormal results flushed to zero), on the integer pipe
__device__ __forceinline__ double minusHalf(double x)
{
    const int hi = __double2hiint(x);
    return hi >= (2 << 20) ? __hiloint2double((hi - (1 << 20)) | static_cast<int>(0x80000000u), __double2loint(x)) : 0.0;
}

// The stress increments (times the weight in pq) of one Gauss point:
// f11, f12, f22 of P/(8 alpha Delta) (5 e11 + 3 e22) - P/(2 alpha) etc. from
// a = e11/2, b = e22/2, s = e12 and Delta^2 = DeltaMin^2 + 4 (a + b)^2 + (a - b)^2 + s^2
// (MEVPStressUpdateStep.hpp:63-77, 80-116).  dminQ = DeltaMin^2 / 4.
__device__ __forceinline__ void pointStress64(double a, double b, double s, double pq, double dminQ, double& f11,
    double& f12, double& f22)
{
    const double pl = a + b, mi = a - b;
    const double t = fma(4.0, fma(pl, pl, dminQ), fma(mi, mi, s * s));
    const double z = timesRsqrt64(pq, t); // 2 P / (8 alpha Delta), weighted
    const double w = fma(z, pl, minusHalf(pq));
    const double d = z * mi;
    f12 = z * s;
    f11 = fma(4.0, w, d);
    f22 = fma(4.0, w, -d);
}

// How an element's map is given.
enum Geometry { RECT = 0, QUAD = 1, SPHERE = 2 };

} // namespace sf
} // namespace nsdg
