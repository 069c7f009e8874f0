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
// The FP32 kernels use the 1-D maps below; the FP64 ones run them in fixed point
// (nsdg_stress_fixed.cuh).
//
// Half strains are used throughout: a = e11 / 2, b = e22 / 2, s = e12.
#pragma once

#include <cstddef>
#include <cstdint>

#include "nsdg_fixed_rows.hpp"
#include "nsdg_kernels.hpp"
#include "nsdg_pdl.cuh"
#include "nsdg_seed64.cuh"
#include "nsdg_viscosity.cuh"

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
// a product that is never fused with a following sum: every arrangement of an
// element's work over threads then rounds alike
__device__ __forceinline__ double mulT(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mulT(float a, float b) { return __fmul_rn(a, b); }

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
    const T m = mulT(Line<T>::c3, s);
    o[0] = fmaT(-Line<T>::g, d, m);
    o[1] = fmaT(Line<T>::c4, s, t[1]);
    o[2] = fmaT(Line<T>::g, d, m);
}
template <typename T> __device__ __forceinline__ void derivT(const T (&t)[3], T (&o)[3])
{
    const T s = t[0] + t[1] + t[2];
    const T k = mulT(Line<T>::g4, t[2] - t[0]);
    o[0] = k - s;
    o[1] = mulT(T(-2), k);
    o[2] = k + s;
}
// The transposed eta maps of one column of nodes: x[r] (to the transposed
// interpolation) and y[r] (to the transposed derivative) from the Gauss rows
// r = 0, 1, 2; o[r] is the node in row r.
template <typename T> __device__ __forceinline__ void columnT(const T (&x)[3], const T (&y)[3], T (&o)[3])
{
    const T sx = x[2] + x[0], dx = x[2] - x[0];
    const T sy = y[2] + y[0], k = mulT(Line<T>::g4, y[2] - y[0]);
    const T p = fmaT(Line<T>::c3, sx, k);
    const T q = fmaT(Line<T>::g, dx, sy + y[1]);
    o[0] = p - q;
    o[1] = fmaT(T(-2), k, fmaT(Line<T>::c4, sx, x[1]));
    o[2] = p + q;
}

// What the stress increments take besides the strain: the weighted pressure
// pq = w P / (4 alpha) (FP32 kernels: as a pair of floats, 48 bits) and
// DeltaMin^2.
template <typename T> struct Rheology;
template <> struct Rheology<float> {
    using Weight = float2;
    float d2h, d2l; // DeltaMin^2 as a pair of floats
    double dmin;
    static __device__ __forceinline__ float2 none() { return make_float2(0.f, 0.f); }
};

// The stress increments (times the weight in pq) of one Gauss point:
// f11, f12, f22 of P/(8 alpha Delta) (5 e11 + 3 e22) - P/(2 alpha) etc. from
// a = e11/2, b = e22/2, s = e12 and Delta^2 = DeltaMin^2 + 4 (a + b)^2 + (a - b)^2 + s^2
// (MEVPStressUpdateStep.hpp:63-77, 80-116).
// FP32: the invariant is a sum of squares (no cancellation); Delta^2 and the
// viscosity in float pairs (VM 3, the default) or in FP64 (VM 0, 1, 2; 4 is
// 3 checked against 2)
template <int VM>
__device__ __forceinline__ void pointStress(float a, float b, float s, float2 pq, const Rheology<float>& rh,
    float& f11, float& f12, float& f22)
{
    const float pl = a + b, mi = a - b;
    const float inv = fmaf(mulT(4.f, pl), pl, fmaf(mi, mi, mulT(s, s)));
    float z;
    if constexpr (VM == 3)
        z = nsdg_ff::viscPair(inv, pq.x, pq.y, rh.d2h, rh.d2l, rsqrtf(inv + rh.d2h));
    else
        z = viscosity8<VM>(inv, static_cast<double>(pq.x) + static_cast<double>(pq.y), rh.dmin, rh.d2h, rh.d2l);
    const float w = fmaf(z, pl, mulT(-0.5f, pq.x));
    const float d = mulT(z, mi);
    f12 = mulT(z, s);
    f11 = fmaf(4.f, w, d);
    f22 = fmaf(4.f, w, -d);
}

// One mEVP iteration in divergence space: tdiv <- (1 - 1/alpha) tdiv +
// K^T P^T f(P K u).  Three threads per element, in three warps of a block of
// E elements: warp R takes node column R (the eta maps of its three
// nodes), then Gauss row R (the xi maps, strain, stress increments, the
// transposed xi maps), then node column R again (the transposed eta maps); the
// 24 and 36 values in between go through shared memory, as do the sums of the
// two projections on general quadrilaterals.
//
template <typename T, int E> struct Exchange {
    union {
        struct {
            T v[2][3][3][E];  // [u, v][Gauss row][column]: values on the columns
            T dv[2][3][3][E]; // eta derivatives
        } in;
        struct {
            T x[2][3][3][E]; // to the transposed interpolation
            T y[2][3][3][E]; // to the transposed derivative
        } out;
    };
};

// sum over the element's three warps of each thread's c[0..2]
template <typename T, int E>
__device__ __forceinline__ void sumRows(T (*part)[3][E], int R, int le, T (&c)[3])
{
#pragma unroll
    for (int k = 0; k < 3; ++k)
        part[R][k][le] = c[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 3; ++k)
        c[k] = part[0][k][le] + part[1][k][le] + part[2][k][le];
}

template <typename T, Geometry GEO, int VM, int E>
__device__ __forceinline__ void gaussRow(int R, bool active, size_t e, size_t N, const StressGeometry<T>& geo,
    const typename Rheology<T>::Weight (&pq)[3], const T (&ke)[4], const Rheology<T>& rh, Exchange<T, E>& ex,
    T (*sums)[3][3][E], int le)
{
    T I[3], D[3], uxi[3], uet[3], vxi[3], vet[3], f11[3], f12[3], f22[3], x[3], y[3];
    [[maybe_unused]] T up[3], vp[3];
    auto take = [&](int c) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            I[i] = ex.in.v[c][R][i][le];
            D[i] = ex.in.dv[c][R][i][le];
        }
    };
    take(0);
    deriv(I, uxi);
    interp(D, uet);
    if constexpr (GEO == SPHERE)
        interp(I, up);
    take(1);
    deriv(I, vxi);
    interp(D, vet);
    if constexpr (GEO == SPHERE)
        interp(I, vp);
    if constexpr (GEO == AFFINE) {
#pragma unroll
        for (int i = 0; i < 3; ++i)
            pointStress<VM>(fmaT(ke[0], uxi[i], mulT(ke[1], uet[i])), fmaT(ke[2], vxi[i], mulT(ke[3], vet[i])),
                fmaT(ke[2], uxi[i], fmaT(ke[3], uet[i], fmaT(ke[0], vxi[i], mulT(ke[1], vet[i])))), pq[i], rh, f11[i],
                f12[i], f22[i]);
        __syncthreads();
        auto put = [&](int c, const T (&f)[3], const T (&h)[3]) {
            T p[3], q[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                p[i] = fmaT(ke[0], f[i], mulT(ke[2], h[i]));
                q[i] = fmaT(ke[1], f[i], mulT(ke[3], h[i]));
            }
            derivT(p, x);
            interpT(q, y);
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                ex.out.x[c][R][i][le] = x[i];
                ex.out.y[c][R][i][le] = y[i];
            }
        };
        put(0, f11, f12);
        put(1, f12, f22);
    } else {
        T k0[3], k1[3], k2[3], k3[3], nq[3], a[3], b[3], s[3];
        [[maybe_unused]] T mq[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const size_t q = 3 * R + i;
            k0[i] = active ? geo.k[q * N + e] : T(0);
            k1[i] = active ? geo.k[(9 + q) * N + e] : T(0);
            k2[i] = active ? geo.k[(18 + q) * N + e] : T(0);
            k3[i] = active ? geo.k[(27 + q) * N + e] : T(0);
            nq[i] = active ? geo.n[q * N + e] : T(0);
            a[i] = fmaT(k0[i], uxi[i], mulT(k1[i], uet[i]));
            b[i] = fmaT(k2[i], vxi[i], mulT(k3[i], vet[i]));
            s[i] = fmaT(k2[i], uxi[i], fmaT(k3[i], uet[i], fmaT(k0[i], vxi[i], mulT(k1[i], vet[i]))));
            if constexpr (GEO == SPHERE) {
                mq[i] = active ? geo.m[q * N + e] : T(0);
                a[i] = fmaT(-mq[i], vp[i], a[i]);
                s[i] = fmaT(mq[i], up[i], s[i]);
            }
        }
        const T nr = R == 1 ? T(-2) : T(1); // nu on this row: nr, -2 nr, nr
        // P: subtract n (nu . g)
        T c[3] = { mulT(nr, fmaT(T(-2), a[1], a[0] + a[2])), mulT(nr, fmaT(T(-2), b[1], b[0] + b[2])),
            mulT(nr, fmaT(T(-2), s[1], s[0] + s[2])) };
        sumRows<T, E>(sums[0], R, le, c);
        T d[3] = { T(0), T(0), T(0) };
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            pointStress<VM>(fmaT(-c[0], nq[i], a[i]), fmaT(-c[1], nq[i], b[i]), fmaT(-c[2], nq[i], s[i]), pq[i], rh,
                f11[i], f12[i], f22[i]);
            d[0] = fmaT(nq[i], f11[i], d[0]);
            d[1] = fmaT(nq[i], f22[i], d[1]);
            d[2] = fmaT(nq[i], f12[i], d[2]);
        }
        // P^T: subtract nu (n . f)
        sumRows<T, E>(sums[1], R, le, d);
        T t0[3], t1[3], t2[3], t3[3];
        [[maybe_unused]] T mu[3], mv[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const T w = i == 1 ? T(-2) * nr : nr;
            f11[i] = fmaT(-w, d[0], f11[i]);
            f22[i] = fmaT(-w, d[1], f22[i]);
            f12[i] = fmaT(-w, d[2], f12[i]);
            t0[i] = fmaT(k0[i], f11[i], mulT(k2[i], f12[i]));
            t1[i] = fmaT(k1[i], f11[i], mulT(k3[i], f12[i]));
            t2[i] = fmaT(k0[i], f12[i], mulT(k2[i], f22[i]));
            t3[i] = fmaT(k1[i], f12[i], mulT(k3[i], f22[i]));
            if constexpr (GEO == SPHERE) {
                mu[i] = mulT(mq[i], f12[i]);
                mv[i] = mulT(-mq[i], f11[i]);
            }
        }
        auto put = [&](int c, const T (&tx)[3], const T (&ty)[3], [[maybe_unused]] const T (&tm)[3]) {
            derivT(tx, x);
            interpT(ty, y);
            if constexpr (GEO == SPHERE) {
                T z[3];
                interpT(tm, z);
#pragma unroll
                for (int i = 0; i < 3; ++i)
                    x[i] += z[i];
            }
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                ex.out.x[c][R][i][le] = x[i];
                ex.out.y[c][R][i][le] = y[i];
            }
        };
        if constexpr (GEO == SPHERE) {
            put(0, t0, t1, mu);
            put(1, t2, t3, mv);
        } else {
            put(0, t0, t1, t0);
            put(1, t2, t3, t2);
        }
    }
}

// The block of elements x0 .. x0 + E - 1 of a grid of nx cells per row.
// Launched as a programmatic dependent of the node kernel: what the previous
// two launches do not write is loaded before the wait (the divergence was
// written two launches ago by this kernel, and the node kernel in between,
// which waited for it, only reads it).
template <typename T, Geometry GEO, int VM, int E>
__device__ __forceinline__ void stressBlock(int nx, size_t N, const uint8_t* __restrict__ ice,
    const StressGeometry<T>& geo, const T* __restrict__ u, const T* __restrict__ v,
    const typename Rheology<T>::Weight* __restrict__ Pw, T* __restrict__ tdiv, const Rheology<T>& rh, T keep, size_t x0,
    Exchange<T, E>& ex, T (*sums)[3][3][E])
{
    const int le = threadIdx.x % E, R = threadIdx.x / E; // R is the same in a warp
    const size_t e = x0 + le;
    const bool active = e < N && ice[e];
    typename Rheology<T>::Weight pq[3];
    T told[6], ke[4] = { T(0), T(0), T(0), T(0) };
#pragma unroll
    for (int i = 0; i < 3; ++i)
        pq[i] = Rheology<T>::none();
    if (active) {
#pragma unroll
        for (int i = 0; i < 3; ++i)
            pq[i] = Pw[(3 * R + i) * N + e];
        if constexpr (GEO == AFFINE)
#pragma unroll
            for (int c = 0; c < 4; ++c)
                ke[c] = geo.k[c * N + e];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            told[r] = beforeWait(tdiv + (3 * r + R) * N + e);
            told[3 + r] = beforeWait(tdiv + (9 + 3 * r + R) * N + e);
        }
    }
    waitForPrevious();
    {
        T n[2][3] = { { T(0), T(0), T(0) }, { T(0), T(0), T(0) } };
        if (active) {
            const unsigned s2 = 2u * static_cast<unsigned>(nx) + 1u;
            const unsigned ix = static_cast<unsigned>(e) % static_cast<unsigned>(nx);
            const unsigned iy = static_cast<unsigned>(e) / static_cast<unsigned>(nx);
            const size_t base = 2 * size_t(s2) * iy + 2 * ix + R;
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                n[0][r] = afterWait(u + base + size_t(r) * s2);
                n[1][r] = afterWait(v + base + size_t(r) * s2);
            }
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            T vr[3], dr[3];
            interpDeriv(n[c], vr, dr);
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                ex.in.v[c][r][R][le] = vr[r];
                ex.in.dv[c][r][R][le] = dr[r];
            }
        }
    }
    __syncthreads();
    gaussRow<T, GEO, VM, E>(R, active, e, N, geo, pq, ke, rh, ex, sums, le);
    __syncthreads();
    if (!active)
        return;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        T x[3], y[3], o[3];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            x[r] = ex.out.x[c][r][R][le];
            y[r] = ex.out.y[c][r][R][le];
        }
        columnT(x, y, o);
#pragma unroll
        for (int r = 0; r < 3; ++r)
            tdiv[(9 * c + 3 * r + R) * N + e] = fmaT(told[3 * c + r], keep, o[r]);
    }
}

// The same update by one thread per element: no exchange through shared
// memory and one set of indices, about 950 instructions per element instead
// of 1,700 with three threads, at a third of the warps.  Bitwise the same
// results.
template <typename T, Geometry GEO, int VM>
__device__ __forceinline__ void stressThread(int nx, size_t N, const uint8_t* __restrict__ ice,
    const StressGeometry<T>& geo, const T* __restrict__ u, const T* __restrict__ v,
    const typename Rheology<T>::Weight* __restrict__ Pw, T* __restrict__ tdiv, const Rheology<T>& rh, T keep, size_t e)
{
    const bool active = e < N && ice[e];
    typename Rheology<T>::Weight pq[9];
    T told[18], ke[4];
    if (active) {
#pragma unroll
        for (int q = 0; q < 9; ++q)
            pq[q] = Pw[q * N + e];
        if constexpr (GEO == AFFINE)
#pragma unroll
            for (int c = 0; c < 4; ++c)
                ke[c] = geo.k[c * N + e];
#pragma unroll
        for (int j = 0; j < 18; ++j)
            told[j] = beforeWait(tdiv + j * N + e);
    }
    waitForPrevious();
    if (!active)
        return;
    T val[2][3][3], der[2][3][3]; // [u, v][Gauss row][column]
    {
        const unsigned s2 = 2u * static_cast<unsigned>(nx) + 1u;
        const unsigned ix = static_cast<unsigned>(e) % static_cast<unsigned>(nx);
        const unsigned iy = static_cast<unsigned>(e) / static_cast<unsigned>(nx);
        const size_t base = 2 * size_t(s2) * iy + 2 * ix;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const T* src = (c ? v : u) + base;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const T n[3] = { afterWait(src + i), afterWait(src + s2 + i), afterWait(src + 2 * s2 + i) };
                T vr[3], dr[3];
                interpDeriv(n, vr, dr);
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    val[c][r][i] = vr[r];
                    der[c][r][i] = dr[r];
                }
            }
        }
    }
    // strain, stress increments and the transposed xi maps; val and der then
    // hold what goes to the transposed interpolation and derivative along eta
    auto strainRow = [&](int r, const T (&k0)[3], const T (&k1)[3], const T (&k2)[3], const T (&k3)[3], T (&a)[3],
                         T (&b)[3], T (&s)[3]) {
        T uxi[3], uet[3], vxi[3], vet[3];
        deriv(val[0][r], uxi);
        interp(der[0][r], uet);
        deriv(val[1][r], vxi);
        interp(der[1][r], vet);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            a[i] = fmaT(k0[i], uxi[i], mulT(k1[i], uet[i]));
            b[i] = fmaT(k2[i], vxi[i], mulT(k3[i], vet[i]));
            s[i] = fmaT(k2[i], uxi[i], fmaT(k3[i], uet[i], fmaT(k0[i], vxi[i], mulT(k1[i], vet[i]))));
        }
        if constexpr (GEO == SPHERE) {
            T up[3], vp[3];
            interp(val[0][r], up);
            interp(val[1][r], vp);
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const T mq = geo.m[(3 * r + i) * N + e];
                a[i] = fmaT(-mq, vp[i], a[i]);
                s[i] = fmaT(mq, up[i], s[i]);
            }
        }
    };
    auto divergenceRow = [&](int r, const T (&k0)[3], const T (&k1)[3], const T (&k2)[3], const T (&k3)[3],
                             const T (&f11)[3], const T (&f12)[3], const T (&f22)[3]) {
        T t0[3], t1[3], t2[3], t3[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            t0[i] = fmaT(k0[i], f11[i], mulT(k2[i], f12[i]));
            t1[i] = fmaT(k1[i], f11[i], mulT(k3[i], f12[i]));
            t2[i] = fmaT(k0[i], f12[i], mulT(k2[i], f22[i]));
            t3[i] = fmaT(k1[i], f12[i], mulT(k3[i], f22[i]));
        }
        derivT(t0, val[0][r]);
        interpT(t1, der[0][r]);
        derivT(t2, val[1][r]);
        interpT(t3, der[1][r]);
        if constexpr (GEO == SPHERE) {
            T mu[3], mv[3], zu[3], zv[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const T mq = geo.m[(3 * r + i) * N + e];
                mu[i] = mulT(mq, f12[i]);
                mv[i] = mulT(-mq, f11[i]);
            }
            interpT(mu, zu);
            interpT(mv, zv);
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                val[0][r][i] += zu[i];
                val[1][r][i] += zv[i];
            }
        }
    };
    if constexpr (GEO == AFFINE) {
        const T k0[3] = { ke[0], ke[0], ke[0] }, k1[3] = { ke[1], ke[1], ke[1] };
        const T k2[3] = { ke[2], ke[2], ke[2] }, k3[3] = { ke[3], ke[3], ke[3] };
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            T a[3], b[3], s[3], f11[3], f12[3], f22[3];
            strainRow(r, k0, k1, k2, k3, a, b, s);
#pragma unroll
            for (int i = 0; i < 3; ++i)
                pointStress<VM>(a[i], b[i], s[i], pq[3 * r + i], rh, f11[i], f12[i], f22[i]);
            divergenceRow(r, k0, k1, k2, k3, f11, f12, f22);
        }
    } else {
        auto loadK = [&](int r, T (&k0)[3], T (&k1)[3], T (&k2)[3], T (&k3)[3]) {
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const size_t q = 3 * r + i;
                k0[i] = geo.k[q * N + e];
                k1[i] = geo.k[(9 + q) * N + e];
                k2[i] = geo.k[(18 + q) * N + e];
                k3[i] = geo.k[(27 + q) * N + e];
            }
        };
        T a[3][3], b[3][3], s[3][3], nq[3][3], ca[3], cb[3], cs[3];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            T k0[3], k1[3], k2[3], k3[3];
            loadK(r, k0, k1, k2, k3);
#pragma unroll
            for (int i = 0; i < 3; ++i)
                nq[r][i] = geo.n[(3 * r + i) * N + e];
            strainRow(r, k0, k1, k2, k3, a[r], b[r], s[r]);
            const T nr = r == 1 ? T(-2) : T(1);
            ca[r] = mulT(nr, fmaT(T(-2), a[r][1], a[r][0] + a[r][2]));
            cb[r] = mulT(nr, fmaT(T(-2), b[r][1], b[r][0] + b[r][2]));
            cs[r] = mulT(nr, fmaT(T(-2), s[r][1], s[r][0] + s[r][2]));
        }
        const T na = ca[0] + ca[1] + ca[2], nb = cb[0] + cb[1] + cb[2], ns = cs[0] + cs[1] + cs[2];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            ca[r] = cb[r] = cs[r] = T(0);
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                T f11, f12, f22;
                pointStress<VM>(fmaT(-na, nq[r][i], a[r][i]), fmaT(-nb, nq[r][i], b[r][i]),
                    fmaT(-ns, nq[r][i], s[r][i]), pq[3 * r + i], rh, f11, f12, f22);
                ca[r] = fmaT(nq[r][i], f11, ca[r]);
                cb[r] = fmaT(nq[r][i], f22, cb[r]);
                cs[r] = fmaT(nq[r][i], f12, cs[r]);
                a[r][i] = f11;
                b[r][i] = f22;
                s[r][i] = f12;
            }
        }
        const T da = ca[0] + ca[1] + ca[2], db = cb[0] + cb[1] + cb[2], ds = cs[0] + cs[1] + cs[2];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const T nr = r == 1 ? T(-2) : T(1);
            T k0[3], k1[3], k2[3], k3[3];
            loadK(r, k0, k1, k2, k3);
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const T w = i == 1 ? T(-2) * nr : nr;
                a[r][i] = fmaT(-w, da, a[r][i]);
                b[r][i] = fmaT(-w, db, b[r][i]);
                s[r][i] = fmaT(-w, ds, s[r][i]);
            }
            divergenceRow(r, k0, k1, k2, k3, a[r], s[r], b[r]);
        }
    }
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const T x[3] = { val[c][0][i], val[c][1][i], val[c][2][i] };
            const T y[3] = { der[c][0][i], der[c][1][i], der[c][2][i] };
            T o[3];
            columnT(x, y, o);
#pragma unroll
            for (int r = 0; r < 3; ++r)
                tdiv[(9 * c + 3 * r + i) * N + e] = fmaT(told[9 * c + 3 * r + i], keep, o[r]);
        }
}

} // namespace sf
} // namespace nsdg
