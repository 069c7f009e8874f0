// nsdg_stress_fixed.cuh — the FP64 mEVP element update (nsdg_sumfact.cuh) with
// its linear maps in 64-bit fixed point (nsdg_fixed.hpp).
//
// The strain's error against extended precision (velocities varying by 1 to
// 1e-6 of their size within an element, rectangles) is 0.35 to 0.5 of that of
// the maps in FP64.
//
// What stays in FP64 is the rheology, ten instructions per Gauss point, and
// the relaxation of the 18 divergence coefficients: 108 FP64 instructions per
// element where the maps in FP64 make it 480 on rectangles and 720 on
// quadrilaterals.
//
// Scales (one per element): the velocities are below 2^top and become integers
// below 2^bits; with V = 2^bits the maps stay within
//   columns    |v| <= 1.2 V, |dv| <= 6.2 V (second differences 25 V)
//   rectangles |strain| <= 7.3 (1 + rho) V        -> bits 58, less for large rho
//   else       products with k / 4: sums <= 7.6 V, the projection's functional
//              <= 122 V and the projected strain <= 130 V -> bits 55
// and the weighted pressure, F = its largest, bounds the stress increments
// (|2 zp -+ d| <= sqrt(5) pq, so |f11|, |f22| <= 4.3 F, |f12| <= F); through the
// transposed maps they stay within 56 (1 + rho) F.  On quadrilaterals they are
// within 22 F after the projection (F = 2^57: below 2^61.5), and after the
// products with k / 4 and a shift by 3 the maps stay within 38 F.
#pragma once

#include "nsdg_fixed.hpp"
#include "nsdg_kernels.hpp"
#include "nsdg_seed64.cuh"
#include "nsdg_sumfact.cuh"

namespace nsdg {
namespace sf {

template <Geometry GEO, int E> struct FixedShared {
    Exchange<fx::i64, E> ex;
    fx::i64 sums[GEO == RECT ? 1 : 2][3][3][E];
    int top[2][3][E];
};

// 2^top bounds a row's or a column's values
__device__ __forceinline__ int topOf(int magnitudeWord) { return magnitudeWord >> 20; }

// One Gauss point: zp = 2 z (a + b), d = z (a - b), f = z s with
// z = w P / (4 alpha Delta), from pl = 2 (a + b), mi = a - b, s; dmin2 = DeltaMin^2
__device__ __forceinline__ void pointStress64(double pl, double mi, double s, double pq, double dmin2, double& zp,
    double& d, double& f)
{
    const double t = fma(pl, pl, fma(mi, mi, fma(s, s, dmin2)));
    const double z = timesRsqrt64(pq, t);
    zp = z * pl;
    d = z * mi;
    f = z * s;
}

// The maps of Gauss row R (nothing on rectangles).
template <Geometry GEO> struct FixedMap {
    fx::Split k0[3], k1[3], k2[3], k3[3], n[3], m[3];
    __device__ __forceinline__ FixedMap(const FixedGeometry& geo, int R, size_t e, size_t N, bool active)
        : FixedMap([&](const fx::i64* p, int row) { return fx::unpacked(active ? p[size_t(row) * N + e] : 0); }, geo,
            3 * R)
    {
    }
    template <typename F>
    __device__ __forceinline__ FixedMap(F at, const FixedGeometry& geo, int q)
        : k0 { at(geo.k, q), at(geo.k, q + 1), at(geo.k, q + 2) }
        , k1 { at(geo.k, q + 9), at(geo.k, q + 10), at(geo.k, q + 11) }
        , k2 { at(geo.k, q + 18), at(geo.k, q + 19), at(geo.k, q + 20) }
        , k3 { at(geo.k, q + 27), at(geo.k, q + 28), at(geo.k, q + 29) }
        , n { at(geo.n, q), at(geo.n, q + 1), at(geo.n, q + 2) }
        , m { metric(at, geo, q), metric(at, geo, q + 1), metric(at, geo, q + 2) }
    {
    }
    template <typename F> static __device__ __forceinline__ fx::Split metric(F at, const FixedGeometry& geo, int q)
    {
        return GEO == SPHERE ? at(geo.m, q) : fx::Split(0);
    }
};
template <> struct FixedMap<RECT> {
    __device__ __forceinline__ FixedMap(const FixedGeometry&, int, size_t, size_t, bool) { }
};

// nu (1, -2 or 4) times t
__device__ __forceinline__ fx::i64 nuTimes(fx::i64 t, int f) { return f == 1 ? t : f == -2 ? -2 * t : fx::four(t); }

// The velocities n[u, v][row] of node column R through the eta maps.
template <int E>
__device__ __forceinline__ void fixedColumn(const double (&n)[2][3], int at, int R, int le, Exchange<fx::i64, E>& ex)
{
    using fx::i64;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const i64 a[3] = { fx::toFixed(n[c][0], at), fx::toFixed(n[c][1], at), fx::toFixed(n[c][2], at) };
        i64 val[3], der[3];
        fx::interp(a, val);
        fx::deriv(a, der);
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            ex.in.v[c][r][R][le] = val[r];
            ex.in.dv[c][r][R][le] = der[r];
        }
    }
}

// The half strains of Gauss row R (on quadrilaterals over 4 and projected; sums
// takes the three rows' parts of nu . g).
template <Geometry GEO, int E>
__device__ __forceinline__ void fixedStrain(int R, int le, const fx::Scaled& sc, const FixedMap<GEO>& map,
    const Exchange<fx::i64, E>& ex, fx::i64 (*sums)[3][E], fx::i64 (&a)[3], fx::i64 (&b)[3], fx::i64 (&s)[3])
{
    using fx::i64;
    i64 I[3], D[3], uxi[3], uet[3], vxi[3], vet[3];
    [[maybe_unused]] i64 up[3], vp[3];
    auto take = [&](int c) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            I[i] = ex.in.v[c][R][i][le];
            D[i] = ex.in.dv[c][R][i][le];
        }
    };
    take(0);
    fx::deriv(I, uxi);
    if constexpr (GEO == RECT)
        sc.interp(D, uet);
    else
        fx::interp(D, uet);
    if constexpr (GEO == SPHERE)
        fx::interp(I, up);
    take(1);
    fx::deriv(I, vxi);
    if constexpr (GEO == RECT)
        sc.interp(D, vet);
    else
        fx::interp(D, vet);
    if constexpr (GEO == SPHERE)
        fx::interp(I, vp);
    if constexpr (GEO == RECT) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            a[i] = uxi[i];
            b[i] = vet[i];
            s[i] = uet[i] + vxi[i];
        }
    } else {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const fx::Split ux(uxi[i]), ue(uet[i]), vx(vxi[i]), ve(vet[i]);
            a[i] = fx::mulHigh(ux, map.k0[i], ue, map.k1[i]);
            b[i] = fx::mulHigh(vx, map.k2[i], ve, map.k3[i]);
            s[i] = fx::mulHigh(ux, map.k2[i], ue, map.k3[i]) + fx::mulHigh(vx, map.k0[i], ve, map.k1[i]);
            if constexpr (GEO == SPHERE) {
                a[i] -= fx::mulHigh(fx::Split(vp[i]), map.m[i]);
                s[i] += fx::mulHigh(fx::Split(up[i]), map.m[i]);
            }
        }
        const int nr = R == 1 ? -2 : 1; // nu on this row: nr, -2 nr, nr
        // P: subtract n (nu . g)
        i64 c[3] = { nuTimes(a[0] + a[2] - 2 * a[1], nr), nuTimes(b[0] + b[2] - 2 * b[1], nr),
            nuTimes(s[0] + s[2] - 2 * s[1], nr) };
        sumRows<i64, E>(sums, R, le, c);
        const fx::Split c0(c[0]), c1(c[1]), c2(c[2]);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            a[i] -= fx::four(fx::mulHigh(c0, map.n[i]));
            b[i] -= fx::four(fx::mulHigh(c1, map.n[i]));
            s[i] -= fx::four(fx::mulHigh(c2, map.n[i]));
        }
    }
}

// Row R's stresses F through the transposed xi maps (on quadrilaterals times
// k / 4 and over 2^SHIFT).
template <Geometry GEO, int SHIFT, int E>
__device__ __forceinline__ void fixedShares(int R, int le, const fx::Scaled& sc, const FixedMap<GEO>& map,
    const fx::i64 (&F11)[3], const fx::i64 (&F12)[3], const fx::i64 (&F22)[3], Exchange<fx::i64, E>& ex)
{
    using fx::i64;
    auto put = [&](int c, const i64 (&tx)[3], const i64 (&ty)[3], [[maybe_unused]] const i64 (&tm)[3]) {
        i64 x[3], y[3];
        fx::derivT(tx, x);
        if constexpr (GEO == RECT)
            sc.interpT(ty, y);
        else
            fx::interpT(ty, y);
        if constexpr (GEO == SPHERE) {
            i64 z[3];
            fx::interpT(tm, z);
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
    if constexpr (GEO == RECT) {
        put(0, F11, F12, F11);
        put(1, F12, F22, F12);
    } else {
        auto over = [](i64 t) {
            if constexpr (SHIFT > 0)
                return (t + (1ll << (SHIFT - 1))) >> SHIFT;
            else
                return t;
        };
        i64 t0[3], t1[3], t2[3], t3[3];
        [[maybe_unused]] i64 mu[3], mv[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const fx::Split f11(F11[i]), f12(F12[i]), f22(F22[i]);
            t0[i] = over(fx::mulHigh(f11, map.k0[i], f12, map.k2[i]));
            t1[i] = over(fx::mulHigh(f11, map.k1[i], f12, map.k3[i]));
            t2[i] = over(fx::mulHigh(f12, map.k0[i], f22, map.k2[i]));
            t3[i] = over(fx::mulHigh(f12, map.k1[i], f22, map.k3[i]));
            if constexpr (GEO == SPHERE) {
                mu[i] = over(fx::mulHigh(f12, map.m[i]));
                mv[i] = over(-fx::mulHigh(f11, map.m[i]));
            }
        }
        if constexpr (GEO == SPHERE) {
            put(0, t0, t1, mu);
            put(1, t2, t3, mv);
        } else {
            put(0, t0, t1, t0);
            put(1, t2, t3, t2);
        }
    }
}

// Node column R's shares of component c.
template <int E>
__device__ __forceinline__ void fixedColumnShares(int c, int R, int le, const Exchange<fx::i64, E>& ex,
    fx::i64 (&o)[3])
{
    fx::i64 x[3], y[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        x[r] = ex.out.x[c][r][R][le];
        y[r] = ex.out.y[c][r][R][le];
    }
    fx::columnT(x, y, o);
}

// the velocities' scale: bits below the largest one
template <Geometry GEO> __device__ __forceinline__ int strainBits(const fx::Scaled& sc)
{
    return GEO == RECT ? min(58, 61 - sc.shift) : 55;
}
// the largest of the three rows' or columns' exponents, at least 2^-900 (below
// which values count as 0)
template <int E> __device__ __forceinline__ int topOfRows(const int (*top)[E], int le)
{
    return max(max(top[0][le], 123), max(top[1][le], top[2][le]));
}
constexpr int kTopMost = 1923; // above: beyond 2^900, or not finite

// Three threads per element as stressBlock: node column R, Gauss row R, node
// column R.
template <Geometry GEO, int E>
__device__ __forceinline__ void stressFixed(int nx, size_t N, const uint8_t* __restrict__ ice,
    const FixedGeometry& geo, const double* __restrict__ u, const double* __restrict__ v,
    const double* __restrict__ Pw, double* __restrict__ tdiv, double dmin2, double keep, bool release, size_t x0,
    FixedShared<GEO, E>& sh)
{
    using fx::i64;
    const int le = threadIdx.x % E, R = threadIdx.x / E;
    const size_t e = x0 + le;
    const bool active = e < N && ice[e];
    double pq[3] = { 0.0, 0.0, 0.0 }, told[6], rho = 1.0;
    [[maybe_unused]] int ke = 0;
    if (active) {
#pragma unroll
        for (int i = 0; i < 3; ++i)
            pq[i] = Pw[(3 * R + i) * N + e];
        if constexpr (GEO == RECT) {
            rho = geo.rect[e];
            dmin2 *= geo.rect[N + e];
        } else
            ke = geo.exponent[e];
    }
    sh.top[1][R][le] = topOf(max(fx::magnitudeWord(pq[0]), max(fx::magnitudeWord(pq[1]), fx::magnitudeWord(pq[2]))));
    waitForPrevious(release);
    double n[2][3] = { { 0.0, 0.0, 0.0 }, { 0.0, 0.0, 0.0 } };
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
#pragma unroll
        for (int r = 0; r < 3; ++r) { // needed at the end
            told[r] = afterWait(tdiv + (3 * r + R) * N + e);
            told[3 + r] = afterWait(tdiv + (9 + 3 * r + R) * N + e);
        }
    }
    int word = 0;
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int r = 0; r < 3; ++r)
            word = max(word, fx::magnitudeWord(n[c][r]));
    sh.top[0][R][le] = topOf(word);
    __syncthreads();
    const int top = topOfRows<E>(sh.top[0], le);
    // the increments' products may round up to 2^topP
    const int topP = topOfRows<E>(sh.top[1], le) + 1;
    bool bad = max(top, topP - 1) > kTopMost;
    const fx::Scaled sc(rho);
    const int bits = strainBits<GEO>(sc);
    fixedColumn<E>(n, fx::fixedShift(bits, top), R, le, sh.ex);
    __syncthreads();
    // Gauss row R
    const int scale = bits - top + 1022; // of the strain
    const int atStrain = fx::doubleExponent(GEO == RECT ? scale : scale - ke - 2);
    const int bitsP = GEO == RECT ? 58 - sc.shift : 58;
    const int atP = fx::fixedShift(bitsP, topP);
    const FixedMap<GEO> map(geo, R, e, N, active);
    i64 a[3], b[3], s[3], F11[3], F12[3], F22[3];
    fixedStrain<GEO, E>(R, le, sc, map, sh.ex, sh.sums[0], a, b, s);
    int most = 0;
    [[maybe_unused]] i64 nf[3] = { 0, 0, 0 }; // n . f
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        double zp, d, f;
        pointStress64(fx::toDouble(a[i] + b[i], atStrain + 1), fx::toDouble(a[i] - b[i], atStrain),
            fx::toDouble(s[i], atStrain), pq[i], dmin2, zp, d, f);
        most = max(most, max(fx::magnitudeWord(zp), max(fx::magnitudeWord(d), fx::magnitudeWord(f))));
        const i64 w = 2 * (fx::toFixed(zp, atP) - fx::toFixed(pq[i], atP)), D = fx::toFixed(d, atP);
        F11[i] = w + D;
        F22[i] = w - D;
        F12[i] = fx::toFixed(f, atP);
        if constexpr (GEO != RECT) {
            nf[0] += fx::mulHigh(fx::Split(F11[i]), map.n[i]);
            nf[1] += fx::mulHigh(fx::Split(F22[i]), map.n[i]);
            nf[2] += fx::mulHigh(fx::Split(F12[i]), map.n[i]);
        }
    }
    if constexpr (GEO == RECT) {
        __syncthreads(); // every warp has taken its row: the buffer changes hands
    } else {
        // P^T: subtract nu (n . f)
        sumRows<i64, E>(sh.sums[1], R, le, nf);
        const int nr = R == 1 ? -2 : 1;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const int w = i == 1 ? -2 * nr : nr;
            F11[i] -= nuTimes(fx::four(nf[0]), w);
            F22[i] -= nuTimes(fx::four(nf[1]), w);
            F12[i] -= nuTimes(fx::four(nf[2]), w);
        }
    }
    fixedShares<GEO, 3, E>(R, le, sc, map, F11, F12, F22, sh.ex);
    sh.top[0][R][le] = bad || most >= 0x7ff00000;
    __syncthreads();
    if (!active)
        return;
    bad = (sh.top[0][0][le] | sh.top[0][1][le] | sh.top[0][2][le]) != 0;
    const int scaleP = bitsP - topP + 1022;
    const int atOut = fx::doubleExponent(GEO == RECT ? scaleP : scaleP - 3 - ke - 2);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        i64 o[3];
        fixedColumnShares<E>(c, R, le, sh.ex, o);
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const double div = bad ? __longlong_as_double(0x7ff8000000000000ll) : fx::toDouble(o[r], atOut);
            tdiv[(9 * c + 3 * r + R) * N + e] = fma(told[3 * c + r], keep, div);
        }
    }
}

} // namespace sf
} // namespace nsdg
