// nsdg_stress_fixed.cuh — the FP64 mEVP element update (nsdg_sumfact.cuh) with
// its linear maps in 64-bit fixed point (nsdg_fixed.hpp).
//
// Errors against extended precision over those of the same maps in FP64, for
// velocities that vary by 3 % of their size, along one side alone or freely
// within an element, and stresses over the pressure's scale: strain 0.4 to 0.7 and
// divergence 0.34 to 0.9, on rectangles, quadrilaterals and spherical cells of side
// ratios from 1/1000 to 1000.
//
// What stays in FP64 is the rheology, ten instructions per Gauss point, and
// the relaxation of the 18 divergence coefficients: 108 FP64 instructions per
// element where the maps in FP64 make it 480 on rectangles and 720 on
// quadrilaterals.
//
// The velocities get one scale per element, 58 bits below the largest; the
// weighted pressure, F = its largest, bounds the stress increments (|2 zp -+ d|
// <= sqrt(5) pq, so |f11|, |f22| <= 4.3 F, |f12| <= F).  What follows is scaled
// row by row (nsdg_fixed_rows.hpp); with one scale per element throughout, from
// bounds on the maps alone, an update was 5 to 7 % shorter on quadrilaterals and
// spheres, and the strain along a cell's long side had the error of the FP64 maps
// times the side ratio.
#pragma once

#include "nsdg_fixed_rows.hpp"
#include "nsdg_kernels.hpp"
#include "nsdg_seed64.cuh"
#include "nsdg_sumfact.cuh"

namespace nsdg {
namespace sf {

template <Geometry GEO, int E> struct FixedShared {
    Exchange<fx::i64, E> ex;
    fx::i64 sums[GEO == RECT ? 1 : 2][3][3][E];
    int top[2][3][E];
    int scale[GEO == RECT ? 1 : 3][3][E]; // the rows': of the strain, and of the shares of u and v
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

// The maps of Gauss row R of element e.
template <Geometry GEO>
__device__ __forceinline__ FixedMap<GEO> rowMap(const FixedGeometry& geo, int R, size_t e, size_t N, bool active)
{
    if constexpr (GEO == RECT) {
        return FixedMap<RECT>(active ? geo.rect[e] : 1.0);
    } else {
        return FixedMap<GEO>(
            [&](int c, int q) {
                const fx::i64* p = c < 4 ? geo.k + size_t(9 * c) * N : c == 4 ? geo.n : geo.m;
                return fx::unpacked(active ? p[size_t(q) * N + e] : 0);
            },
            [&](int g) { return active ? geo.exponent[size_t(g) * N + e] : 0; }, R);
    }
}

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

// The half strains of Gauss row R times 2^-(returned value) of the velocities'
// unit (on quadrilaterals projected; sums takes the three rows' parts of nu . g,
// scale their scales).
template <Geometry GEO, int E>
__device__ __forceinline__ int fixedStrain(int R, int le, const FixedMap<GEO>& map, const Exchange<fx::i64, E>& ex,
    [[maybe_unused]] fx::i64 (*sums)[3][E], [[maybe_unused]] int (*scale)[E], fx::i64 (&a)[3], fx::i64 (&b)[3],
    fx::i64 (&s)[3])
{
    using fx::i64;
    int mine = strainRow<GEO>(
        [&](int c, i64 (&I)[3], i64 (&D)[3]) {
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                I[i] = ex.in.v[c][R][i][le];
                D[i] = ex.in.dv[c][R][i][le];
            }
        },
        map, a, b, s);
    if constexpr (GEO != RECT) {
        sums[R][0][le] = nuPart(R, a);
        sums[R][1][le] = nuPart(R, b);
        sums[R][2][le] = nuPart(R, s);
        scale[R][le] = mine;
        __syncthreads();
        const int all = max(scale[0][le], max(scale[1][le], scale[2][le]));
        i64 c[3] = { 0, 0, 0 };
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const int d = min(all - scale[r][le], 63);
#pragma unroll
            for (int k = 0; k < 3; ++k)
                c[k] += sums[r][k][le] >> d;
        }
        const int d = min(all - mine, 63);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            a[i] >>= d;
            b[i] >>= d;
            s[i] >>= d;
        }
        subtractN(map, c[0], a);
        subtractN(map, c[1], b);
        subtractN(map, c[2], s);
        mine = all;
    }
    return mine;
}

// Row R's stresses F through the transposed xi maps.
template <Geometry GEO, int E>
__device__ __forceinline__ void fixedShares(int R, int le, const FixedMap<GEO>& map, const fx::i64 (&F11)[3],
    const fx::i64 (&F12)[3], const fx::i64 (&F22)[3], Exchange<fx::i64, E>& ex, int (*scale)[3][E])
{
    using fx::i64;
    auto put = [&](int c, const i64 (&F0)[3], const i64 (&F1)[3], const i64 (&FM)[3]) {
        i64 x[3], y[3];
        const int mine = sharesRow<GEO>(map, F0, F1, FM, x, y);
        if constexpr (GEO != RECT)
            scale[c][R][le] = mine;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            ex.out.x[c][R][i][le] = x[i];
            ex.out.y[c][R][i][le] = y[i];
        }
    };
    put(0, F11, F12, F12);
    if constexpr (GEO == SPHERE) {
        const i64 minus[3] = { -F11[0], -F11[1], -F11[2] };
        put(1, F12, F22, minus);
    } else {
        put(1, F12, F22, F12);
    }
}

// Node column R's shares of component c, times 2^-(returned value) of the
// stresses' unit.
template <Geometry GEO, int E>
__device__ __forceinline__ int fixedColumnShares(int c, int R, int le, const Exchange<fx::i64, E>& ex,
    [[maybe_unused]] const int (*scale)[3][E], fx::i64 (&o)[3])
{
    fx::i64 x[3], y[3];
    int all = 0;
    if constexpr (GEO != RECT)
        all = max(scale[c][0][le], max(scale[c][1][le], scale[c][2][le]));
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        x[r] = ex.out.x[c][r][R][le];
        y[r] = ex.out.y[c][r][R][le];
        if constexpr (GEO != RECT) {
            const int d = min(all - scale[c][r][le], 63);
            x[r] >>= d;
            y[r] >>= d;
        }
    }
    fx::columnT(x, y, o);
    return all;
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
    double pq[3] = { 0.0, 0.0, 0.0 }, told[6];
    if (active) {
#pragma unroll
        for (int i = 0; i < 3; ++i)
            pq[i] = Pw[(3 * R + i) * N + e];
        if constexpr (GEO == RECT)
            dmin2 *= geo.rect[N + e];
    }
    sh.top[1][R][le] = topOf(max(fx::magnitudeWord(pq[0]), max(fx::magnitudeWord(pq[1]), fx::magnitudeWord(pq[2]))));
    const FixedMap<GEO> map = rowMap<GEO>(geo, R, e, N, active);
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
    fixedColumn<E>(n, fx::fixedShift(kVelocityBits, top), R, le, sh.ex);
    __syncthreads();
    // Gauss row R
    const int atP = fx::fixedShift(kPressureBits<GEO>, topP);
    i64 a[3], b[3], s[3], F11[3], F12[3], F22[3];
    const int strainScale = fixedStrain<GEO, E>(R, le, map, sh.ex, sh.sums[0], sh.scale[0], a, b, s);
    const int atStrain = fx::doubleExponent(kVelocityBits - top + 1022 - strainScale);
    int most = 0;
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
    }
    if constexpr (GEO == RECT) {
        __syncthreads(); // every warp has taken its row: the buffer changes hands
    } else {
        // P^T: subtract nu (n . f)
        i64 nf[3] = { projectedPart(map, F11), projectedPart(map, F22), projectedPart(map, F12) };
        sumRows<i64, E>(sh.sums[1], R, le, nf);
        subtractNu(R, nf[0], F11);
        subtractNu(R, nf[1], F22);
        subtractNu(R, nf[2], F12);
    }
    // needed at the end (loaded with the velocities, 256 x 256 update 3.65 against 3.60 ms)
    if (active) {
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            told[r] = afterWait(tdiv + (3 * r + R) * N + e);
            told[3 + r] = afterWait(tdiv + (9 + 3 * r + R) * N + e);
        }
    }
    fixedShares<GEO, E>(R, le, map, F11, F12, F22, sh.ex, sh.scale + (GEO == RECT ? 0 : 1));
    sh.top[0][R][le] = bad || most >= 0x7ff00000;
    __syncthreads();
    if (!active)
        return;
    bad = (sh.top[0][0][le] | sh.top[0][1][le] | sh.top[0][2][le]) != 0;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        i64 o[3];
        const int scale = fixedColumnShares<GEO, E>(c, R, le, sh.ex, sh.scale + (GEO == RECT ? 0 : 1), o);
        const int atOut = fx::doubleExponent(kPressureBits<GEO> - topP + 1022 - scale);
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const double div = bad ? __longlong_as_double(0x7ff8000000000000ll) : fx::toDouble(o[r], atOut);
            tdiv[(9 * c + 3 * r + R) * N + e] = fma(told[3 * c + r], keep, div);
        }
    }
}

} // namespace sf
} // namespace nsdg
