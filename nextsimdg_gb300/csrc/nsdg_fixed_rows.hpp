// nsdg_fixed_rows.hpp — one row's and one column's part of the FP64 element
// update in fixed point (nsdg_stress_fixed.cuh; host and device).
//
// Scales.  The velocities are below 2^top and become integers below V =
// 2^bits; the 1-D maps stay within
//   columns    |v| <= 1.2 V, |dv| <= 6.2 V (second differences 25 V)
//   rows       derivatives along xi and eta <= 7.3 V (second differences 25 V)
// -> 58 bits.  Rectangles (rho < 2): |strain| <= 22 V; F11, F12, F22 within 4.3 F come
// out of the transposed maps within 11 (1 + rho) 4.3 F = 142 F -> F = 2^55.
//
// Elsewhere an element's factors come in groups with an exponent each: those of
// the xi derivatives, those of the eta derivatives and, on a sphere, the metric
// term's.  A row shifts each group's derivatives so that the larger products
// have 58 bits: the unit is 2^-58 of the row's largest strain, however slender the
// element is and however little the velocity varies in it.  The rows then
// share the largest row's scale: |a|, |b|, |s| <= 5 2^56, the projection's
// functional <= 16 5 2^56 < 2^62.4, the projected strain, and a + b of it, < 2^62.8.
// In the divergence the stresses after their projection are within 22 F (F =
// 2^57: below 2^61.5), and each component's products get 58 bits in the same way:
// through the transposed maps they stay within 25.4 2^58 < 2^62.7.
#pragma once

#include "nsdg_fixed.hpp"

namespace nsdg {
namespace sf {

// How an element's map is given: one pair (k_y / k_x, 1 / k_x^2) on
// rectangles (FP64), four derivatives on parallelograms (FP32), four per Gauss
// point else.  On rectangles the strain is carried over k_x (strain' = strain /
// k_x, the eta derivatives times rho = k_y / k_x, DeltaMin^2 over k_x^2) and k_x
// is part of the pressure's weight, so only rho is multiplied in.
enum Geometry { RECT = 0, AFFINE = 1, QUAD = 2, SPHERE = 3 };

constexpr int kRowBits = 58; // of the products that set a row's scale

// The factors of Gauss row R (rectangles: rho).
template <Geometry GEO> struct FixedMap {
    fx::Split k0[3], k1[3], k2[3], k3[3], n[3], m[3];
    int xi, eta, metric; // the groups' exponents
    // at(c, q): factor c (0 .. 3; 4: n, 5: m) at point q, exponent(g): group g's
    template <typename F, typename X>
    NSDG_FX_HD FixedMap(F at, X exponent, int R)
        : k0 { at(0, 3 * R), at(0, 3 * R + 1), at(0, 3 * R + 2) }
        , k1 { at(1, 3 * R), at(1, 3 * R + 1), at(1, 3 * R + 2) }
        , k2 { at(2, 3 * R), at(2, 3 * R + 1), at(2, 3 * R + 2) }
        , k3 { at(3, 3 * R), at(3, 3 * R + 1), at(3, 3 * R + 2) }
        , n { at(4, 3 * R), at(4, 3 * R + 1), at(4, 3 * R + 2) }
        , m { GEO == SPHERE ? at(5, 3 * R) : fx::Split(0), GEO == SPHERE ? at(5, 3 * R + 1) : fx::Split(0),
            GEO == SPHERE ? at(5, 3 * R + 2) : fx::Split(0) }
        , xi(exponent(0))
        , eta(exponent(1))
        , metric(GEO == SPHERE ? exponent(2) : 0)
    {
    }
};
constexpr int kRectShift = 3; // k_y / k_x is below kRectWide = 2
template <> struct FixedMap<RECT> {
    fx::Scaled<kRectShift> rho;
    NSDG_FX_HD explicit FixedMap(double r) : rho(r) { }
};

// nu (1, -2 or 4) times t
NSDG_FX_HD fx::i64 nuTimes(fx::i64 t, int f) { return f == 1 ? t : f == -2 ? -2 * t : fx::shiftLeft(t, 2); }
NSDG_FX_HD int nuRow(int R) { return R == 1 ? -2 : 1; } // nu on row R: nr, -2 nr, nr

constexpr int kVelocityBits = 58;
// of the pressure (stresses within 4.3 times it), and of a stress that needs no
// projection
template <Geometry GEO> constexpr int kPressureBits = GEO == RECT ? 59 - kRectShift : 58;
template <Geometry GEO> constexpr int kStressBits = GEO == RECT ? 59 - kRectShift : 59;

// The half strains of Gauss row R before their projection, times 2^-(returned
// value) of the velocities' unit; I[c], D[c] by load(c, I, D): velocity
// component c and its eta derivative on the row's columns.
template <Geometry GEO, typename L>
NSDG_FX_HD int strainRow(L load, const FixedMap<GEO>& map, fx::i64 (&a)[3], fx::i64 (&b)[3], fx::i64 (&s)[3])
{
    using fx::i64;
    using fx::Split;
    i64 I[3], D[3], uxi[3], uet[3], vxi[3], vet[3];
    [[maybe_unused]] i64 up[3], vp[3];
    load(0, I, D);
    fx::deriv(I, uxi);
    if constexpr (GEO == RECT)
        map.rho.interp(D, uet);
    else
        fx::interp(D, uet);
    if constexpr (GEO == SPHERE)
        fx::interp(I, up);
    load(1, I, D);
    fx::deriv(I, vxi);
    if constexpr (GEO == RECT)
        map.rho.interp(D, vet);
    else
        fx::interp(D, vet);
    if constexpr (GEO == SPHERE)
        fx::interp(I, vp);
    if constexpr (GEO == RECT) {
        for (int i = 0; i < 3; ++i) {
            a[i] = uxi[i];
            b[i] = vet[i];
            s[i] = uet[i] + vxi[i];
        }
        return 0;
    } else {
        int x = 0, e = 0;
        for (int i = 0; i < 3; ++i) {
            x |= fx::upperMagnitude(uxi[i]) | fx::upperMagnitude(vxi[i]);
            e |= fx::upperMagnitude(uet[i]) | fx::upperMagnitude(vet[i]);
        }
        int top = map.xi + fx::lengthOf(x);
        const int topE = map.eta + fx::lengthOf(e);
        top = top > topE ? top : topE;
        if constexpr (GEO == SPHERE) { // values, not differences: up to 1.4 V
            const int topM = map.metric + kVelocityBits + 1;
            top = top > topM ? top : topM;
        }
        const fx::Shift sx(kRowBits - top + map.xi), se(kRowBits - top + map.eta);
        for (int i = 0; i < 3; ++i) {
            const Split ux(sx(uxi[i])), ue(se(uet[i])), vx(sx(vxi[i])), ve(se(vet[i]));
            a[i] = fx::mulHigh(ux, map.k0[i], ue, map.k1[i]);
            b[i] = fx::mulHigh(vx, map.k2[i], ve, map.k3[i]);
            s[i] = fx::mulHigh(ux, map.k2[i], ue, map.k3[i]) + fx::mulHigh(vx, map.k0[i], ve, map.k1[i]);
        }
        if constexpr (GEO == SPHERE) {
            const int d = top - kRowBits - map.metric; // at least 1
            const int sm = d > 63 ? 63 : d;
            for (int i = 0; i < 3; ++i) {
                a[i] -= fx::mulHigh(Split(vp[i] >> sm), map.m[i]);
                s[i] += fx::mulHigh(Split(up[i] >> sm), map.m[i]);
            }
        }
        return top - kRowBits + 2;
    }
}

// Row R's stresses F through the transposed xi maps, component c: x to the
// transposed interpolation along eta, y to the transposed derivative, times
// 2^-(returned value) of the stresses' unit.  F0, F1: (F11, F12) for c = 0, (F12,
// F22) for c = 1; on a sphere FM: F12 for c = 0, -F11 for c = 1.
template <Geometry GEO>
NSDG_FX_HD int sharesRow(const FixedMap<GEO>& map, const fx::i64 (&F0)[3], const fx::i64 (&F1)[3],
    [[maybe_unused]] const fx::i64 (&FM)[3], fx::i64 (&x)[3], fx::i64 (&y)[3])
{
    using fx::i64;
    using fx::Split;
    if constexpr (GEO == RECT) {
        fx::derivT(F0, x);
        map.rho.interpT(F1, y);
        return 0;
    } else {
        i64 t0[3], t1[3];
        [[maybe_unused]] i64 tm[3];
        int o0 = 0, o1 = 0;
        for (int i = 0; i < 3; ++i) {
            const Split f(F0[i]), h(F1[i]);
            t0[i] = fx::mulHigh(f, map.k0[i], h, map.k2[i]);
            t1[i] = fx::mulHigh(f, map.k1[i], h, map.k3[i]);
            o0 |= fx::upperMagnitude(t0[i]);
            o1 |= fx::upperMagnitude(t1[i]);
        }
        int top = map.xi + fx::lengthOf(o0);
        const int topE = map.eta + fx::lengthOf(o1);
        top = top > topE ? top : topE;
        if constexpr (GEO == SPHERE) { // below 2^59.5
            for (int i = 0; i < 3; ++i)
                tm[i] = fx::mulHigh(Split(FM[i]), map.m[i]);
            const int topM = map.metric + 60;
            top = top > topM ? top : topM;
        }
        const fx::Shift sx(kRowBits - top + map.xi), se(kRowBits - top + map.eta);
        for (int i = 0; i < 3; ++i) {
            t0[i] = sx(t0[i]);
            t1[i] = se(t1[i]);
        }
        fx::derivT(t0, x);
        fx::interpT(t1, y);
        if constexpr (GEO == SPHERE) {
            const int d = top - kRowBits - map.metric; // at least 2
            const int sm = d > 63 ? 63 : d;
            i64 z[3];
            for (int i = 0; i < 3; ++i)
                tm[i] >>= sm;
            fx::interpT(tm, z);
            for (int i = 0; i < 3; ++i)
                x[i] += z[i];
        }
        return top - kRowBits + 2;
    }
}

// P^T of a row's stresses: its part of n . f, and f minus nu times the sum of
// the rows' parts
template <Geometry GEO> NSDG_FX_HD fx::i64 projectedPart(const FixedMap<GEO>& map, const fx::i64 (&f)[3])
{
    const fx::Split s[3] = { fx::Split(f[0]), fx::Split(f[1]), fx::Split(f[2]) };
    return fx::dotUnit(s, map.n);
}
NSDG_FX_HD void subtractNu(int R, fx::i64 sum, fx::i64 (&f)[3])
{
    const int nr = nuRow(R);
    for (int i = 0; i < 3; ++i)
        f[i] -= nuTimes(sum, i == 1 ? -2 * nr : nr);
}
// P of a row's strains g: its part of nu . g, and g minus n times the sum
NSDG_FX_HD fx::i64 nuPart(int R, const fx::i64 (&g)[3]) { return nuTimes(g[0] + g[2] - 2 * g[1], nuRow(R)); }
template <Geometry GEO> NSDG_FX_HD void subtractN(const FixedMap<GEO>& map, fx::i64 sum, fx::i64 (&g)[3])
{
    const fx::Split c(sum);
    for (int i = 0; i < 3; ++i)
        g[i] -= fx::mulUnit(c, map.n[i]);
}

} // namespace sf
} // namespace nsdg
