"""The FP64 element update in fixed point (nsdg_fixed_rows.hpp), run on the host
row by row as the kernel does: strains and divergence shares against extended
precision, on rectangles, quadrilaterals and spherical cells from square to a
side ratio of 1000, beside the same maps in FP64; and the largest inputs that
its scales allow."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

SOURCE = r"""
#include "nsdg_fixed_rows.hpp"
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
using namespace nsdg;
using namespace nsdg::sf;
using fx::i64;
using LD = long double;
struct Element {
    double k[4][9], n[9], m[9], w[9], rho;
    i64 K[4][9], N[9], M[9];
    int x[3];
    bool sphere, rect;
};
static const double gp[3] = { 0.5 - std::sqrt(0.15), 0.5, 0.5 + std::sqrt(0.15) }, gw[3] = { 5. / 18, 8. / 18, 5. / 18 };
static int nuAt(int q) { return (q % 3 == 1 ? -2 : 1) * (q / 3 == 1 ? -2 : 1); }
static Element element(const double (*c)[2], bool sphere, bool rect)
{
    Element e;
    e.sphere = sphere;
    e.rect = rect;
    const double radius = 6371000.0;
    double iw[9], sum = 0, most[3] = { 0, 0, 0 };
    for (int q = 0; q < 9; ++q) {
        const double p = gp[q % 3], t = gp[q / 3];
        double xi[2], et[2];
        for (int d = 0; d < 2; ++d) {
            xi[d] = (1 - t) * (c[1][d] - c[0][d]) + t * (c[3][d] - c[2][d]);
            et[d] = (1 - p) * (c[2][d] - c[0][d]) + p * (c[3][d] - c[1][d]);
        }
        const double lat = (1 - t) * ((1 - p) * c[0][1] + p * c[1][1]) + t * ((1 - p) * c[2][1] + p * c[3][1]);
        const double J = xi[0] * et[1] - xi[1] * et[0], cl = sphere ? std::cos(lat) : 1.0;
        const double hx = 0.5 / (J * (sphere ? radius * cl : 1.0)), hy = 0.5 / (J * (sphere ? radius : 1.0));
        e.k[0][q] = et[1] * hx;
        e.k[1][q] = -xi[1] * hx;
        e.k[2][q] = -et[0] * hy;
        e.k[3][q] = xi[0] * hy;
        e.m[q] = sphere ? 0.5 * std::tan(lat) / radius : 0.0;
        e.w[q] = 2 * gw[q % 3] * gw[q / 3] * J;
        iw[q] = nuAt(q) / (e.w[q] * cl);
        sum += nuAt(q) * iw[q];
    }
    e.rho = e.k[3][4] / e.k[0][4];
    for (int q = 0; q < 9 && rect; ++q) { // the same at every point
        e.k[0][q] = e.k[0][4];
        e.k[1][q] = e.k[2][q] = 0.0;
        e.k[3][q] = e.k[3][4];
    }
    for (int q = 0; q < 9; ++q) {
        e.n[q] = iw[q] / sum;
        for (int k = 0; k < 4; ++k)
            most[k % 2] = std::max(most[k % 2], std::fabs(e.k[k][q]));
        most[2] = std::max(most[2], std::fabs(e.m[q]));
    }
    for (int g = 0; g < 3; ++g)
        std::frexp(most[g], e.x + g);
    for (int q = 0; q < 9; ++q) {
        for (int k = 0; k < 4; ++k)
            e.K[k][q] = fx::packed(std::llrint(std::ldexp(e.k[k][q], 62 - e.x[k % 2])));
        e.N[q] = fx::packed(std::llrint(std::ldexp(e.n[q], 62)));
        e.M[q] = sphere ? fx::packed(std::llrint(std::ldexp(e.m[q], 62 - e.x[2]))) : 0;
    }
    return e;
}
// the maps in T
static double mad(double a, double b, double c) { return std::fma(a, b, c); }
static LD mad(LD a, LD b, LD c) { return a * b + c; }
template <typename T> struct Maps {
    T g = std::sqrt(T(3) / 20), c3 = T(3) / 10, c4 = T(4) / 10;
    void interp(const T* n, T* o) const
    {
        const T d = n[2] - n[0], m = mad(c3, n[0] + n[2] - 2 * n[1], n[1]);
        o[0] = mad(-g, d, m); o[1] = n[1]; o[2] = mad(g, d, m);
    }
    void deriv(const T* n, T* o) const
    {
        const T d = n[2] - n[0], e = n[0] + n[2] - 2 * n[1];
        o[0] = mad(-4 * g, e, d); o[1] = d; o[2] = mad(4 * g, e, d);
    }
    void interpT(const T* t, T* o) const
    {
        const T s = t[0] + t[2], d = t[2] - t[0], m = c3 * s;
        o[0] = mad(-g, d, m); o[1] = mad(c4, s, t[1]); o[2] = mad(g, d, m);
    }
    void derivT(const T* t, T* o) const
    {
        const T s = t[0] + t[1] + t[2], k = 4 * g * (t[2] - t[0]);
        o[0] = k - s; o[1] = -2 * k; o[2] = k + s;
    }
    void strain(const Element& e, const double (*u)[9], T (*f)[9]) const
    {
        T v[2][3][3], d[2][3][3];
        for (int c = 0; c < 2; ++c)
            for (int i = 0; i < 3; ++i) {
                const T n[3] = { T(u[c][i]), T(u[c][3 + i]), T(u[c][6 + i]) };
                T a[3], b[3];
                interp(n, a);
                deriv(n, b);
                for (int r = 0; r < 3; ++r) { v[c][r][i] = a[r]; d[c][r][i] = b[r]; }
            }
        for (int r = 0; r < 3; ++r) {
            T x[2][3], y[2][3], p[2][3];
            for (int c = 0; c < 2; ++c) { deriv(v[c][r], x[c]); interp(d[c][r], y[c]); interp(v[c][r], p[c]); }
            for (int i = 0; i < 3; ++i) {
                const int q = 3 * r + i;
                const T k0 = e.k[0][q], k1 = e.k[1][q], k2 = e.k[2][q], k3 = e.k[3][q], m = e.m[q];
                f[0][q] = mad(k0, x[0][i], k1 * y[0][i]);
                f[1][q] = mad(k2, x[1][i], k3 * y[1][i]);
                f[2][q] = mad(k2, x[0][i], mad(k3, y[0][i], mad(k0, x[1][i], k1 * y[1][i])));
                f[0][q] = mad(-m, p[1][i], f[0][q]);
                f[2][q] = mad(m, p[0][i], f[2][q]);
            }
        }
        for (int k = 0; k < 3 && !e.rect; ++k) {
            T c = 0;
            for (int q = 0; q < 9; ++q) c += nuAt(q) * f[k][q];
            for (int q = 0; q < 9; ++q) f[k][q] = mad(-c, T(e.n[q]), f[k][q]);
        }
    }
    void shares(const Element& e, const T (*F)[9], T (*o)[9]) const // F11, F12, F22
    {
        T f[3][9];
        for (int k = 0; k < 3; ++k) {
            T c = 0;
            for (int q = 0; q < 9 && !e.rect; ++q) c = mad(T(e.n[q]), F[k][q], c);
            for (int q = 0; q < 9; ++q) f[k][q] = mad(T(-nuAt(q)), c, F[k][q]);
        }
        for (int c = 0; c < 2; ++c) {
            T x[3][3], y[3][3];
            for (int r = 0; r < 3; ++r) {
                T t0[3], t1[3], tm[3], z[3];
                for (int i = 0; i < 3; ++i) {
                    const int q = 3 * r + i;
                    t0[i] = mad(T(e.k[0][q]), f[c][q], T(e.k[2][q]) * f[c + 1][q]);
                    t1[i] = mad(T(e.k[1][q]), f[c][q], T(e.k[3][q]) * f[c + 1][q]);
                    tm[i] = T(e.m[q]) * (c == 0 ? f[1][q] : -f[0][q]);
                }
                derivT(t0, x[r]);
                interpT(t1, y[r]);
                interpT(tm, z);
                for (int i = 0; i < 3; ++i) x[r][i] += z[i];
            }
            for (int i = 0; i < 3; ++i) {
                const T a[3] = { x[0][i], x[1][i], x[2][i] }, b[3] = { y[0][i], y[1][i], y[2][i] };
                T p[3], q[3];
                interpT(a, p);
                derivT(b, q);
                for (int r = 0; r < 3; ++r) o[c][3 * r + i] = p[r] + q[r];
            }
        }
    }
};
// the fixed-point rows, as the kernel puts them together
template <Geometry GEO> static FixedMap<GEO> rowMap(const Element& e, int R)
{
    if constexpr (GEO == RECT)
        return FixedMap<RECT>(e.rho);
    else
        return FixedMap<GEO>([&](int c, int q) { return fx::unpacked(c < 4 ? e.K[c][q] : c == 4 ? e.N[q] : e.M[q]); },
            [&](int g) { return e.x[g]; }, R);
}
template <Geometry GEO> static void fixedStrains(const Element& e, const double (*u)[9], LD (*f)[9])
{
    int word = 0;
    for (int c = 0; c < 2; ++c)
        for (int j = 0; j < 9; ++j) word = std::max(word, fx::magnitudeWord(u[c][j]));
    const int top = word >> 20, bits = kVelocityBits, at = fx::fixedShift(bits, top);
    i64 v[2][3][3], d[2][3][3], g[3][3][3], part[3][3];
    int scale[3];
    for (int c = 0; c < 2; ++c)
        for (int i = 0; i < 3; ++i) {
            const i64 n[3] = { fx::toFixed(u[c][i], at), fx::toFixed(u[c][3 + i], at), fx::toFixed(u[c][6 + i], at) };
            i64 a[3], b[3];
            fx::interp(n, a);
            fx::deriv(n, b);
            for (int r = 0; r < 3; ++r) { v[c][r][i] = a[r]; d[c][r][i] = b[r]; }
        }
    for (int R = 0; R < 3; ++R) {
        scale[R] = strainRow<GEO>([&](int c, i64 (&I)[3], i64 (&D)[3]) {
            std::copy_n(v[c][R], 3, I);
            std::copy_n(d[c][R], 3, D);
        }, rowMap<GEO>(e, R), g[0][R], g[1][R], g[2][R]);
        for (int k = 0; k < 3; ++k) part[k][R] = nuPart(R, g[k][R]);
    }
    const int all = std::max({ scale[0], scale[1], scale[2] });
    if constexpr (GEO != RECT)
        for (int k = 0; k < 3; ++k) {
            i64 c = 0;
            for (int R = 0; R < 3; ++R) {
                c += part[k][R] >> std::min(63, all - scale[R]);
                for (int i = 0; i < 3; ++i) g[k][R][i] >>= std::min(63, all - scale[R]);
            }
            for (int R = 0; R < 3; ++R) subtractN(rowMap<GEO>(e, R), c, g[k][R]);
        }
    for (int k = 0; k < 3; ++k)
        for (int q = 0; q < 9; ++q)
            f[k][q] = ldexpl(g[k][q / 3][q % 3], all - (bits - top + 1022)) * (GEO == RECT ? LD(e.k[0][4]) : 1);
}
// F in units of 2^-bits
template <Geometry GEO> static void fixedShares(const Element& e, const i64 (*F)[9], LD (*o)[9])
{
    i64 f[3][3][3];
    for (int k = 0; k < 3; ++k) {
        i64 sum = 0;
        for (int R = 0; R < 3; ++R) {
            std::copy_n(F[k] + 3 * R, 3, f[k][R]);
            if constexpr (GEO != RECT) sum += projectedPart(rowMap<GEO>(e, R), f[k][R]);
        }
        for (int R = 0; R < 3; ++R) subtractNu(R, sum, f[k][R]);
    }
    for (int c = 0; c < 2; ++c) {
        i64 x[3][3], y[3][3];
        int scale[3];
        for (int R = 0; R < 3; ++R) {
            i64 fm[3];
            for (int i = 0; i < 3; ++i) fm[i] = c == 0 ? f[1][R][i] : -f[0][R][i];
            scale[R] = sharesRow<GEO>(rowMap<GEO>(e, R), f[c][R], f[c + 1][R], fm, x[R], y[R]);
        }
        const int all = std::max({ scale[0], scale[1], scale[2] });
        for (int i = 0; i < 3; ++i) {
            i64 a[3], b[3], r[3];
            for (int R = 0; R < 3; ++R) {
                a[R] = x[R][i] >> std::min(63, all - scale[R]);
                b[R] = y[R][i] >> std::min(63, all - scale[R]);
            }
            fx::columnT(a, b, r);
            for (int j = 0; j < 3; ++j) o[c][3 * j + i] = ldexpl(r[j], all) * (GEO == RECT ? LD(e.k[0][4]) : 1);
        }
    }
}
static std::mt19937_64 gen(7);
static double U() { return std::uniform_real_distribution<double>(-1, 1)(gen); }
template <Geometry GEO> static int run(double ratio, bool turned)
{
    const Maps<double> fp;
    const Maps<LD> ld;
    LD strain[2] = { 0, 0 }, share[2] = { 0, 0 }, worst[2] = { 0, 0 };
    for (int t = 0; t < 4000; ++t) {
        const double hx = ratio < 1 ? 4000 * ratio : 4000, hy = ratio < 1 ? 4000 : 4000 / ratio;
        double c[4][2] = { { 0, 0 }, { hx, 0 }, { 0, hy }, { hx, hy } };
        for (auto& p : c) {
            if (GEO == QUAD) { p[0] += 0.08 * hx * U(); p[1] += 0.08 * hy * U(); }
            if (turned) { const double a = p[0], b = p[1]; p[0] = 0.6 * a - 0.8 * b; p[1] = 0.8 * a + 0.6 * b; }
            if (GEO == SPHERE) { p[0] /= 6371000. * std::cos(1.1); p[1] = 1.1 + p[1] / 6371000.; }
        }
        const Element e = element(c, GEO == SPHERE, GEO == RECT);
        // flows: smooth, along xi alone, along eta alone, rough; the last 1000 the largest values
        double u[2][9];
        for (int k = 0; k < 2; ++k) {
            const double a = U(), b = U(), d = U();
            for (int j = 0; j < 9; ++j) {
                const double xi = 0.5 * (j % 3), et = 0.5 * (j / 3);
                const double s = t % 4 == 1 ? a * xi + d * xi * xi : t % 4 == 2 ? b * et + d * et * et : a * xi + b * et + d * xi * et;
                u[k][j] = t >= 3000 ? (gen() & 1 ? 1 : -1) * (1 - 0x1p-53) : t % 4 == 3 ? U() : 0.3 + 1e-2 * s;
            }
        }
        double a[3][9];
        LD b[3][9], x[3][9], most = 0;
        fp.strain(e, u, a);
        ld.strain(e, u, x);
        fixedStrains<GEO>(e, u, b);
        for (int k = 0; k < 3; ++k)
            for (int q = 0; q < 9; ++q) most = std::max(most, fabsl(x[k][q]));
        // the largest stress increments (4.3, 1 and 4.3 times the pressure), or any
        const int bits = kPressureBits<GEO> - 1;
        i64 F[3][9];
        double Fd[3][9];
        LD Fx[3][9], o[2][9], z[2][9];
        double od[2][9];
        for (int k = 0; k < 3; ++k)
            for (int q = 0; q < 9; ++q) {
                const double s = t >= 3000 ? (gen() & 1 ? 1 : -1) * (k == 1 ? 1 : 4.3) : (k == 1 ? U() : -2 + 2 * U());
                Fd[k][q] = s * (1ll << 40);
                F[k][q] = static_cast<i64>(std::ldexp(Fd[k][q], bits - 40));
                Fx[k][q] = Fd[k][q];
            }
        fp.shares(e, Fd, od);
        ld.shares(e, Fx, z);
        fixedShares<GEO>(e, F, o);
        for (int k = 0; k < 3; ++k)
            for (int q = 0; q < 9; ++q) {
                const LD h = (b[k][q] - x[k][q]) / most, d = (a[k][q] - x[k][q]) / most;
                if (t >= 3000) worst[0] = std::max(worst[0], fabsl(h));
                else { strain[0] += h * h; strain[1] += d * d; }
            }
        for (int k = 0; k < 2; ++k) { // over the largest factor and the pressure
            LD f = 0;
            for (int q = 0; q < 9; ++q)
                f = std::max({ f, fabsl(e.k[0][q]), fabsl(e.k[1][q]), fabsl(e.k[2][q]), fabsl(e.k[3][q]) });
            f *= 2 * ldexpl(1, 40);
            for (int j = 0; j < 9; ++j) {
                const LD h = (ldexpl(o[k][j], 40 - bits) - z[k][j]) / f, d = (od[k][j] - z[k][j]) / f;
                if (t >= 3000) worst[1] = std::max(worst[1], fabsl(h));
                else { share[0] += h * h; share[1] += d * d; }
            }
        }
    }
    std::printf("%.4Lf %.4Lf %.3Le %.3Le\n", sqrtl(strain[0] / strain[1]), sqrtl(share[0] / share[1]), worst[0], worst[1]);
    return 0;
}
int main(int, char** argv)
{
    const double ratio = std::atof(argv[2]);
    const char* kind = argv[1];
    return !std::strcmp(kind, "rect") ? run<RECT>(ratio, false)
        : !std::strcmp(kind, "sphere") ? run<SPHERE>(ratio, false)
                                       : run<QUAD>(ratio, !std::strcmp(kind, "turned"));
}
"""

CASES = [("rect", r) for r in (1 / 1.9999, 0.7, 0.9999, 1.0, 1.9999)] \
    + [(k, r) for k in ("quad", "turned", "sphere") for r in (1e-3, 0.01, 1 / 32, 0.25, 1.0, 4.0, 32.0, 100.0, 1e3)]


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("fixed_rows")
    (d / "a.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(ROOT / "nextsimdg_gb300" / "csrc"),
                    str(d / "a.cpp"), "-o", str(d / "a")], check=True)
    return d / "a"


@pytest.mark.parametrize("kind,ratio", CASES)
def test_no_further_off_than_fp64_maps(program, kind, ratio):
    """RMS errors, of the strain over the element's largest and of the divergence
    over the pressure's scale, are at most those of the same maps in FP64; with
    the largest inputs of the scales' bounds an error stays a rounding (an overflow
    would be of order 1): 200 roundings of 2^-53."""
    strain, share, worst, worstShare = map(float, subprocess.check_output([str(program), kind, repr(ratio)]).split())
    assert strain <= 1.0
    assert share <= 1.0
    assert worst <= 200 * 2.0 ** -53
    assert worstShare <= 200 * 2.0 ** -53
