"""The element update's linear maps in 64-bit fixed point, on the host against
extended precision: conversions, products, and the chains from node velocities
to strains and from stress increments to divergence shares with the largest
inputs their scales allow (an overflow would be off by 2^63 units)."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

SOURCE = r"""
#include "nsdg_fixed.hpp"
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
using namespace nsdg::fx;
using R = long double;
static const R g = sqrtl(R(3) / 20);
static void interpR(const R* n, R* o)
{
    const R d = n[2] - n[0], e = n[0] + n[2] - 2 * n[1];
    o[0] = n[1] + R(3) / 10 * e - g * d; o[1] = n[1]; o[2] = n[1] + R(3) / 10 * e + g * d;
}
static void derivR(const R* n, R* o)
{
    const R d = n[2] - n[0], e = n[0] + n[2] - 2 * n[1];
    o[0] = d - 4 * g * e; o[1] = d; o[2] = d + 4 * g * e;
}
static void transposed(void (*map)(const R*, R*), const R* t, R* o)
{
    for (int j = 0; j < 3; ++j) {
        R n[3] = { 0, 0, 0 }, c[3];
        n[j] = 1;
        map(n, c);
        o[j] = c[0] * t[0] + c[1] * t[1] + c[2] * t[2];
    }
}
static void columns(const i64 (&n)[9], i64 (&val)[3][3], i64 (&der)[3][3]) // [row][column]
{
    for (int c = 0; c < 3; ++c) {
        const i64 a[3] = { n[c], n[3 + c], n[6 + c] };
        i64 v[3], d[3];
        interp(a, v);
        deriv(a, d);
        for (int r = 0; r < 3; ++r) { val[r][c] = v[r]; der[r][c] = d[r]; }
    }
}
int main(int argc, char** argv)
{
    const double rho = std::atof(argv[1]);
    std::mt19937_64 gen(3);
    std::uniform_real_distribution<double> U(-1, 1);
    R conv = 0, near = 0, prod = 0, strain = 0, share = 0;
    for (int i = 0; i < 200000; ++i) {
        const int top = 200 + int(gen() % 1600), bits = 50 + int(gen() % 9);
        const double x = std::ldexp(U(gen), top - 1022 - int(gen() % 70) * (i & 1));
        const i64 X = toFixed(x, fixedShift(bits, top));
        const int scale = bits - top + 1022;
        conv = std::max(conv, fabsl(ldexpl(R(x), scale) - X));
        const i64 Y = static_cast<i64>(gen()) >> (gen() % 63);
        const double y = toDouble(Y, doubleExponent(scale));
        near = std::max(near, fabsl(R(y) - ldexpl(R(Y), -scale)) / std::max(fabsl(R(y)) * 0x1p-53L, ldexpl(1, -1074)));
        const u64 c = gen() >> (1 + gen() % 20);
        if (c < (0x7fffffffull << 32))
            prod = std::max(prod, R(std::llabs(mul(Y, coefOf(c)) - static_cast<i64>((static_cast<__int128>(Y) * c) >> 64))));
    }
    const R unit = ldexpl(1, 64);
    R high = 0;
    for (int i = 0; i < 200000; ++i) {
        const i64 most = static_cast<i64>(0x1p61 * 1.41), one = 1ll << 62;
        auto any = [&](i64 m) { return i < 64 ? (gen() & 1 ? m - 1 : 1 - m) : static_cast<i64>(U(gen) * m) >> (gen() % 40); };
        const i64 x = any(most), y = any(most), k = any(one), l = any(one);
        const R a = R(x) * k / unit, b = R(y) * l / unit;
        high = std::max(high, fabsl(mulHigh(Split(x), unpacked(packed(k))) - a) / 2);
        high = std::max(high, fabsl(mulHigh(Split(x), unpacked(packed(k)), Split(y), unpacked(packed(l))) - (a + b)) / 3);
    }
    const Scaled sc(rho);
    const int bits = std::min(58, 61 - sc.shift), bitsP = 58 - sc.shift;
    for (int i = 0; i < 20000; ++i) {
        i64 u[9], val[3][3], der[3][3];
        R v[3][3], d[3][3];
        const i64 most = (1ll << bits) - 1;
        for (int j = 0; j < 9; ++j)
            u[j] = i < 512 ? ((i >> j) & 1 ? most : -most) : static_cast<i64>(U(gen) * most);
        columns(u, val, der);
        for (int c = 0; c < 3; ++c) {
            const R a[3] = { R(u[c]), R(u[3 + c]), R(u[6 + c]) };
            R x[3], y[3];
            interpR(a, x);
            derivR(a, y);
            for (int r = 0; r < 3; ++r) { v[r][c] = x[r]; d[r][c] = y[r]; }
        }
        for (int r = 0; r < 3; ++r) {
            i64 a[3], b[3];
            R x[3], y[3];
            deriv(val[r], a);
            sc.interp(der[r], b);
            derivR(v[r], x);
            interpR(d[r], y);
            for (int j = 0; j < 3; ++j) // the largest of the three sums taken of a strain's parts
                strain = std::max(strain, fabsl(R(a[j] + b[j]) - (x[j] + rho * y[j])));
        }
        // increments f (to the derivative along xi) and h (along eta)
        const i64 F = (1ll << (bitsP - 1));
        i64 ox[3][3], oy[3][3];
        R px[3][3], py[3][3];
        for (int r = 0; r < 3; ++r) {
            i64 f[3], h[3];
            R fr[3], hr[3];
            for (int j = 0; j < 3; ++j) {
                const int sign = (i >> (3 * r + j)) & 1 ? 1 : -1;
                f[j] = static_cast<i64>(F * (i < 512 ? sign * 4.3 : 4.3 * U(gen)));
                h[j] = static_cast<i64>(F * (i < 512 ? sign * 4.3 : 4.3 * U(gen)));
                fr[j] = f[j];
                hr[j] = h[j];
            }
            derivT(f, ox[r]);
            sc.interpT(h, oy[r]);
            transposed(derivR, fr, px[r]);
            transposed(interpR, hr, py[r]);
        }
        for (int c = 0; c < 3; ++c) {
            const i64 x[3] = { ox[0][c], ox[1][c], ox[2][c] }, y[3] = { oy[0][c], oy[1][c], oy[2][c] };
            i64 o[3];
            columnT(x, y, o);
            const R xr[3] = { px[0][c], px[1][c], px[2][c] }, yr[3] = { rho * py[0][c], rho * py[1][c], rho * py[2][c] };
            R a[3], b[3];
            transposed(interpR, xr, a);
            transposed(derivR, yr, b);
            for (int r = 0; r < 3; ++r)
                share = std::max(share, fabsl(R(o[r]) - (a[r] + b[r])));
        }
    }
    std::printf("%.6Lf %.6Lf %.6Lf %.6Lf %.6Lf %.6Lf %d\n", conv, near, prod, high, strain, share, sc.shift);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("fixed_maps")
    (d / "a.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", str(ROOT / "nextsimdg_gb300" / "csrc"), str(d / "a.cpp"), "-o",
                    str(d / "a")], check=True)
    return d / "a"


@pytest.mark.parametrize("rho", [1 / 31.999, 0.26, 0.9999999999999999, 1.0, 1.9999999999999998, 2.0, 7.3, 31.999])
def test_within_units_of_the_exact_maps(program, rho):
    """A conversion to fixed point is truncated (below one unit), one to FP64
    rounded to nearest (half an ulp, at most 2^-53 of the value), a product
    within two units (a sum of two with packed factors within three).  A strain then has at most 4 units from a column's value
    and 8 from its derivative, 8 + 4 (2 + 16 g) = 41 in a row's derivative and
    rho (1.2 8 + 2^shift / rho 3 2) from a row's scaled interpolation; a share 2 4
    = 8 from a row's transposed derivative and 2^shift 4 from its transposed
    interpolation, which a column's maps multiply by at most 2 (1.2 + 4 g) with 12
    of their own."""
    conv, near, prod, high, strain, share, shift = map(float, subprocess.check_output([str(program), repr(rho)]).split())
    assert conv < 1.0
    assert near <= 1.0
    assert prod <= 2.0
    assert high <= 1.0
    assert strain <= 41 + 10 * rho + 6 * 2 ** shift
    assert share <= 12 + 6.2 * (8 + 4 * 2 ** shift)
