// nsdg_fixed.hpp — linear maps of FP64 data in 64-bit fixed point (host and
// device).
//
// GB300 issues an FP64 addition or FMA of a warp every 18 SM cycles, a 64-bit
// integer addition every 0.6 and the product below every 5, on pipes of their
// own.  Where a block of values goes through linear maps with known bounds, the
// block's largest exponent gives it one binary scale, and the maps run on
// integers: sums are exact, a product is rounded to the block's unit, and with
// 56 to 58 bits below the largest input the unit is below the rounding error of
// the same maps in FP64.
#pragma once

#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#define NSDG_FX_HD __host__ __device__ __forceinline__
#else
#define NSDG_FX_HD inline
#endif

namespace nsdg {
namespace fx {

using i64 = long long;
using u64 = unsigned long long;

NSDG_FX_HD u64 bitsOf(double d)
{
#if defined(__CUDA_ARCH__)
    return static_cast<u64>(__double_as_longlong(d));
#else
    u64 u;
    std::memcpy(&u, &d, sizeof u);
    return u;
#endif
}
NSDG_FX_HD double doubleOf(u64 u)
{
#if defined(__CUDA_ARCH__)
    return __longlong_as_double(static_cast<i64>(u));
#else
    double d;
    std::memcpy(&d, &u, sizeof d);
    return d;
#endif
}
// a >> s, 0 for s > 63
NSDG_FX_HD u64 shiftRight(u64 a, unsigned s)
{
#if defined(__CUDA_ARCH__)
    u64 r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(a), "r"(s)); // clamps s
    return r;
#else
    return s > 63 ? 0 : a >> s;
#endif
}
NSDG_FX_HD int leadingZeros(u64 a) // a != 0
{
#if defined(__CUDA_ARCH__)
    return __clzll(static_cast<i64>(a));
#else
    return __builtin_clzll(a);
#endif
}
NSDG_FX_HD i64 shiftLeft(i64 x, int s) { return static_cast<i64>(static_cast<u64>(x) << s); }

// the upper word of |x|: orders magnitudes, its bits 20 .. 30 are the exponent
NSDG_FX_HD int magnitudeWord(double x) { return static_cast<int>(bitsOf(x) >> 32) & 0x7fffffff; }

// x 2^(bits - (top - 1022)) truncated, for |x| < 2^(top - 1022), top > 63:
// a value below 2^bits; at = fixedShift(bits, top)
NSDG_FX_HD int fixedShift(int bits, int top) { return 64 - bits + top; }
NSDG_FX_HD i64 toFixed(double x, int at)
{
    const u64 b = bitsOf(x);
    const unsigned ex = static_cast<unsigned>(b >> 52) & 0x7ffu;
    const i64 a = static_cast<i64>(shiftRight((b << 11) | (1ull << 63), static_cast<unsigned>(at) - ex));
    const i64 neg = static_cast<i64>(b) >> 63;
    return (a ^ neg) - neg;
}
// X 2^-scale to nearest (ties away), for results below 2^1023; 0 below 2^-1022;
// at = doubleExponent(scale)
NSDG_FX_HD int doubleExponent(int scale) { return 1086 - scale; }
NSDG_FX_HD double toDouble(i64 X, int at)
{
    const i64 neg = X >> 63;
    const u64 a = static_cast<u64>((X ^ neg) - neg);
    const int z = leadingZeros(a | 1);
    const u64 m = a << z;
    const int ex = at - z;
    const u64 r = (m >> 11) + ((m >> 10) & 1);
    const u64 v = (static_cast<u64>(static_cast<unsigned>(ex - 1)) << 52) + r;
    return X == 0 || ex < 1 ? 0.0 : doubleOf(v | (static_cast<u64>(neg) & (1ull << 63)));
}

// a factor 0 <= c < 1/2 - 2^-32 as hi 2^-32 + lo 2^-64
struct Coef {
    int hi, lo;
};
NSDG_FX_HD constexpr Coef coefOf(u64 c) // c 2^-64
{
    return Coef { static_cast<int>((c >> 32) + ((c >> 31) & 1)), static_cast<int>(static_cast<unsigned>(c)) };
}
// x = hi 2^32 + lo with lo signed (|x| < 2^63 - 2^32)
struct Split {
    int hi, lo;
    NSDG_FX_HD explicit Split(i64 x) : lo(static_cast<int>(static_cast<unsigned>(x)))
    {
        hi = static_cast<int>(x >> 32) + static_cast<int>(static_cast<unsigned>(x) >> 31);
    }
};
constexpr i64 kHalfWord = 1ll << 31;
NSDG_FX_HD i64 wide(int a, int b, i64 c) { return static_cast<i64>(a) * b + c; }
// c x to nearest (within a unit: the product of the lower words is left out):
// three multiplications with 64-bit addends
NSDG_FX_HD i64 mul(Split x, Coef c)
{
    return wide(x.hi, c.hi, wide(x.lo, c.hi, wide(x.hi, c.lo, kHalfWord)) >> 32);
}
NSDG_FX_HD i64 mul(i64 x, Coef c) { return mul(Split(x), c); }
// a factor |k| < 2^62 for the products below, hi and lo as in Split
NSDG_FX_HD i64 packed(i64 k)
{
    const Split s(k);
    return static_cast<i64>((static_cast<u64>(static_cast<unsigned>(s.hi)) << 32) | static_cast<unsigned>(s.lo));
}
NSDG_FX_HD Split unpacked(i64 p)
{
    Split s(0);
    s.hi = static_cast<int>(p >> 32);
    s.lo = static_cast<int>(static_cast<unsigned>(p));
    return s;
}
// (k x) 2^-64 and (k x + l y) 2^-64, to nearest within a unit, for |x|, |y| <
// 2^61.5: the middle sums stay below 2^63
NSDG_FX_HD i64 mulHigh(Split x, Split k)
{
    return wide(x.hi, k.hi, wide(x.lo, k.hi, wide(x.hi, k.lo, kHalfWord)) >> 32);
}
NSDG_FX_HD i64 mulHigh(Split x, Split k, Split y, Split l)
{
    const i64 t = wide(y.lo, l.hi, wide(y.hi, l.lo, wide(x.lo, k.hi, wide(x.hi, k.lo, kHalfWord))));
    return wide(x.hi, k.hi, wide(y.hi, l.hi, t >> 32));
}
// (c x) 2^-62 for |c| <= 2^62 and |c x| < 2^124.5, and the sum of three such
// products with |c0| + |c1| + |c2| <= 2^62 and |x| < 2^60
NSDG_FX_HD i64 mulUnit(Split x, Split c)
{
    return shiftLeft(wide(x.hi, c.hi, 0), 2) + (wide(x.lo, c.hi, wide(x.hi, c.lo, 1ll << 29)) >> 30);
}
NSDG_FX_HD i64 dotUnit(const Split (&x)[3], const Split (&c)[3])
{
    i64 t = 1ll << 29, h = 0;
    for (int i = 0; i < 3; ++i) {
        t = wide(x[i].lo, c[i].hi, wide(x[i].hi, c[i].lo, t));
        h = wide(x[i].hi, c[i].hi, h);
    }
    return shiftLeft(h, 2) + (t >> 30);
}

// Scales that follow the values.  The upper words of some values, each as a
// magnitude, or'ed: the values are below 2^(their length); 2^32 is the least.
NSDG_FX_HD int upperMagnitude(i64 x)
{
    const int h = static_cast<int>(x >> 32);
    return h ^ (h >> 31);
}
NSDG_FX_HD int lengthOf(int upper)
{
#if defined(__CUDA_ARCH__)
    return 64 - __clz(upper);
#else
    return upper ? 64 - __builtin_clz(static_cast<unsigned>(upper)) : 32;
#endif
}
// x 2^s, floored for s < 0
struct Shift {
    int left, right;
    NSDG_FX_HD explicit Shift(int s) : left(s > 0 ? s : 0), right(s > 0 ? 0 : s < -63 ? 63 : -s) { }
    NSDG_FX_HD i64 operator()(i64 x) const { return shiftLeft(x, left) >> right; }
};

// The 1-D maps of the element update on a line of three nodes or Gauss points
// (Line in nsdg_sumfact.cuh).
constexpr Coef kG = coefOf(0x6325fbd0fdc91f05ull);  // sqrt(3/20)
constexpr Coef kC3 = coefOf(0x4ccccccccccccccdull); // 0.3
constexpr Coef kC4 = coefOf(0x6666666666666666ull); // 0.4

// 4 g x = x + 2 (2 g - 1/2) x
constexpr Coef kG4 = coefOf(0x464bf7a1fb923e09ull); // 2 sqrt(3/20) - 1/2
NSDG_FX_HD i64 times4G(i64 x) { return x + 2 * mul(x, kG4); }
NSDG_FX_HD void interp(const i64 (&n)[3], i64 (&o)[3])
{
    const i64 m = n[1] + mul(n[0] + n[2] - 2 * n[1], kC3), q = mul(n[2] - n[0], kG);
    o[0] = m - q;
    o[1] = n[1];
    o[2] = m + q;
}
NSDG_FX_HD void deriv(const i64 (&n)[3], i64 (&o)[3])
{
    const i64 d = n[2] - n[0], k = times4G(n[0] + n[2] - 2 * n[1]);
    o[0] = d - k;
    o[1] = d;
    o[2] = d + k;
}
NSDG_FX_HD void interpT(const i64 (&t)[3], i64 (&o)[3])
{
    const i64 s = t[0] + t[2], m = mul(s, kC3), q = mul(t[2] - t[0], kG);
    o[0] = m - q;
    o[1] = t[1] + mul(s, kC4);
    o[2] = m + q;
}
NSDG_FX_HD void derivT(const i64 (&t)[3], i64 (&o)[3])
{
    const i64 s = t[0] + t[1] + t[2], k = times4G(t[2] - t[0]);
    o[0] = k - s;
    o[1] = -2 * k;
    o[2] = k + s;
}
// interp and interpT times rho = m 2^shift, m < 1/4; S: the shift where it is
// known (rho < 2^(S - 2))
template <int S = 0> struct Scaled {
    Coef m, g, c3, c4;
    int shift;
    NSDG_FX_HD explicit Scaled(double rho) // 2^-5 <= rho <= 2^5
    {
        const u64 b = bitsOf(rho);
        const int ex = static_cast<int>(b >> 52) & 0x7ff;
        shift = S > 0 ? S : ex < 1023 ? 2 : ex - 1020;
        const u64 f = (b & 0xfffffffffffffull) | (1ull << 52);
        const u64 r = f << (ex - 1011 - shift);
        m = coefOf(r);
        g = coefOf(static_cast<u64>(fx::mul(static_cast<i64>(r), kG)));
        c3 = coefOf(static_cast<u64>(fx::mul(static_cast<i64>(r), kC3)));
        c4 = coefOf(static_cast<u64>(fx::mul(static_cast<i64>(r), kC4)));
    }
    // c x 2^shift to nearest (within a unit and 2^(shift - 2))
    NSDG_FX_HD i64 times(Split x, Coef c) const
    {
        const int s = S > 0 ? S : shift;
        return shiftLeft(wide(x.hi, c.hi, 0), s)
            + (wide(x.lo, c.hi, wide(x.hi, c.lo, kHalfWord >> s)) >> (32 - s));
    }
    NSDG_FX_HD i64 times(i64 x, Coef c) const { return times(Split(x), c); }
    NSDG_FX_HD void interp(const i64 (&n)[3], i64 (&o)[3]) const
    {
        const i64 c = times(n[1], m), t = c + times(n[0] + n[2] - 2 * n[1], c3), q = times(n[2] - n[0], g);
        o[0] = t - q;
        o[1] = c;
        o[2] = t + q;
    }
    NSDG_FX_HD void interpT(const i64 (&t)[3], i64 (&o)[3]) const
    {
        const i64 s = t[0] + t[2], a = times(s, c3), q = times(t[2] - t[0], g);
        o[0] = a - q;
        o[1] = times(s, c4) + times(t[1], m);
        o[2] = a + q;
    }
};
// the transposed maps of a column (columnT in nsdg_sumfact.cuh)
NSDG_FX_HD void columnT(const i64 (&x)[3], const i64 (&y)[3], i64 (&o)[3])
{
    const i64 s = x[2] + x[0], k = times4G(y[2] - y[0]);
    const i64 p = mul(s, kC3) + k, q = mul(x[2] - x[0], kG) + y[0] + y[1] + y[2];
    o[0] = p - q;
    o[1] = x[1] + mul(s, kC4) - 2 * k;
    o[2] = p + q;
}

} // namespace fx
} // namespace nsdg
