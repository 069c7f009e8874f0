// nsdg_bbm.cu — the brittle (BBM) sub-cycle (BBMStressUpdateStep.hpp:31-195,
// BrittleCGDynamicsKernel.hpp:206-254).
//
// Through the sub-steps of a model step the stress and the damage are kept as
// their values at the 3 x 3 Gauss points instead of 8 and DG coefficients.
// The update works on point values, and the projection back onto the modes is
// all that a sub-step needs of the coefficients:
//   stress   g <- P f,  P = I - n nu^T   (nsdg_sumfact.cuh: one rank is lost)
//   damage   d <- Psi (Psi^T W Psi)^{-1} Psi^T W d
// Point values of a field in the modes' span and its coefficients carry the
// same information, so kBbmLoad forms the values once per step and kBbmStore
// the coefficients.  Thickness and concentration do not change through the
// sub-steps either: the terms formed from them (exponentials, powers, roots)
// are six constants per point and step.
#include <cmath>
#include <type_traits>

#include "nsdg_exp64.cuh"
#include "nsdg_modes.cuh"
#include "nsdg_nodes.cuh"
#include "nsdg_prep.cuh"
#include "nsdg_stress_fixed.cuh"
#include "nsdg_sumfact.cuh"
#include "nsdg_visc_ff.hpp"

namespace nsdg {
namespace {

using namespace sf;

// x^y for x >= 0: by multiplication when y is a small integer (mode 1), times
// sqrt(x) when it is a small half-integer (mode 2), else pow().  Differs from
// pow() by a few ulps.
template <typename T> __device__ __forceinline__ T powByMode(T x, T y, int mode, int k)
{
    if (mode == 0)
        return pow(x, y);
    T r = T(1);
    for (int i = 0; i < k; ++i)
        r *= x;
    return mode == 2 ? r * sqrt(x) : r;
}

// FP64 <-> the point values' and node constants' type on the integer pipe
template <typename T> __device__ __forceinline__ T store(double x)
{
    if constexpr (sizeof(T) == 8)
        return x;
    else
        return nsdg_ff::narrowAny(x);
}
__device__ __forceinline__ double load(double x) { return x; }
__device__ __forceinline__ double load(float x)
{
    const unsigned b = __float_as_uint(x), m = b & 0x7fffffffu;
    if (m >= 0x7f800000u)
        return static_cast<double>(x);
    const double y = nsdg_ff::widenNonneg(__uint_as_float(m));
    return __hiloint2double(__double2hiint(y) | static_cast<int>(b & 0x80000000u), __double2loint(y));
}
// sqrt(x), x often 0 (open water, calm)
__device__ __forceinline__ double rootOf(double x) { return __double_as_longlong(x) == 0 ? 0.0 : sqrt64(x); }

// 1-D Gauss weights and points on [-1/2, 1/2], Legendre mode 2 there
constexpr double kG = 0.38729833462074168852;
constexpr double kL2Norm = 1. / 180.; // sum w L2^2
__host__ __device__ constexpr double kW(int i) { return i == 1 ? 8. / 18. : 5. / 18.; }
__host__ __device__ constexpr double kX(int i) { return i == 0 ? -kG : i == 1 ? 0.0 : kG; }
__host__ __device__ constexpr double kL2(int i) { return (i == 1 ? 0.0 : 0.15) - 1. / 12.; }
__host__ __device__ constexpr double kN(int i) { return i == 1 ? -5. / 18. : 2. / 9.; } // (nu / w) / sum(nu^2 / w)

// DG mode j (x-y degrees) at Gauss point (ix, iy) and 1 / (its squared norm)
__device__ constexpr int modeX(int j) { return j == 1 || j == 5 || j == 7 ? 1 : j == 3 || j == 6 ? 2 : 0; }
__device__ constexpr int modeY(int j) { return j == 2 || j == 5 || j == 6 ? 1 : j == 4 || j == 7 ? 2 : 0; }
__device__ __forceinline__ constexpr double leg(int n, int i) { return n == 0 ? 1.0 : n == 1 ? kX(i) : kL2(i); }
__device__ __forceinline__ constexpr double psiAt(int j, int q) { return leg(modeX(j), q % 3) * leg(modeY(j), q / 3); }

// Step constants and point values from the advected fields, and the Lagrange
// values of h and A for the nodes.  Bound by FP64 issue: 256 x 256 elements with
// six modes, FP32 targets, 130 us (155 us with dense products and CUDA's exp,
// roots and divisions, without the Lagrange values).
template <typename T, int DG>
__global__ void __launch_bounds__(128) kBbmLoad(size_t N, const double* __restrict__ h, const double* __restrict__ a,
    const double* __restrict__ damage, const double* __restrict__ s11, const double* __restrict__ s12,
    const double* __restrict__ s22, const double* __restrict__ hsize, const double* __restrict__ invKx2,
    BbmPoints<T> pt, double* __restrict__ lagH, double* __restrict__ lagA, BbmParams p)
{
    const size_t e = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
    if (e >= N)
        return;
    double hc[DG], ac[DG], dc[DG];
#pragma unroll
    for (int j = 0; j < DG; ++j) {
        hc[j] = h[j * N + e];
        ac[j] = a[j * N + e];
        dc[j] = damage[j * N + e];
    }
    storeLagrange<DG>(hc, ac, N, e, lagH, lagA);
    double hg[9], ag[9], dg[9];
    gaussValues<DG>(hc, hg);
    gaussValues<DG>(ac, ag);
    gaussValues<DG>(dc, dg);
    const double size = hsize[e];
    const double sizeScale = sqrt64(0.1 * recip64(size));
    // relax = (1 - dcrit) dt / td, td = size sqrt(2 (1 + nu0) rho) / sqrt(elasticity)
    const double relaxScale = p.dt * recip64(size * p.soundRoot);
    // the kernels' half strains, over k_x on rectangles
    const double strain = invKx2 ? timesRsqrt64(p.strainScale, invKx2[e]) : p.strainScale;
    const double lab = p.C_lab * sizeScale, crush = p.compr_strength * sizeScale;
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        const double hG = atLeast(hg[q], 0.0), aG = atMost(atLeast(ag[q], 0.0), 1.0);
        const double expC = exp64(p.compaction_param * (1.0 - aG));
        const double hE = hG * expC;
        const size_t at = q * N + e;
        pt.c[0 * 9 * N + at] = store<T>(hE * strain);
        pt.c[1 * 9 * N + at] = store<T>(
            p.P0 * powByMode(hG, p.exponent_compression_factor + 1., p.powCmode, p.powCk) * expC);
        const double tv = p.lambda * powByMode(expC, p.exponent_relaxation_sigma - 1., p.powRmode, p.powRk);
        // FP64: the viscous relaxation time over damage^(n-1); FP32: dt over it
        // (the time itself underflows in open water)
        if constexpr (sizeof(T) == 8)
            pt.c[2 * 9 * N + at] = tv;
        else
            pt.c[2 * 9 * N + at] = store<T>(p.dt * recip64(tv));
        pt.c[3 * 9 * N + at] = store<T>(lab * hG);
        pt.c[4 * 9 * N + at] = store<T>(crush * hG);
        pt.c[5 * 9 * N + at] = store<T>(relaxScale * rootOf(hE * p.young)); // of elasticity / damage
        pt.d[at] = store<T>(dg[q]);
    }
    const double* src[3] = { s11, s12, s22 };
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        double m[8], v[9];
#pragma unroll
        for (int j = 0; j < 8; ++j)
            m[j] = src[c][j * N + e];
        gaussValues<8>(m, v);
#pragma unroll
        for (int q = 0; q < 9; ++q)
            pt.s[(c * 9 + q) * N + e] = store<T>(v[q]);
    }
}

// The coefficients of the point values (which lie in the modes' span: the
// unit square's projection gives them on every mesh).
template <typename T, int DG>
__global__ void __launch_bounds__(128) kBbmStore(size_t N, BbmPoints<T> pt, double* __restrict__ damage,
    double* __restrict__ s11, double* __restrict__ s12, double* __restrict__ s22)
{
    const size_t e = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
    if (e >= N)
        return;
    auto project = [&](const T* src, auto modes, double* out) {
        constexpr int M = decltype(modes)::value;
        double v[9], c[M];
#pragma unroll
        for (int q = 0; q < 9; ++q)
            v[q] = load(src[q * N + e]);
        modesOf<M>(v, c);
#pragma unroll
        for (int j = 0; j < M; ++j)
            out[j * N + e] = c[j];
    };
    project(pt.d, std::integral_constant<int, DG>(), damage);
    double* dst[3] = { s11, s12, s22 };
#pragma unroll
    for (int c = 0; c < 3; ++c)
        project(pt.s + size_t(9) * c * N, std::integral_constant<int, 8>(), dst[c]);
}

// min(max(d, 1e-12), 1) on the integer pipe (NaN gives 1e-12, as fmax does)
__device__ __forceinline__ double clampDamage(double d)
{
    const long long b = __double_as_longlong(d);
    constexpr long long lo = 0x3d719799812dea11ll, hi = 0x3ff0000000000000ll; // 1e-12, 1
    const bool nan = (b & 0x7fffffffffffffffll) > 0x7ff0000000000000ll;
    return __longlong_as_double(nan || b < lo ? lo : b > hi ? hi : b);
}
__device__ __forceinline__ float clampDamage(float d) { return fminf(fmaxf(d, 1e-12f), 1.f); }
// comparisons on the bit patterns (an FP64 comparison issues at the FP64 rate)
__device__ __forceinline__ long long bitsT(double x) { return __double_as_longlong(x); }
__device__ __forceinline__ int bitsT(float x) { return __float_as_int(x); }
__device__ __forceinline__ unsigned long long magnitudeT(double x) { return static_cast<unsigned long long>(bitsT(x)); }
__device__ __forceinline__ unsigned magnitudeT(float x) { return static_cast<unsigned>(bitsT(x)); }
template <typename T> __device__ __forceinline__ bool above0(T x) { return bitsT(x) > 0; }
// min(x, 1) for x >= 0; NaN of either sign (0 / 0 in open water) gives 1, as fmin does
template <typename T> __device__ __forceinline__ T min1(T x) { return magnitudeT(x) < magnitudeT(T(1)) ? x : T(1); }
__device__ __forceinline__ bool finiteT(double x) { return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000; }
__device__ __forceinline__ bool finiteT(float x) { return (__float_as_int(x) & 0x7f800000) != 0x7f800000; }
__device__ __forceinline__ double recipT(double x) { return recip64(x); }
__device__ __forceinline__ float recipT(float x) { return 1.f / x; }
__device__ __forceinline__ double sqrtT(double x) { return sqrt64(x); }
__device__ __forceinline__ float sqrtT(float x) { return sqrtf(x); }

template <typename T> struct BbmScalars {
    T dt, nu0, halfOneMinusNu, tanPhi, relaxExp;
    int powRmode, powRk;
};

// One Gauss point: the elastic-viscous stress update and the damage
// (BBMStressUpdateStep.hpp:89-166) from half strains a, b, s times the
// element's factor in c[0].
template <typename T>
__device__ __forceinline__ void bbmPoint(T a, T b, T s, const T (&c)[6], const BbmScalars<T>& k, T& g11, T& g12,
    T& g22, T& d)
{
    d = clampDamage(d);
    T press = T(-0.5) * (g11 + g22); // -sigma_n
    T open = T(1);
    if (above0(press))
        open = T(1) - min1(c[1] * recipT(press));
    T mult;
    if constexpr (sizeof(T) == 8) {
        const T tv = c[2] * powByMode(d, k.relaxExp, k.powRmode, k.powRk);
        mult = tv * recipT(fmaT(open, k.dt, tv));
    } else {
        const T r = above0(open) ? open * c[2] * powByMode(T(1) / d, k.relaxExp, k.powRmode, k.powRk) : T(0);
        mult = T(1) / (T(1) + r);
    }
    const T du = c[0] * d;
    g11 = mult * fmaT(du, fmaT(k.nu0, b, a), g11);
    g22 = mult * fmaT(du, fmaT(k.nu0, a, b), g22);
    g12 = mult * fmaT(du, k.halfOneMinusNu * s, g12);
    press = T(-0.5) * (g11 + g22);
    const T dd = T(0.5) * (g11 - g22);
    const T tau = sqrtT(fmaT(dd, dd, g12 * g12));
    // dcrit: cohesion / (tau + tan_phi sigma_n) above the Mohr-Coulomb line,
    // -compr / sigma_n beyond the compressive strength
    const T mc = fmaT(-k.tanPhi, press, tau);
    const bool crush = bitsT(press) > bitsT(c[4]); // press > the strength (>= 0)
    const T num = crush ? c[4] : c[3], den = crush ? press : mc;
    T dcrit = T(1);
    if (above0(den))
        dcrit = min1(num * recipT(den));
    const T keep = fmaT(dcrit - T(1), c[5] * sqrtT(d), T(1));
    d *= keep;
    g11 *= keep;
    g12 *= keep;
    g22 *= keep;
}

// P f and the damage's projection of row R, and the new state: sums over the
// three rows in sum[row][9][E] (nu . f, 3, and the damage's moments, 3 or DG).
template <typename T, Geometry GEO, int DG, int E>
__device__ __forceinline__ void bbmProject(int R, size_t e, size_t N, bool in, const T* __restrict__ wdam,
    const T (&nq)[3], const BbmPoints<T>& pt, T (&g)[3][3], T (&d)[3], T (*sum)[9][E], int le)
{
    const bool mid = R == 1;
    const T nr = mid ? T(-2) : T(1);
#pragma unroll
    for (int f = 0; f < 3; ++f)
        sum[R][f][le] = nr * fmaT(T(-2), g[f][1], g[f][0] + g[f][2]);
    [[maybe_unused]] T m0 = T(0), m1 = T(0), m2 = T(0);
    if constexpr (GEO == QUAD) {
#pragma unroll
        for (int j = 0; j < DG; ++j) {
            T t = T(0);
#pragma unroll
            for (int i = 0; i < 3; ++i)
                t = fmaT(in ? wdam[(j * 9 + 3 * R + i) * N + e] : T(0), d[i], t);
            sum[R][3 + j][le] = t;
        }
    } else {
        // the row's Legendre coefficients along xi
        // (the mean as d[1] plus differences: constants stay exact)
        const T t2 = fmaT(T(-2), d[1], d[0] + d[2]);
        m0 = fmaT(T(kW(0)), t2, d[1]);
        m1 = T(0.5 / kG) * (d[2] - d[0]);
        m2 = T(0.5 / (kG * kG)) * t2;
        sum[R][3][le] = m0;
        sum[R][4][le] = m1;
        sum[R][5][le] = m2;
    }
    __syncthreads();
    [[maybe_unused]] const T nRow = mid ? T(kN(1)) : T(kN(0));
#pragma unroll
    for (int f = 0; f < 3; ++f) {
        const T l = sum[0][f][le] + sum[1][f][le] + sum[2][f][le];
#pragma unroll
        for (int i = 0; i < 3; ++i)
            g[f][i] = fmaT(-l, GEO == QUAD ? nq[i] : nRow * T(kN(i)), g[f][i]);
    }
    if constexpr (GEO == QUAD) {
        T cf[DG];
#pragma unroll
        for (int j = 0; j < DG; ++j)
            cf[j] = sum[0][3 + j][le] + sum[1][3 + j][le] + sum[2][3 + j][le];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            T t = T(0);
#pragma unroll
            for (int j = 0; j < DG; ++j)
                t = fmaT(cf[j], mid ? T(psiAt(j, 3 + i)) : R == 0 ? T(psiAt(j, i)) : T(psiAt(j, 6 + i)), t);
            d[i] = t;
        }
    } else {
        // modes of total degree <= 2 (DG 6), 1 (DG 3) or 0 (DG 1) stay
        auto at = [&](int m, int r) { return sum[r][3 + m][le]; };
        auto second = [&](int m) { return fmaT(T(-2), at(m, 1), at(m, 0) + at(m, 2)); };
        auto mean = [&](int m) { return fmaT(T(kW(0)), second(m), at(m, 1)); };
        // the row value of the part of a coefficient that is quadratic in eta
        const T qRow = (mid ? T(kL2(1)) : T(kL2(0))) * T(kW(0) * kL2(0) / kL2Norm);
        auto quadratic = [&](int m) { return qRow * second(m); };
        if constexpr (DG == 6) {
            const T d1 = quadratic(1), d2 = m2 - mean(2);
#pragma unroll
            for (int i = 0; i < 3; ++i)
                d[i] = fmaT(-d2, T(kL2(i)), fmaT(-d1, T(kX(i)), d[i]));
        } else if constexpr (DG == 3) {
            const T c0 = m0 - quadratic(0), c1 = mean(1);
#pragma unroll
            for (int i = 0; i < 3; ++i)
                d[i] = fmaT(c1, T(kX(i)), c0);
        } else {
            const T c0 = mean(0);
#pragma unroll
            for (int i = 0; i < 3; ++i)
                d[i] = c0;
        }
    }
    if (in) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const size_t q = 3 * R + i;
            pt.d[q * N + e] = d[i];
#pragma unroll
            for (int f = 0; f < 3; ++f)
                pt.s[(9 * f + q) * N + e] = g[f][i];
        }
    }
}

template <typename T, int E> struct BbmShared {
    Exchange<T, E> ex;
    T strain[3][3][E]; // nu . strain per row
    T sum[3][9][E];
};

// Row R of an element in FP32: see kBbmStress.
template <Geometry GEO, int DG, int E>
__device__ __forceinline__ void bbmRow(int R, size_t e, size_t N, bool in, const StressGeometry<float>& geo,
    const float* __restrict__ wdam, const float* __restrict__ wj, const BbmPoints<float>& pt, const float (&ke)[4],
    float weight, const float (&c)[3][6], float (&g)[3][3], float (&d)[3], const BbmScalars<float>& k,
    BbmShared<float, E>& sh, int le)
{
    using T = float;
    T I[3], D[3], uxi[3], uet[3], vxi[3], vet[3], a[3], b[3], s[3];
    auto take = [&](int f) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            I[i] = sh.ex.in.v[f][R][i][le];
            D[i] = sh.ex.in.dv[f][R][i][le];
        }
    };
    take(0);
    deriv(I, uxi);
    interp(D, uet);
    take(1);
    deriv(I, vxi);
    interp(D, vet);
    const bool mid = R == 1;
    const T nr = mid ? T(-2) : T(1);
    T k0[3], k1[3], k2[3], k3[3];
    [[maybe_unused]] T nq[3] = { T(0), T(0), T(0) };
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const size_t q = 3 * R + i;
        if constexpr (GEO == AFFINE) {
            k0[i] = ke[0];
            k1[i] = ke[1];
            k2[i] = ke[2];
            k3[i] = ke[3];
        } else {
            k0[i] = in ? geo.k[q * N + e] : T(0);
            k1[i] = in ? geo.k[(9 + q) * N + e] : T(0);
            k2[i] = in ? geo.k[(18 + q) * N + e] : T(0);
            k3[i] = in ? geo.k[(27 + q) * N + e] : T(0);
            nq[i] = in ? geo.n[q * N + e] : T(0);
        }
        a[i] = fmaT(k0[i], uxi[i], k1[i] * uet[i]);
        b[i] = fmaT(k2[i], vxi[i], k3[i] * vet[i]);
        s[i] = fmaT(k2[i], uxi[i], fmaT(k3[i], uet[i], fmaT(k0[i], vxi[i], k1[i] * vet[i])));
    }
    if constexpr (GEO == QUAD) {
        T l[3] = { nr * fmaT(T(-2), a[1], a[0] + a[2]), nr * fmaT(T(-2), b[1], b[0] + b[2]),
            nr * fmaT(T(-2), s[1], s[0] + s[2]) };
        sumRows<T, E>(sh.strain, R, le, l);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            a[i] = fmaT(-l[0], nq[i], a[i]);
            b[i] = fmaT(-l[1], nq[i], b[i]);
            s[i] = fmaT(-l[2], nq[i], s[i]);
        }
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
        bbmPoint(a[i], b[i], s[i], c[i], k, g[0][i], g[1][i], g[2][i], d[i]);
    bbmProject<T, GEO, DG, E>(R, e, N, in, wdam, nq, pt, g, d, sh.sum, le);
    // the divergence K^T (w J g) of this row: xi maps transposed
    T x[3], y[3];
    auto put = [&](int f, const T (&tx)[3], const T (&ty)[3]) {
        derivT(tx, x);
        interpT(ty, y);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            sh.ex.out.x[f][R][i][le] = x[i];
            sh.ex.out.y[f][R][i][le] = y[i];
        }
    };
    T w[3];
    [[maybe_unused]] const T rowWeight = (mid ? T(kW(1)) : T(kW(0))) * weight;
#pragma unroll
    for (int i = 0; i < 3; ++i)
        w[i] = GEO == QUAD ? (in ? wj[(3 * R + i) * N + e] : T(0)) : T(kW(i)) * rowWeight;
#pragma unroll
    for (int f = 0; f < 3; ++f)
#pragma unroll
        for (int i = 0; i < 3; ++i)
            g[f][i] *= w[i];
#pragma unroll
    for (int f = 0; f < 2; ++f) {
        T p[3], q[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            p[i] = fmaT(k0[i], g[f][i], k2[i] * g[f + 1][i]);
            q[i] = fmaT(k1[i], g[f][i], k3[i] * g[f + 1][i]);
        }
        put(f, p, q);
    }
}

// One sub-step of the stress, the damage and the divergence.  Three threads
// per element in three warps, as the mEVP kernel (nsdg_sumfact.cuh): node
// column R, Gauss row R, node column R.
//
// In FP32 bound by memory (900 bytes per element): 256 x 256 parallelograms 12.3
// us per launch in a row of them, the launch included (45.2 us with the state as
// FP64 coefficients, its conversions and 168 registers), quadrilaterals 16.4.  One
// thread per element, as the mEVP kernel takes on large grids, was slower here on
// 128 x 128 (twice the time) and no faster on 256 x 256.
template <Geometry GEO, int DG, int E>
__global__ void __launch_bounds__(3 * E) kBbmStress32(DevMesh m, StressGeometry<float> geo,
    const float* __restrict__ wdam, const float* __restrict__ wj, const float* __restrict__ u,
    const float* __restrict__ v, BbmPoints<float> pt, float* __restrict__ contrib, BbmScalars<float> k,
    int* __restrict__ err)
{
    using T = float;
    __shared__ BbmShared<T, E> sh;
    const int le = threadIdx.x % E, R = threadIdx.x / E;
    const size_t N = m.N, e = blockIdx.x * size_t(E) + le;
    const bool in = e < N, ice = in && m.ice[e];
    T ke[4] = { T(0), T(0), T(0), T(0) }, weight = T(0), c[3][6], g[3][3], d[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const size_t q = 3 * R + i;
#pragma unroll
        for (int j = 0; j < 6; ++j)
            c[i][j] = in ? pt.c[(9 * j + q) * N + e] : T(1);
#pragma unroll
        for (int f = 0; f < 3; ++f)
            g[f][i] = in ? beforeWait(pt.s + (9 * f + q) * N + e) : T(0);
        d[i] = in ? beforeWait(pt.d + q * N + e) : T(1);
    }
    if (in) {
        if constexpr (GEO == AFFINE) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                ke[j] = geo.k[j * N + e];
            weight = wj[e];
        }
    }
    waitForPrevious();
    {
        T n[2][3] = { { T(0), T(0), T(0) }, { T(0), T(0), T(0) } };
        if (ice) {
            const unsigned s2 = 2u * static_cast<unsigned>(m.nx) + 1u;
            const unsigned ix = static_cast<unsigned>(e) % static_cast<unsigned>(m.nx);
            const unsigned iy = static_cast<unsigned>(e) / static_cast<unsigned>(m.nx);
            const size_t base = 2 * size_t(s2) * iy + 2 * ix + R;
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                n[0][r] = afterWait(u + base + size_t(r) * s2);
                n[1][r] = afterWait(v + base + size_t(r) * s2);
            }
        }
#pragma unroll
        for (int f = 0; f < 2; ++f) {
            T vr[3], dr[3];
            interpDeriv(n[f], vr, dr);
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                sh.ex.in.v[f][r][R][le] = vr[r];
                sh.ex.in.dv[f][r][R][le] = dr[r];
            }
        }
    }
    __syncthreads();
    bbmRow<GEO, DG, E>(R, e, N, in, geo, wdam, wj, pt, ke, weight, c, g, d, k, sh, le);
    bool finite = true; // g holds the weighted stress
#pragma unroll
    for (int f = 0; f < 3; ++f)
#pragma unroll
        for (int i = 0; i < 3; ++i)
            finite = finite && finiteT(g[f][i]);
    if (in && !finite)
        atomicOr(err, DEV_ERR_NONFINITE_STRESS);
    __syncthreads();
    if (!ice)
        return;
#pragma unroll
    for (int f = 0; f < 2; ++f) {
        T x[3], y[3], o[3];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            x[r] = sh.ex.out.x[f][r][R][le];
            y[r] = sh.ex.out.y[f][r][R][le];
        }
        columnT(x, y, o);
#pragma unroll
        for (int r = 0; r < 3; ++r)
            contrib[(9 * f + 3 * r + R) * N + e] = o[r];
    }
}

// The same in FP64, its linear maps in fixed point as the mEVP kernel's
// (nsdg_stress_fixed.cuh): the strain's scale comes from the velocities, the
// divergence's from the new weighted stress, F its largest (exchanged by a
// barrier of its own); the maps stay within 16 (1 + rho) F on rectangles and 9 F
// elsewhere.  The brittle update and the projections of the state stay in FP64.
// Bound by FP64 issue (about 600 instructions per element, most in the update's
// divisions and roots; 900 with the maps in FP64, 3000 on coefficients): 96 x 80
// rectangles 20.2 us per launch, the launch included (without it 21.8 with the
// maps in FP64 and 121.8 on coefficients); update of 100 sub-steps, 192 x 192
// rectangles 7.5 ms, quadrilaterals 8.6 (10.2 and 10.8 with the maps in FP64).  On
// quadrilaterals four blocks per SM, 168 registers: left alone the compiler takes
// 254 and two blocks (9.8 ms).
template <Geometry GEO, int E> struct BbmFixedShared {
    Exchange<fx::i64, E> ex;
    fx::i64 strain[3][3][E];
    double sum[3][9][E];
    int top[2][3][E];
    int scale[GEO == RECT ? 1 : 3][3][E];
};
template <Geometry GEO, int DG, int E>
__global__ void __launch_bounds__(3 * E, GEO == QUAD ? 4 : 1) kBbmStress64(DevMesh m, FixedGeometry geo,
    const double* __restrict__ proj, const double* __restrict__ wdam, const double* __restrict__ wj, const double* __restrict__ u,
    const double* __restrict__ v, BbmPoints<double> pt, double* __restrict__ contrib, BbmScalars<double> k,
    int* __restrict__ err)
{
    using fx::i64;
    __shared__ BbmFixedShared<GEO, E> sh;
    const int le = threadIdx.x % E, R = threadIdx.x / E;
    const size_t N = m.N, e = blockIdx.x * size_t(E) + le;
    const bool in = e < N, ice = in && m.ice[e];
    double c[3][6], g[3][3], d[3], w[3], nq[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const size_t q = 3 * R + i;
#pragma unroll
        for (int j = 0; j < 6; ++j)
            c[i][j] = in ? pt.c[(9 * j + q) * N + e] : 1.0;
#pragma unroll
        for (int f = 0; f < 3; ++f)
            g[f][i] = in ? beforeWait(pt.s + (9 * f + q) * N + e) : 0.0;
        d[i] = in ? beforeWait(pt.d + q * N + e) : 1.0;
        if constexpr (GEO == RECT) {
            w[i] = in ? kW(i) * wj[e] : 0.0; // the row's weight below
            nq[i] = 0.0;
        } else {
            nq[i] = in ? proj[q * N + e] : 0.0;
        }
    }
    waitForPrevious(false);
    double n[2][3] = { { 0.0, 0.0, 0.0 }, { 0.0, 0.0, 0.0 } };
    if (ice) {
        const unsigned s2 = 2u * static_cast<unsigned>(m.nx) + 1u;
        const unsigned ix = static_cast<unsigned>(e) % static_cast<unsigned>(m.nx);
        const unsigned iy = static_cast<unsigned>(e) / static_cast<unsigned>(m.nx);
        const size_t base = 2 * size_t(s2) * iy + 2 * ix + R;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            n[0][r] = afterWait(u + base + size_t(r) * s2);
            n[1][r] = afterWait(v + base + size_t(r) * s2);
        }
    }
    int word = 0;
#pragma unroll
    for (int f = 0; f < 2; ++f)
#pragma unroll
        for (int r = 0; r < 3; ++r)
            word = max(word, fx::magnitudeWord(n[f][r]));
    sh.top[0][R][le] = topOf(word);
    __syncthreads();
    const int top = topOfRows<E>(sh.top[0], le);
    const bool bad = top > kTopMost; // not finite
    FixedMap<GEO> map = rowMap<GEO>(geo, R, e, N, in);
    fixedColumn<E>(n, fx::fixedShift(kVelocityBits, top), R, le, sh.ex);
    __syncthreads();
    i64 F11[3], F12[3], F22[3];
    {
        i64 a[3], b[3], s[3];
        const int scale = fixedStrain<GEO, E>(R, le, map, sh.ex, sh.strain, sh.scale[0], a, b, s);
        const int at = fx::doubleExponent(kVelocityBits - top + 1022 - scale);
        const double none = __longlong_as_double(0x7ff8000000000000ll);
#pragma unroll
        for (int i = 0; i < 3; ++i)
            bbmPoint(bad ? none : fx::toDouble(a[i], at), bad ? none : fx::toDouble(b[i], at),
                bad ? none : fx::toDouble(s[i], at), c[i], k, g[0][i], g[1][i], g[2][i], d[i]);
    }
    bbmProject<double, GEO, DG, E>(R, e, N, in, wdam, nq, pt, g, d, sh.sum, le);
    word = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        if constexpr (GEO == RECT)
            w[i] *= R == 1 ? kW(1) : kW(0);
        else
            w[i] = in ? wj[size_t(3 * R + i) * N + e] : 0.0;
#pragma unroll
        for (int f = 0; f < 3; ++f) {
            g[f][i] *= w[i];
            word = max(word, fx::magnitudeWord(g[f][i]));
        }
    }
    if (in && word >= 0x7ff00000)
        atomicOr(err, DEV_ERR_NONFINITE_STRESS);
    sh.top[1][R][le] = topOf(word);
    __syncthreads();
    const int topG = topOfRows<E>(sh.top[1], le);
    const int atG = fx::fixedShift(kStressBits<GEO>, topG);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        F11[i] = fx::toFixed(g[0][i], atG);
        F12[i] = fx::toFixed(g[1][i], atG);
        F22[i] = fx::toFixed(g[2][i], atG);
    }
    if constexpr (GEO == QUAD) // read again: kept through the brittle update it would cost registers and a block per SM
        map = rowMap<GEO>(geo, R, e, N, in);
    fixedShares<GEO, E>(R, le, map, F11, F12, F22, sh.ex, sh.scale + (GEO == RECT ? 0 : 1));
    __syncthreads();
    if (!ice)
        return;
#pragma unroll
    for (int f = 0; f < 2; ++f) {
        i64 o[3];
        const int scale = fixedColumnShares<GEO, E>(f, R, le, sh.ex, sh.scale + (GEO == RECT ? 0 : 1), o);
        const int at = fx::doubleExponent(kStressBits<GEO> - topG + 1022 - scale);
#pragma unroll
        for (int r = 0; r < 3; ++r)
            contrib[(9 * f + 3 * r + R) * N + e]
                = topG > kTopMost ? __longlong_as_double(0x7ff8000000000000ll) : fx::toDouble(o[r], at);
    }
}

// Step constants of the nodes, over dt / (rho H) (BrittleCGDynamicsKernel.hpp:206-254)
// with c = dt / (rho H):
//   a = c A F_ocean, kx = c (A F_atm |wind| uwind - rho H g dxSSH), ky likewise,
//   im = c / lumped mass, and the ocean velocity turned by the ocean angle.
template <typename T, bool CONST>
__global__ void __launch_bounds__(128) kBbmPrepNodes(int nx, int ny, size_t N, NodeInputs in, BbmNodeState st,
    BbmNodeConst<T> c, BbmParams p)
{
    const CellNodes cell(blockIdx.x * 128 + threadIdx.x, nx, ny);
    if (!cell.exists[0])
        return;
    double A[4], H[4], gx[4], gy[4];
    nodeFields<CONST>(cell, nx, ny, N, in, A, H, gx, gy);
#pragma unroll
    for (int n = 0; n < 4; ++n) {
        if (!cell.exists[n])
            continue;
        const size_t i = cell.id[n];
        st.avgU[i] = 0.0;
        st.avgV[i] = 0.0;
        const double cm = p.dt * recip64(p.rho_ice * H[n]);
        const double ua = in.ua[i], va = in.va[i], uo = in.uo[i], vo = in.vo[i];
        const double ca = cm * A[n], drag = ca * (p.F_atm * rootOf(fma(ua, ua, va * va)));
        const double im = in.invm2[i] * cm;
        c.a[i] = store<T>(ca * p.F_ocean);
        c.kx[i] = store<T>(fma(drag, ua, -p.dt * p.gravity * gx[n]));
        c.ky[i] = store<T>(fma(drag, va, -p.dt * p.gravity * gy[n]));
        const T hi = store<T>(im);
        c.im[i] = hi;
        if constexpr (sizeof(T) == 4)
            c.imLo[i] = store<T>(im - load(hi));
        c.uo[i] = store<T>(uo);
        c.vo[i] = store<T>(vo);
        c.uor[i] = store<T>(fma(uo, p.cosA, -vo * p.sinA));
        c.vor[i] = store<T>(fma(vo, p.cosA, uo * p.sinA));
        if constexpr (sizeof(T) == 4) {
            c.u[i] = store<T>(in.u[i]);
            c.v[i] = store<T>(in.v[i]);
        }
    }
}

template <typename T> struct BbmNodeScalars {
    T cosA, sinA, fcdt;
    double invNSteps;
};

// The node update of one sub-step: with G = c F,
//   u_new = (al (u + Gx) + be (v + Gy)) / (al^2 + be^2),
//   v_new = (al (v + Gy) + be (Gx - u)) / (al^2 + be^2)
// as increments, so that roundings of the factors act on the increment.  Per
// launch in a row of them, the launch included: 193 x 161 nodes, FP64, 6.2 us
// (without it 5.0, and 12.4 with hypot, a division and the step's terms formed again
// in every sub-step); 513 x 513 nodes, mixed, 7.0 us (without it 4.7, and 11.4 on
// FP64 arrays).
template <typename T>
__global__ void __launch_bounds__(128) kBbmMomentum(DevMesh m, BbmNodeConst<T> c, double* __restrict__ avgU,
    double* __restrict__ avgV, const T* __restrict__ contrib, BbmNodeScalars<T> k, int* __restrict__ err)
{
    const size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
    if (i >= m.Ncg)
        return;
    const unsigned s2 = 2u * static_cast<unsigned>(m.nx) + 1u;
    const int i2 = static_cast<int>(static_cast<unsigned>(i) % s2), j2 = static_cast<int>(static_cast<unsigned>(i) / s2);
    const bool dir = m.cg2Dir[i] != 0;
    // before the wait for the stress kernel: the step's constants, and what
    // the node kernel before that one wrote
    const T a = c.a[i], kx = c.kx[i], ky = c.ky[i], im = c.im[i];
    const T uo = c.uo[i], vo = c.vo[i], uor = c.uor[i], vor = c.vor[i];
    const T u = beforeWait(c.u + i), v = beforeWait(c.v + i);
    const T imLo = sizeof(T) == 4 ? c.imLo[i] : T(0);
    const double au = beforeWait(avgU + i), av = beforeWait(avgV + i);
    waitForPrevious(sizeof(T) == 4);
    T dSx = T(0), dSy = T(0);
    if (!dir)
        gatherDivergence(m, i2, j2, contrib, dSx, dSy);
    const T ur = uo - u, vr = vo - v;
    const T cp = a * sqrtT(fmaT(ur, ur, vr * vr));
    const T cpc = cp * k.cosA, al = T(1) + cpc, be = fmaT(cp, k.sinA, k.fcdt);
    const T rd = recipT(fmaT(al, al, be * be));
    T gx = fmaT(dSx, im, kx), gy = fmaT(dSy, im, ky);
    if constexpr (sizeof(T) == 4) {
        gx = fmaT(dSx, imLo, gx);
        gy = fmaT(dSy, imLo, gy);
    }
    gx = fmaT(cp, uor, gx);
    gy = fmaT(cp, vor, gy);
    T un = fmaT(rd, fmaT(al, fmaT(-cpc, u, gx), be * fmaT(-be, u, v + gy)), u);
    T vn = fmaT(rd, fmaT(al, fmaT(-cpc, v, gy), be * fmaT(-be, v, gx - u)), v);
    if (!finiteT(un) || !finiteT(vn))
        atomicOr(err, DEV_ERR_NONFINITE_VELOCITY);
    if constexpr (sizeof(T) == 8) {
        avgU[i] = fma(un, k.invNSteps, au);
        avgV[i] = fma(vn, k.invNSteps, av);
    } else {
        avgU[i] = fma(static_cast<double>(un), k.invNSteps, au);
        avgV[i] = fma(static_cast<double>(vn), k.invNSteps, av);
    }
    if (dir)
        un = vn = T(0);
    c.u[i] = un;
    c.v[i] = vn;
}

template <int DG>
cudaError_t stressFor(cudaStream_t s, const DevMesh& m, const BbmElements<float>& el, const float* u, const float* v,
    float* contrib, const BbmScalars<float>& k, int* err, bool programmatic)
{
    constexpr int E = kBbmElems;
    auto kernel = el.parallelogram ? kBbmStress32<AFFINE, DG, E> : kBbmStress32<QUAD, DG, E>;
    return launchAfter(programmatic, s, kernel, (m.N + E - 1) / E, 3 * E, 0, m, el.geo, el.wdam, el.w, u, v, el.pt,
        contrib, k, err);
}
template <int DG>
cudaError_t stressFor(cudaStream_t s, const DevMesh& m, const BbmElements<double>& el, const double* u,
    const double* v, double* contrib, const BbmScalars<double>& k, int* err,
    bool programmatic)
{
    constexpr int E = kBbmElems;
    auto kernel = el.fixed.rect ? kBbmStress64<RECT, DG, E> : kBbmStress64<QUAD, DG, E>;
    return launchAfter(programmatic, s, kernel, (m.N + E - 1) / E, 3 * E, 0, m, el.fixed, el.geo.n, el.wdam, el.w, u,
        v, el.pt, contrib, k, err);
}

} // namespace

template <typename T>
cudaError_t launchBbmLoad(cudaStream_t s, const DevMesh& m, int dg, const BbmElements<T>& el, const double* h,
    const double* a, const double* damage, const double* s11, const double* s12, const double* s22,
    const double* hsize, double* lagH, double* lagA, const BbmParams& p)
{
    const unsigned g = static_cast<unsigned>((m.N + 127) / 128);
    const double* invKx2 = nullptr;
    if constexpr (sizeof(T) == 8)
        invKx2 = el.geo.rect ? el.geo.k + m.N : nullptr;
    switch (dg) {
    case 1: kBbmLoad<T, 1><<<g, 128, 0, s>>>(m.N, h, a, damage, s11, s12, s22, hsize, invKx2, el.pt, lagH, lagA, p); break;
    case 3: kBbmLoad<T, 3><<<g, 128, 0, s>>>(m.N, h, a, damage, s11, s12, s22, hsize, invKx2, el.pt, lagH, lagA, p); break;
    case 6: kBbmLoad<T, 6><<<g, 128, 0, s>>>(m.N, h, a, damage, s11, s12, s22, hsize, invKx2, el.pt, lagH, lagA, p); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

template <typename T>
cudaError_t launchBbmStore(cudaStream_t s, const DevMesh& m, int dg, const BbmElements<T>& el, double* damage,
    double* s11, double* s12, double* s22)
{
    const unsigned g = static_cast<unsigned>((m.N + 127) / 128);
    switch (dg) {
    case 1: kBbmStore<T, 1><<<g, 128, 0, s>>>(m.N, el.pt, damage, s11, s12, s22); break;
    case 3: kBbmStore<T, 3><<<g, 128, 0, s>>>(m.N, el.pt, damage, s11, s12, s22); break;
    case 6: kBbmStore<T, 6><<<g, 128, 0, s>>>(m.N, el.pt, damage, s11, s12, s22); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

template <typename T>
cudaError_t launchBbmPrepNodes(cudaStream_t s, const DevMesh& m, const NodeInputs& in, const BbmNodeState& st,
    const BbmNodeConst<T>& c, const BbmParams& p)
{
    const unsigned g = static_cast<unsigned>((cellsAndBorder(m.nx, m.ny) + 127) / 128);
    if (in.constant)
        kBbmPrepNodes<T, true><<<g, 128, 0, s>>>(m.nx, m.ny, m.N, in, st, c, p);
    else
        kBbmPrepNodes<T, false><<<g, 128, 0, s>>>(m.nx, m.ny, m.N, in, st, c, p);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launchBbmStress(cudaStream_t s, const DevMesh& m, int dg, const BbmElements<T>& el, const T* u,
    const T* v, T* contrib, const BbmParams& p, int* err, bool programmatic)
{
    const BbmScalars<T> k { static_cast<T>(p.dt), static_cast<T>(p.nu0), static_cast<T>(0.5 * (1. - p.nu0)),
        static_cast<T>(p.tan_phi), static_cast<T>(p.exponent_relaxation_sigma - 1.), p.powRmode, p.powRk };
    switch (dg) {
    case 1: return stressFor<1>(s, m, el, u, v, contrib, k, err, programmatic);
    case 3: return stressFor<3>(s, m, el, u, v, contrib, k, err, programmatic);
    case 6: return stressFor<6>(s, m, el, u, v, contrib, k, err, programmatic);
    default: return cudaErrorInvalidValue;
    }
}

template <typename T>
cudaError_t launchBbmMomentum(cudaStream_t s, const DevMesh& m, const BbmNodeState& st, const BbmNodeConst<T>& c,
    const T* contrib, const BbmParams& p, int* err, bool programmatic)
{
    const BbmNodeScalars<T> k { static_cast<T>(p.cosA), static_cast<T>(p.sinA), static_cast<T>(p.dt * p.fc),
        p.invNSteps };
    return launchAfter(programmatic, s, kBbmMomentum<T>, (m.Ncg + 127) / 128, 128, 0, m, c, st.avgU, st.avgV, contrib,
        k, err);
}

#define NSDG_BBM_INSTANCES(T)                                                                                       \
    template cudaError_t launchBbmLoad<T>(cudaStream_t, const DevMesh&, int, const BbmElements<T>&, const double*,  \
        const double*, const double*, const double*, const double*, const double*, const double*, double*, double*,  \
        const BbmParams&);                                                                                          \
    template cudaError_t launchBbmStore<T>(cudaStream_t, const DevMesh&, int, const BbmElements<T>&, double*,       \
        double*, double*, double*);                                                                                 \
    template cudaError_t launchBbmPrepNodes<T>(cudaStream_t, const DevMesh&, const NodeInputs&,                     \
        const BbmNodeState&, const BbmNodeConst<T>&, const BbmParams&);                                             \
    template cudaError_t launchBbmStress<T>(cudaStream_t, const DevMesh&, int, const BbmElements<T>&, const T*,     \
        const T*, T*, const BbmParams&, int*, bool);                                                                \
    template cudaError_t launchBbmMomentum<T>(cudaStream_t, const DevMesh&, const BbmNodeState&,                    \
        const BbmNodeConst<T>&, const T*, const BbmParams&, int*, bool);
NSDG_BBM_INSTANCES(double)
NSDG_BBM_INSTANCES(float)

} // namespace nsdg
