// nsdg_stress_sumfact.cu — the FP64 mEVP element kernel (nsdg_sumfact.cuh).
#include "nsdg_sumfact.cuh"

namespace nsdg {
namespace {

using namespace sf;

// One mEVP iteration in divergence space, FP64: tdiv <- (1 - 1/alpha) tdiv +
// K^T P^T f(P K u).  Three threads per element, in three warps of a block of
// kElems elements: warp R takes node column R (the eta maps of its three
// nodes), then Gauss row R (the xi maps, strain, stress increments, the
// transposed xi maps), then node column R again (the transposed eta maps); the
// 24 and 36 values in between go through shared memory, as do the sums of the
// two projections on general quadrilaterals.
//
// On rectangles the strain is carried over k_x (strain' = strain / k_x, the
// eta derivatives times rho = k_y / k_x, DeltaMin^2 over k_x^2) and k_x is
// part of the pressure's weight, so only rho is multiplied in.
//
// Bound by FP64 issue: about 480 FP64 instructions per element on rectangles,
// 720 on quadrilaterals and 800 on a sphere; at the rate cuBLAS DGEMM reaches
// (0.55 T FMA/s) 57 us for 256 x 256 rectangles.  Timed alone (CUDA events):
// 60.8 us for 256 x 256 rectangles (112 us with 9 x 9 operators streamed from
// memory), 42 us for 201 x 143 quadrilaterals (49 us), 32 us for 154 x 121
// cells of a sphere (44 us), 7.4 us for 64 x 64 rectangles (20.5 us).  Three
// threads per element rather than one: the same time on large grids, but on
// 64 x 64 one warp per SM waits out every instruction's latency (17.1 us).
constexpr int kElems = 32;

struct Exchange {
    union {
        struct {
            double v[2][3][3][kElems];  // [u, v][Gauss row][column]: values on the columns
            double dv[2][3][3][kElems]; // eta derivatives
        } in;
        struct {
            double x[2][3][3][kElems]; // to the transposed interpolation
            double y[2][3][3][kElems]; // to the transposed derivative
        } out;
    };
};

// The block's three warps meet here from different instances of the row code:
// a barrier by its number (PTX bar.sync counts warps, whatever their place in
// the code).
__device__ __forceinline__ void rowsBarrier() { asm volatile("bar.sync 1, %0;" ::"n"(3 * kElems) : "memory"); }

// sum over the element's three warps of each thread's c[0..2]
__device__ __forceinline__ void sumRows(double (*part)[3][kElems], int R, int le, double (&c)[3])
{
#pragma unroll
    for (int k = 0; k < 3; ++k)
        part[R][k][le] = c[k];
    rowsBarrier();
#pragma unroll
    for (int k = 0; k < 3; ++k)
        c[k] = part[0][k][le] + part[1][k][le] + part[2][k][le];
}

template <int R, Geometry GEO>
__device__ __forceinline__ void row64(bool active, size_t e, size_t N, const StressGeometry& geo,
    const double (&pq)[3], double rho, double dminQ, Exchange& ex, double (*sums)[3][3][kElems], int le)
{
    double I[3], D[3], uxi[3], uet[3], vxi[3], vet[3], f11[3], f12[3], f22[3], x[3], y[3];
    [[maybe_unused]] double up[3], vp[3];
    const Scaled<double> sc(GEO == RECT ? rho : 1.0);
    auto take = [&](int c) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            I[i] = ex.in.v[c][R][i][le];
            D[i] = ex.in.dv[c][R][i][le];
        }
    };
    take(0);
    deriv(I, uxi);
    if constexpr (GEO == RECT)
        sc.interp(D, uet);
    else
        interp(D, uet);
    if constexpr (GEO == SPHERE)
        interp(I, up);
    take(1);
    deriv(I, vxi);
    if constexpr (GEO == RECT)
        sc.interp(D, vet);
    else
        interp(D, vet);
    if constexpr (GEO == SPHERE)
        interp(I, vp);
    if constexpr (GEO == RECT) {
#pragma unroll
        for (int i = 0; i < 3; ++i)
            pointStress64(uxi[i], vet[i], uet[i] + vxi[i], pq[i], dminQ, f11[i], f12[i], f22[i]);
        rowsBarrier(); // every warp has taken its row: the buffer changes hands
        auto put = [&](int c, const double (&fx)[3], const double (&fy)[3]) {
            derivT(fx, x);
            sc.interpT(fy, y);
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                ex.out.x[c][R][i][le] = x[i];
                ex.out.y[c][R][i][le] = y[i];
            }
        };
        put(0, f11, f12);
        put(1, f12, f22);
    } else {
        double k0[3], k1[3], k2[3], k3[3], nq[3], a[3], b[3], s[3];
        [[maybe_unused]] double mq[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const size_t q = 3 * R + i;
            k0[i] = active ? geo.k[q * N + e] : 0.0;
            k1[i] = active ? geo.k[(9 + q) * N + e] : 0.0;
            k2[i] = active ? geo.k[(18 + q) * N + e] : 0.0;
            k3[i] = active ? geo.k[(27 + q) * N + e] : 0.0;
            nq[i] = active ? geo.n[q * N + e] : 0.0;
            a[i] = fma(k0[i], uxi[i], k1[i] * uet[i]);
            b[i] = fma(k2[i], vxi[i], k3[i] * vet[i]);
            s[i] = fma(k2[i], uxi[i], fma(k3[i], uet[i], fma(k0[i], vxi[i], k1[i] * vet[i])));
            if constexpr (GEO == SPHERE) {
                mq[i] = active ? geo.m[q * N + e] : 0.0;
                a[i] = fma(-mq[i], vp[i], a[i]);
                s[i] = fma(mq[i], up[i], s[i]);
            }
        }
        constexpr double nr = R == 1 ? -2.0 : 1.0; // nu on this row: nr, -2 nr, nr
        // P: subtract n (nu . g)
        double c[3] = { nr * fma(-2.0, a[1], a[0] + a[2]), nr * fma(-2.0, b[1], b[0] + b[2]),
            nr * fma(-2.0, s[1], s[0] + s[2]) };
        sumRows(sums[0], R, le, c);
        double d[3] = { 0.0, 0.0, 0.0 };
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            pointStress64(fma(-c[0], nq[i], a[i]), fma(-c[1], nq[i], b[i]), fma(-c[2], nq[i], s[i]), pq[i], dminQ,
                f11[i], f12[i], f22[i]);
            d[0] = fma(nq[i], f11[i], d[0]);
            d[1] = fma(nq[i], f22[i], d[1]);
            d[2] = fma(nq[i], f12[i], d[2]);
        }
        // P^T: subtract nu (n . f)
        sumRows(sums[1], R, le, d);
        double t0[3], t1[3], t2[3], t3[3];
        [[maybe_unused]] double mu[3], mv[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const double w = i == 1 ? -2.0 * nr : nr;
            f11[i] = fma(-w, d[0], f11[i]);
            f22[i] = fma(-w, d[1], f22[i]);
            f12[i] = fma(-w, d[2], f12[i]);
            t0[i] = fma(k0[i], f11[i], k2[i] * f12[i]);
            t1[i] = fma(k1[i], f11[i], k3[i] * f12[i]);
            t2[i] = fma(k0[i], f12[i], k2[i] * f22[i]);
            t3[i] = fma(k1[i], f12[i], k3[i] * f22[i]);
            if constexpr (GEO == SPHERE) {
                mu[i] = mq[i] * f12[i];
                mv[i] = -mq[i] * f11[i];
            }
        }
        auto put = [&](int c, const double (&tx)[3], const double (&ty)[3], [[maybe_unused]] const double (&tm)[3]) {
            derivT(tx, x);
            interpT(ty, y);
            if constexpr (GEO == SPHERE) {
                double z[3];
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

template <Geometry GEO>
__global__ void __launch_bounds__(3 * kElems) kMevpStress(DevMesh m, StressGeometry geo, const double* __restrict__ u,
    const double* __restrict__ v, const double* __restrict__ Pw, double* __restrict__ tdiv, double dminQ, double keep)
{
    __shared__ Exchange ex;
    __shared__ double sums[GEO == RECT ? 1 : 2][3][3][kElems];
    const int le = threadIdx.x % kElems, R = threadIdx.x / kElems;
    const size_t N = m.N, e = blockIdx.x * size_t(kElems) + le;
    const bool active = e < N && m.ice[e];
    // everything the previous two launches do not write comes before the wait
    // (the divergence was written two launches ago by this kernel and is only
    // read by the node kernel in between)
    double pq[3] = { 0.0, 0.0, 0.0 }, told[6], rho = 0.0;
    if (active) {
#pragma unroll
        for (int i = 0; i < 3; ++i)
            pq[i] = Pw[(3 * R + i) * N + e];
        if constexpr (GEO == RECT) {
            rho = geo.k[e];
            dminQ *= geo.k[N + e];
        }
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            told[r] = tdiv[(3 * r + R) * N + e];
            told[3 + r] = tdiv[(9 + 3 * r + R) * N + e];
        }
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    {
        double n[2][3] = { { 0.0, 0.0, 0.0 }, { 0.0, 0.0, 0.0 } };
        if (active) {
            const unsigned s2 = 2u * static_cast<unsigned>(m.nx) + 1u;
            const unsigned ix = static_cast<unsigned>(e) % static_cast<unsigned>(m.nx);
            const unsigned iy = static_cast<unsigned>(e) / static_cast<unsigned>(m.nx);
            const size_t base = 2 * size_t(s2) * iy + 2 * ix + R;
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                n[0][r] = u[base + size_t(r) * s2];
                n[1][r] = v[base + size_t(r) * s2];
            }
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            double vr[3], dr[3];
            interpDeriv(n[c], vr, dr);
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                ex.in.v[c][r][R][le] = vr[r];
                ex.in.dv[c][r][R][le] = dr[r];
            }
        }
    }
    __syncthreads();
    switch (R) {
    case 0: row64<0, GEO>(active, e, N, geo, pq, rho, dminQ, ex, sums, le); break;
    case 1: row64<1, GEO>(active, e, N, geo, pq, rho, dminQ, ex, sums, le); break;
    default: row64<2, GEO>(active, e, N, geo, pq, rho, dminQ, ex, sums, le); break;
    }
    __syncthreads();
    if (!active)
        return;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        double x[3], y[3], o[3];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            x[r] = ex.out.x[c][r][R][le];
            y[r] = ex.out.y[c][r][R][le];
        }
        columnT(x, y, o);
#pragma unroll
        for (int r = 0; r < 3; ++r)
            tdiv[(9 * c + 3 * r + R) * N + e] = fma(told[3 * c + r], keep, o[r]);
    }
}

} // namespace

cudaError_t launchMevpStress(cudaStream_t s, const DevMesh& m, const StressGeometry& geo, const double* u,
    const double* v, const double* Pw, double* tdiv, const MevpParams& pIn)
{
    const MevpParams p = withDerived(pIn);
    const double dminQ = 0.25 * (p.DeltaMin * p.DeltaMin);
    cudaLaunchConfig_t cfg {};
    cfg.gridDim = dim3(static_cast<unsigned>((m.N + kElems - 1) / kElems));
    cfg.blockDim = dim3(3 * kElems);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (geo.rect)
        return cudaLaunchKernelEx(&cfg, kMevpStress<RECT>, m, geo, u, v, Pw, tdiv, dminQ, p.keepd);
    if (geo.m)
        return cudaLaunchKernelEx(&cfg, kMevpStress<SPHERE>, m, geo, u, v, Pw, tdiv, dminQ, p.keepd);
    return cudaLaunchKernelEx(&cfg, kMevpStress<QUAD>, m, geo, u, v, Pw, tdiv, dminQ, p.keepd);
}

} // namespace nsdg
