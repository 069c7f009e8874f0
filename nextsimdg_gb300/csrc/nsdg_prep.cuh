// nsdg_prep.cuh — the node values a step's preparation takes from the cells.
#pragma once

#include "nsdg_modes.cuh"
#include "nsdg_nodes.cuh"

namespace nsdg {
namespace {

// The DG2CG averages at a cell's four nodes (Interpolations.cpp:144-204): the
// mean over the cells around a node of their Lagrange values there, odd cell
// rows first.  f: [9][N] Lagrange values, or (CONST) one value per cell.  The
// weights 1/4 and 1/2 and the doubling on the mesh's border are powers of two,
// applied to the sum.
template <bool CONST>
__device__ __forceinline__ double lagAt(const double* __restrict__ f, size_t N, bool ok, int j, size_t cell)
{
    return ok ? f[CONST ? cell : j * N + cell] : 0.0;
}
template <bool CONST>
__device__ __forceinline__ double gatherCorner(const CellNodes& c, int nx, int ny, size_t N,
    const double* __restrict__ f)
{
    const bool left = c.ix > 0, right = c.ix < nx, below = c.iy > 0, above = c.iy < ny;
    const size_t e = size_t(c.iy) * nx + c.ix;
    const double b0 = lagAt<CONST>(f, N, below && left, 8, e - nx - 1), b1 = lagAt<CONST>(f, N, below && right, 6, e - nx);
    const double a0 = lagAt<CONST>(f, N, above && left, 2, e - 1), a1 = lagAt<CONST>(f, N, above && right, 0, e);
    const bool belowFirst = (c.iy & 1) == 0; // row iy - 1 is odd
    const double s = belowFirst ? ((b0 + b1) + a0) + a1 : ((a0 + a1) + b0) + b1;
    return s * ((left && right ? 0.5 : 1.0) * (below && above ? 0.5 : 1.0));
}
template <bool CONST>
__device__ __forceinline__ void gatherMean(const CellNodes& c, int nx, int ny, size_t N,
    const double* __restrict__ f, double (&v)[4])
{
    const bool left = c.ix > 0, right = c.ix < nx, below = c.iy > 0, above = c.iy < ny;
    const size_t e = size_t(c.iy) * nx + c.ix;
    v[0] = gatherCorner<CONST>(c, nx, ny, N, f);
    const double mb = lagAt<CONST>(f, N, below && right, 7, e - nx), ma = lagAt<CONST>(f, N, above && right, 1, e);
    v[1] = (mb + ma) * (below && above ? 0.5 : 1.0);
    const double l0 = lagAt<CONST>(f, N, above && left, 5, e - 1), l1 = lagAt<CONST>(f, N, above && right, 3, e);
    v[2] = (l0 + l1) * (left && right ? 0.5 : 1.0);
    v[3] = lagAt<CONST>(f, N, above && right, 4, e);
}

// prepareIteration's node fields (CGDynamicsKernel.cpp:205-276): A and H
// clamped, and the sea-surface-height gradient, interpolated from its CG1
// values (a border node takes the neighbouring interior node's).
template <bool CONST>
__device__ __forceinline__ void nodeFields(const CellNodes& c, int nx, int ny, size_t N, const NodeInputs& in,
    double (&A)[4], double (&H)[4], double (&gx)[4], double (&gy)[4])
{
    gatherMean<CONST>(c, nx, ny, N, in.a, A);
    gatherMean<CONST>(c, nx, ny, N, in.h, H);
#pragma unroll
    for (int n = 0; n < 4; ++n) {
        A[n] = sf::atLeast(sf::isNan64(A[n]) ? 1.0 : sf::atMost(sf::atLeast(A[n], 0.0), 1.0), 1.e-4);
        H[n] = sf::atLeast(H[n], 1.e-4);
    }
    auto src = [&](int i, int j) {
        const int si = i < 1 ? 1 : i > nx - 1 ? nx - 1 : i, sj = j < 1 ? 1 : j > ny - 1 ? ny - 1 : j;
        return size_t(sj) * (size_t(nx) + 1) + si;
    };
    const size_t p = src(c.ix, c.iy), q = src(c.ix + 1, c.iy), r = src(c.ix, c.iy + 1), s = src(c.ix + 1, c.iy + 1);
    auto four = [&](const double* __restrict__ g, double (&o)[4]) {
        const double a = g[p], b = g[q], d = g[r], e = g[s];
        o[0] = a;
        o[1] = 0.5 * (a + b);
        o[2] = 0.5 * (a + d);
        o[3] = 0.25 * (a + b + d + e);
    };
    four(in.ug, gx);
    four(in.vg, gy);
}

// the nine Lagrange values of h and A of one cell (nothing for DG 1, whose
// cells are constant)
template <int DG>
__device__ __forceinline__ void storeLagrange(const double (&hc)[DG], const double (&ac)[DG], size_t N, size_t e,
    double* __restrict__ lagH, double* __restrict__ lagA)
{
    if constexpr (DG > 1) {
        double v[9];
        sf::lagrangeValues<DG>(hc, v);
#pragma unroll
        for (int q = 0; q < 9; ++q)
            lagH[q * N + e] = v[q];
        sf::lagrangeValues<DG>(ac, v);
#pragma unroll
        for (int q = 0; q < 9; ++q)
            lagA[q * N + e] = v[q];
    }
}

} // namespace
} // namespace nsdg
