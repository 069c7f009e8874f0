// nsdg_nodes.cuh — the cells around a CG2 node, and the gather of their
// contributions.
#pragma once

#include "nsdg_kernels.hpp"
#include "nsdg_pdl.cuh"
#include "nsdg_visc_ff.hpp"

namespace nsdg {
namespace {

// The cells along one direction touching CG2 index i2 (0..2n) and the node's
// local index in each (0, 1, 2), ascending; kept in registers (no local
// arrays): n of them
struct NodeCand {
    int n, c0, l0, c1, l1;
};
__device__ __forceinline__ NodeCand nodeCand(int i2, int n)
{
    NodeCand r { 1, 0, 0, 0, 0 };
    if (i2 & 1) {
        r.c0 = (i2 - 1) / 2;
        r.l0 = 1;
    } else if (i2 >= 2 && i2 / 2 < n) {
        r.n = 2;
        r.c0 = i2 / 2 - 1;
        r.l0 = 2;
        r.c1 = i2 / 2;
        r.l1 = 0;
    } else if (i2 >= 2) {
        r.c0 = i2 / 2 - 1;
        r.l0 = 2;
    } else {
        r.c0 = i2 / 2;
        r.l0 = 0;
    }
    return r;
}

// Gathers the divergence contributions of the (up to four) ice cells around
// a CG2 node in the reference's scatter order (even cell rows first, then
// odd; ascending x) and returns -sum.
template <typename T>
__device__ __forceinline__ void gatherDivergence(const DevMesh& m, int i2, int j2, const T* __restrict__ contrib,
    T& dx, T& dy)
{
    const NodeCand X = nodeCand(i2, m.nx);
    NodeCand Y = nodeCand(j2, m.ny);
    if (Y.n == 2 && (Y.c0 & 1)) { // even cell rows first
        const int c = Y.c0, l = Y.l0;
        Y.c0 = Y.c1;
        Y.l0 = Y.l1;
        Y.c1 = c;
        Y.l1 = l;
    }
    const size_t N = m.N;
    auto at = [&](int cy, int cx, int j) { return contrib + size_t(j) * N + size_t(cy) * m.nx + cx; };
    // all loads first, a missing cell's from the first one's place
    const bool x2 = X.n == 2, y2 = Y.n == 2;
    const T* p[4] = { at(Y.c0, X.c0, X.l0 + 3 * Y.l0), at(Y.c0, X.c1, X.l1 + 3 * Y.l0),
        at(Y.c1, X.c0, X.l0 + 3 * Y.l1), at(Y.c1, X.c1, X.l1 + 3 * Y.l1) };
    p[1] = x2 ? p[1] : p[0];
    p[2] = y2 ? p[2] : p[0];
    p[3] = x2 && y2 ? p[3] : p[0];
    T x[4], y[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        x[k] = afterWait(p[k]);
        y[k] = afterWait(p[k] + 9 * N);
    }
    T ax = -x[0], ay = -y[0];
    if (x2) {
        ax -= x[1];
        ay -= y[1];
    }
    if (y2) {
        if (sizeof(T) == 4 && x2) { // rounded once, as a sum in FP64 (which made the update 35 % longer)
            ax = -nsdg_ff::sumOfFour(x[0], x[1], x[2], x[3]);
            ay = -nsdg_ff::sumOfFour(y[0], y[1], y[2], y[3]);
        } else {
            ax -= x[2];
            ay -= y[2];
            if (x2) {
                ax -= x[3];
                ay -= y[3];
            }
        }
    }
    dx = ax;
    dy = ay;
}

// The four CG2 nodes that cell (ix, iy) of the (nx + 1) x (ny + 1) cells and
// border cells owns: its lower left corner and, where the cell is one of the
// mesh, the middles of its lower and left sides and its centre.
struct CellNodes {
    size_t id[4];   // (2 ix, 2 iy), (2 ix + 1, 2 iy), (2 ix, 2 iy + 1), (2 ix + 1, 2 iy + 1)
    bool exists[4];
    int ix, iy;
    __device__ __forceinline__ CellNodes(unsigned t, int nx, int ny)
    {
        const unsigned w = static_cast<unsigned>(nx) + 1u;
        iy = static_cast<int>(t / w);
        ix = static_cast<int>(t % w);
        const size_t s2 = 2 * size_t(nx) + 1;
        id[0] = 2 * s2 * iy + 2 * ix;
        id[1] = id[0] + 1;
        id[2] = id[0] + s2;
        id[3] = id[2] + 1;
        exists[0] = iy <= ny;
        exists[1] = exists[0] && ix < nx;
        exists[2] = iy < ny;
        exists[3] = exists[2] && ix < nx;
    }
};

// minus the sums of the contributions of the cells around those four nodes,
// in the order of gatherDivergence (even cell rows first, ascending x).  One
// thread for four nodes: every lane of a warp does the same loads, where one
// thread per node makes the lanes of a warp wait for each other's cells.  The
// mixed mEVP node kernel takes this form (1025 x 1025 nodes 9.1 -> 6.9 us,
// 11.2 with the launch, the same results bit for bit); with the FP64 and the BBM kernels'
// larger node state it is slower (513 x 513 nodes: FP64 18.6 -> 20.5 us, BBM
// FP64 23.1 -> 27.0, BBM mixed 4.6 -> 5.5), and they keep one thread per node.
template <typename T>
__device__ __forceinline__ void gatherCell(const CellNodes& c, int nx, int ny, size_t N,
    const T* __restrict__ contrib, T (&dx)[4], T (&dy)[4])
{
    const bool left = c.ix > 0, right = c.ix < nx, below = c.iy > 0, above = c.iy < ny;
    const size_t e = size_t(c.iy) * nx + c.ix; // the cell itself
    auto at = [&](bool ok, int j, size_t cell, T& x, T& y) {
        x = ok ? afterWait(contrib + j * N + cell) : T(0);
        y = ok ? afterWait(contrib + (9 + j) * N + cell) : T(0);
    };
    // corner: local nodes 8, 6 of the row below and 2, 0 of the cell's row
    T bx[2], by[2], ax[2], ay[2], mbx, mby, max_, may, lx[2], ly[2], cx, cy;
    at(below && left, 8, e - nx - 1, bx[0], by[0]);
    at(below && right, 6, e - nx, bx[1], by[1]);
    at(above && left, 2, e - 1, ax[0], ay[0]);
    at(above && right, 0, e, ax[1], ay[1]);
    at(below && right, 7, e - nx, mbx, mby);  // middle of the lower side
    at(above && right, 1, e, max_, may);
    at(above && left, 5, e - 1, lx[0], ly[0]); // middle of the left side
    at(above && right, 3, e, lx[1], ly[1]);
    at(above && right, 4, e, cx, cy);          // centre
    const bool belowFirst = (c.iy & 1) != 0;   // row iy - 1 is even
    auto four = [&](const T (&b)[2], const T (&a)[2]) {
        const T p0 = belowFirst ? b[0] : a[0], p1 = belowFirst ? b[1] : a[1];
        const T q0 = belowFirst ? a[0] : b[0], q1 = belowFirst ? a[1] : b[1];
        return T(0) - p0 - p1 - q0 - q1;
    };
    auto two = [&](T b, T a) { return belowFirst ? T(0) - b - a : T(0) - a - b; };
    dx[0] = four(bx, ax);
    dy[0] = four(by, ay);
    dx[1] = two(mbx, max_);
    dy[1] = two(mby, may);
    dx[2] = T(0) - lx[0] - lx[1];
    dy[2] = T(0) - ly[0] - ly[1];
    dx[3] = T(0) - cx;
    dy[3] = T(0) - cy;
}

} // namespace
} // namespace nsdg
