// nsdg_nodes.cuh — the cells around a CG2 node, and the gather of their
// contributions.
#pragma once

#include "nsdg_kernels.hpp"

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
    T ax = T(0), ay = T(0);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        if (r < Y.n) {
            const int cy = r ? Y.c1 : Y.c0, ly = r ? Y.l1 : Y.l0;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                if (k < X.n) {
                    const size_t c = size_t(cy) * m.nx + (k ? X.c1 : X.c0);
                    const int j = (k ? X.l1 : X.l0) + 3 * ly;
                    ax -= contrib[j * N + c];
                    ay -= contrib[(9 + j) * N + c];
                }
            }
        }
    }
    dx = ax;
    dy = ay;
}

} // namespace
} // namespace nsdg
