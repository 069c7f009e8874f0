// nsdg_step.cu — what a model step prepares before its sub-cycle
// (CGDynamicsKernel.cpp:126-276): the CG2 node values of thickness and
// concentration, the sea-surface-height gradient, the pressure at the Gauss
// points and the step's node constants.
//
// These kernels are bound by FP64 issue (GB300 issues FP64 at about 1/60 of
// its FP32 rate): expansions are evaluated by 1-D factors (nsdg_modes.cuh),
// exponentials, roots and reciprocals take few instructions
// (nsdg_exp64.cuh, nsdg_seed64.cuh), clamps and conversions work on the bit
// patterns, and weights that are powers of two are applied once to a sum.
#include "nsdg_exp64.cuh"
#include "nsdg_kernels.hpp"
#include "nsdg_modes.cuh"
#include "nsdg_nodes.cuh"
#include "nsdg_prep.cuh"
#include "nsdg_seed64.cuh"
#include "nsdg_visc_ff.hpp"

namespace nsdg {
namespace {

using namespace sf;

constexpr int kBlock = 128;
inline unsigned blocksFor(size_t n) { return static_cast<unsigned>((n + kBlock - 1) / kBlock); }

// CG2 node values of one-component fields (DG2CG, Interpolations.cpp:144-204),
// four of them per launch: a module step's wind and ocean on 512 x 512 cells
// 26 us (four launches of one thread per node 116 us, bound by FP64 issue: five
// of its instructions per cell around the node).
template <int NF>
__global__ void __launch_bounds__(kBlock) kAverage(int nx, int ny, AverageFields f)
{
    const CellNodes c(blockIdx.x * kBlock + threadIdx.x, nx, ny);
    if (!c.exists[0])
        return;
#pragma unroll
    for (int k = 0; k < NF; ++k) {
        double v[4];
        gatherMean<true>(c, nx, ny, 0, f.src[k], v);
#pragma unroll
        for (int n = 0; n < 4; ++n)
            if (c.exists[n])
                f.dst[k][c.id[n]] = v[n];
    }
}

// CG1 Lagrange average of the DG0 ssh (reversed parity: odd rows first)
__global__ void __launch_bounds__(kBlock) kSSHToCG1(DevMesh m, const double* __restrict__ ssh, double* __restrict__ cg1)
{
    const CellNodes c(blockIdx.x * kBlock + threadIdx.x, m.nx, m.ny);
    if (!c.exists[0])
        return;
    cg1[size_t(c.iy) * (size_t(m.nx) + 1) + c.ix] = gatherCorner<true>(c, m.nx, m.ny, 0, ssh);
}
// CG1 gradient by element gather (even rows first), over the lumped mass
__global__ void __launch_bounds__(kBlock) kSSHGrad1(DevMesh m, DevOps o, const double* __restrict__ cg1,
    double* __restrict__ ug, double* __restrict__ vg)
{
    const size_t t = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
    if (t >= m.Ncg1)
        return;
    const unsigned s1 = static_cast<unsigned>(m.nx) + 1u;
    const int i1 = static_cast<int>(static_cast<unsigned>(t) % s1), j1 = static_cast<int>(static_cast<unsigned>(t) / s1);
    // the cell rows touching the node with the node's local row in each, even
    // rows first (registers, no local arrays)
    const bool below = j1 >= 1, above = j1 < m.ny;
    const int nr = int(below) + int(above);
    int row0 = below ? j1 - 1 : j1, ly0 = below ? 1 : 0, row1 = j1, ly1 = 0;
    if (nr == 2 && (row0 % 2) == 1) {
        row0 = j1;
        ly0 = 0;
        row1 = j1 - 1;
        ly1 = 1;
    }
    double au = 0.0, av = 0.0;
    const size_t N = m.N;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        if (r >= nr)
            continue;
        for (int lx = 1; lx >= 0; --lx) {
            const int cx = i1 - lx;
            if (cx < 0 || cx >= m.nx)
                continue;
            const int cy = r ? row1 : row0, ly = r ? ly1 : ly0;
            const size_t e = size_t(cy) * m.nx + cx;
            const size_t n0 = size_t(cy) * s1 + cx;
            const double loc[4] = { cg1[n0], cg1[n0 + 1], cg1[n0 + s1], cg1[n0 + s1 + 1] };
            const int k = lx + 2 * ly;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                au = fma(-o.dxssh[(k * 4 + j) * N + e], loc[j], au);
                av = fma(-o.dyssh[(k * 4 + j) * N + e], loc[j], av);
            }
        }
    }
    const double im = o.invm1[t];
    ug[t] = au * im;
    vg[t] = av * im;
}

// Pressure at the 3 x 3 Gauss points (MEVPStressUpdateStep.hpp:54-57, 75-77)
// and the nine Lagrange values of h and A, which the nodes average.  Bound by
// FP64 issue, about 230 instructions per element: 154 us for 512 x 512 elements
// with six modes (201 us with dense products and CUDA's exp and without the
// Lagrange values; the averages then took 103 us more).
template <int DG>
__global__ void __launch_bounds__(kBlock) kMevpPrepElements(size_t N, const double* __restrict__ h,
    const double* __restrict__ a, double* __restrict__ lagH, double* __restrict__ lagA, PressureOut out, double pAlpha,
    const float* __restrict__ tdiv32, float* __restrict__ tdivLast)
{
    const size_t e = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
    if (e >= N)
        return;
    if (tdivLast) // the divergence at the start of this sub-cycle (warm-start features)
#pragma unroll
        for (int k = 0; k < 18; ++k)
            tdivLast[k * N + e] = tdiv32[k * N + e];
    double hc[DG], ac[DG], hg[9], ag[9];
#pragma unroll
    for (int j = 0; j < DG; ++j) {
        hc[j] = h[j * N + e];
        ac[j] = a[j * N + e];
    }
    storeLagrange<DG>(hc, ac, N, e, lagH, lagA);
    gaussValues<DG>(hc, hg);
    gaussValues<DG>(ac, ag);
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        const double hq = atLeast(hg[q], 0.0);
        const double aq = atMost(atLeast(ag[q], 0.0), 1.0);
        const double pa = pAlpha * hq * exp64(fma(20.0, aq, -20.0));
        const size_t at = q * N + e;
        if (out.weighted)
            out.weighted[at] = pa * (0.25 * out.w[at]);
        if (out.weightedPair) {
            const double x = pa * (0.25 * out.w[at]);
            const float hi = nsdg_ff::narrowAny(x);
            out.weightedPair[at] = make_float2(hi, nsdg_ff::narrowAny(x - nsdg_ff::widenNonneg(hi)));
        }
        if (out.alpha)
            out.alpha[at] = pa;
        if (out.visc) {
            out.visc[at] = 0.125 * pa;
            out.half[at] = nsdg_ff::narrowAny(0.5 * pa);
        }
    }
}

// The nodes' preparation: averages, clamps, gradient and the constants in one
// pass, one thread for a cell's four nodes (in pieces, 1025 x 1025 nodes: 103 us
// for the averages, 21 for the gradient's interpolation and 91 for the
// constants; together 89).
//
// The FP64 path's node constants (kMevpMomentum).
template <bool CONST>
__global__ void __launch_bounds__(kBlock) kMevpPrepNodes(int nx, int ny, size_t N, NodeInputs in, MevpNodeState st,
    MevpParams p)
{
    const CellNodes c(blockIdx.x * kBlock + threadIdx.x, nx, ny);
    if (!c.exists[0])
        return;
    double A[4], H[4], gx[4], gy[4];
    nodeFields<CONST>(c, nx, ny, N, in, A, H, gx, gy);
#pragma unroll
    for (int n = 0; n < 4; ++n) {
        if (!c.exists[n])
            continue;
        const size_t i = c.id[n];
        const double rc1 = p.dt * recip64(p.rho_ice * H[n]);
        const double ua = in.ua[i], va = in.va[i];
        const double af = A[n] * rc1, w = af * (p.F_atm * sqrt64(fma(ua, ua, va * va)));
        st.a[i] = af * p.F_ocean;
        st.ku[i] = fma(w, ua, fma(-p.dt * p.gravity, gx[n], in.u[i]));
        st.kv[i] = fma(w, va, fma(-p.dt * p.gravity, gy[n], in.v[i]));
        st.im[i] = in.invm2[i] * rc1;
    }
}

// The mixed path's: the same, as floats (kMevpMomentum32).
template <bool CONST>
__global__ void __launch_bounds__(kBlock) kMevpPrepNodes32(int nx, int ny, size_t N, NodeInputs in, MevpNodeState32 f,
    const uint8_t* __restrict__ dir, MevpParams p, float* __restrict__ uLast, float* __restrict__ vLast)
{
    const CellNodes c(blockIdx.x * kBlock + threadIdx.x, nx, ny);
    if (!c.exists[0])
        return;
    double A[4], H[4], gx[4], gy[4];
    nodeFields<CONST>(c, nx, ny, N, in, A, H, gx, gy);
#pragma unroll
    for (int n = 0; n < 4; ++n) {
        if (!c.exists[n])
            continue;
        const size_t i = c.id[n];
        const double u = in.u[i], v = in.v[i];
        const float uf = nsdg_ff::narrowAny(u), vf = nsdg_ff::narrowAny(v);
        f.u[i] = uf;
        f.v[i] = vf;
        f.u0[i] = uf;
        f.v0[i] = vf;
        if (uLast) { // the velocity at the start of this sub-cycle (warm-start features)
            uLast[i] = uf;
            vLast[i] = vf;
        }
        const double rc1 = p.dt * recip64(p.rho_ice * H[n]);
        const double ua = in.ua[i], va = in.va[i];
        const double af = A[n] * rc1, w = af * (p.F_atm * sqrt64(fma(ua, ua, va * va)));
        const double ku = fma(w, ua, fma(-p.dt * p.gravity, gx[n], u));
        const double kv = fma(w, va, fma(-p.dt * p.gravity, gy[n], v));
        const double im = in.invm2[i] * rc1;
        const float hi = nsdg_ff::narrowAny(im);
        f.k0[i] = make_float4(nsdg_ff::narrowAny(af), nsdg_ff::narrowAny(ku), nsdg_ff::narrowAny(kv),
            nsdg_ff::narrowAny(in.uo[i]));
        f.k1[i] = make_float4(nsdg_ff::narrowAny(in.vo[i]), hi,
            nsdg_ff::narrowAny(im - nsdg_ff::widenNonneg(hi)), dir[i] ? 1.f : 0.f);
    }
}

} // namespace

__global__ void kJoin() { }
cudaError_t launchJoin(cudaStream_t s)
{
    kJoin<<<1, 1, 0, s>>>();
    return cudaGetLastError();
}

cudaError_t launchAverage(cudaStream_t s, const DevMesh& m, const AverageFields& f)
{
    const unsigned g = blocksFor(cellsAndBorder(m.nx, m.ny));
    switch (f.count) {
    case 1: kAverage<1><<<g, kBlock, 0, s>>>(m.nx, m.ny, f); break;
    case 2: kAverage<2><<<g, kBlock, 0, s>>>(m.nx, m.ny, f); break;
    case 3: kAverage<3><<<g, kBlock, 0, s>>>(m.nx, m.ny, f); break;
    case 4: kAverage<4><<<g, kBlock, 0, s>>>(m.nx, m.ny, f); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launchSSHGradient(cudaStream_t s, const DevMesh& m, const DevOps& o, const double* ssh, double* cg1,
    double* ug, double* vg)
{
    kSSHToCG1<<<blocksFor(cellsAndBorder(m.nx, m.ny)), kBlock, 0, s>>>(m, ssh, cg1);
    kSSHGrad1<<<blocksFor(m.Ncg1), kBlock, 0, s>>>(m, o, cg1, ug, vg);
    return cudaGetLastError();
}

cudaError_t launchMevpPrepElements(cudaStream_t s, const DevMesh& m, int dg, const double* h, const double* a,
    double* lagH, double* lagA, const PressureOut& out, const MevpParams& p, const float* tdiv32, float* tdivLast)
{
    const unsigned g = blocksFor(m.N);
    const double pa = p.Pstar * (1.0 / p.alpha);
    switch (dg) {
    case 1: kMevpPrepElements<1><<<g, kBlock, 0, s>>>(m.N, h, a, lagH, lagA, out, pa, tdiv32, tdivLast); break;
    case 3: kMevpPrepElements<3><<<g, kBlock, 0, s>>>(m.N, h, a, lagH, lagA, out, pa, tdiv32, tdivLast); break;
    case 6: kMevpPrepElements<6><<<g, kBlock, 0, s>>>(m.N, h, a, lagH, lagA, out, pa, tdiv32, tdivLast); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launchMevpPrepNodes(cudaStream_t s, const DevMesh& m, const NodeInputs& in, const MevpNodeState& st,
    const MevpParams& p)
{
    const unsigned g = blocksFor(cellsAndBorder(m.nx, m.ny));
    if (in.constant)
        kMevpPrepNodes<true><<<g, kBlock, 0, s>>>(m.nx, m.ny, m.N, in, st, p);
    else
        kMevpPrepNodes<false><<<g, kBlock, 0, s>>>(m.nx, m.ny, m.N, in, st, p);
    return cudaGetLastError();
}

cudaError_t launchMevpPrepNodes32(cudaStream_t s, const DevMesh& m, const NodeInputs& in, const MevpNodeState32& st32,
    const MevpParams& p, float* uLast, float* vLast)
{
    const unsigned g = blocksFor(cellsAndBorder(m.nx, m.ny));
    if (in.constant)
        kMevpPrepNodes32<true><<<g, kBlock, 0, s>>>(m.nx, m.ny, m.N, in, st32, m.cg2Dir, p, uLast, vLast);
    else
        kMevpPrepNodes32<false><<<g, kBlock, 0, s>>>(m.nx, m.ny, m.N, in, st32, m.cg2Dir, p, uLast, vLast);
    return cudaGetLastError();
}

} // namespace nsdg
