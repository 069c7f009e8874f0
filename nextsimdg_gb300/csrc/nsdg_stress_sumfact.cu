// nsdg_stress_sumfact.cu — the sum-factorised mEVP element kernels
// (nsdg_sumfact.cuh): FP64, mixed precision, and mixed precision batched over
// an ensemble's members.
#include "nsdg_stress_fixed.cuh"
#include "nsdg_sumfact.cuh"

namespace nsdg {
namespace {

using namespace sf;

// FP64 (nsdg_stress_fixed.cuh).  Bound by FP64 issue (108 instructions per
// element) and the integer work beside it.  Per launch in a row of them, the
// launch included (about 3 us): 21.4 us for 256 x 256 rectangles, 20.4 us for 201 x
// 143 quadrilaterals, 14.4 us for 154 x 121 cells of a sphere, 6.7 us for 64 x 64
// rectangles.  (Without the launch, with the linear maps in FP64 60.8, 42, 32 and
// 7.4 us, with 9 x 9 operators streamed from memory 112, 49, 44 and 20.5.)  Three
// threads per element: with one, a 64 x 64 grid is one warp per SM that waits out
// every instruction's latency.  The blocks per SM bound the registers at 80, 128
// and 168: with five a sphere's kernel spills (update of 154 x 121 cells 2.08
// against 1.92 ms), with six quadrilaterals' did (16.9 against 16.5 us per launch).
constexpr int kElems = kFixedElems;

template <Geometry GEO>
__global__ void __launch_bounds__(3 * kElems, GEO == RECT ? 8 : GEO == QUAD ? 5 : 4) kMevpStress(DevMesh m,
    FixedGeometry geo, const double* __restrict__ u, const double* __restrict__ v, const double* __restrict__ Pw,
    double* __restrict__ tdiv, double dmin2, double keep, bool release)
{
    __shared__ FixedShared<GEO, kElems> sh;
    stressFixed<GEO, kElems>(m.nx, m.N, m.ice, geo, u, v, Pw, tdiv, dmin2, keep, release, blockIdx.x * size_t(kElems),
        sh);
}

// Mixed precision: FP32 velocities, divergence and arithmetic, Delta^2 and the
// viscosity in float pairs.  Per element and iteration 260 bytes on
// parallelograms (divergence 144, weighted pressure 72, coefficients 16, its
// share of the velocities) and 430 on quadrilaterals (+ 180 of map, 216 on a
// sphere), where the 9 x 9 operators were 1,580 (2,228).  Bound by L2 / HBM
// traffic: per launch in a row of them, the launch included, 12.3 us for 512 x 512
// parallelograms = 5.6 TB/s (24.9 us with dense unit-square operators and the
// viscosity in FP64, which was bound by FP64 issue), 10.3 us for 384 x 320
// quadrilaterals (42.7 us with TMA-staged operators), 9.2 us for 301 x 257 cells of
// a sphere (38.6 us).
//
// Three threads per element keep small grids' latency down; from
// kOneThreadElems elements the SMs are full either way and one thread per
// element issues about 950 instructions instead of 1,700 (shared-memory
// exchange, indices).  Updates of 100 iterations, three threads against one, ms:
//   parallelograms  64^2 .459 / .489   96^2 .484 / .496  128^2 .540 / .519
//                  192^2 .687 / .658  256^2 .875 / .838  512^2 2.66 / 2.29
//   quadrilaterals  64^2 .530 / .565   96^2 .571 / .580  128^2 .684 / .621
//                  192^2 .781 / .795  256^2 1.13 / .973  384^2 2.16 / 1.83
template <Geometry GEO, int VM, int E>
__global__ void __launch_bounds__(3 * E) kMevpStress32(DevMesh m, StressGeometry<float> geo,
    const float* __restrict__ u, const float* __restrict__ v, const float2* __restrict__ Pw, float* __restrict__ tdiv,
    Rheology<float> rh, float keep)
{
    __shared__ Exchange<float, E> ex;
    __shared__ float sums[GEO == AFFINE ? 1 : 2][3][3][E];
    stressBlock<float, GEO, VM, E>(m.nx, m.N, m.ice, geo, u, v, Pw, tdiv, rh, keep, blockIdx.x * size_t(E), ex, sums);
}

// One thread per element, for kOneThreadElems elements or more.
template <Geometry GEO>
__global__ void __launch_bounds__(kQuadElems) kMevpStress32Thread(DevMesh m, StressGeometry<float> geo,
    const float* __restrict__ u, const float* __restrict__ v, const float2* __restrict__ Pw, float* __restrict__ tdiv,
    Rheology<float> rh, float keep)
{
    stressThread<float, GEO, 3>(m.nx, m.N, m.ice, geo, u, v, Pw, tdiv, rh, keep,
        blockIdx.x * size_t(kQuadElems) + threadIdx.x);
}

// One launch over the elements of every member of an ensemble: block b belongs
// to member blockMember[b] and covers E consecutive elements of it.
template <Geometry GEO, int VM, int E>
__global__ void __launch_bounds__(3 * E) kMevpStress32Batched(const EnsembleMember* __restrict__ members,
    const uint16_t* __restrict__ blockMember, Rheology<float> rh, float keep)
{
    __shared__ Exchange<float, E> ex;
    __shared__ float sums[GEO == AFFINE ? 1 : 2][3][3][E];
    const EnsembleMember& M = members[blockMember[blockIdx.x]];
    const int b = static_cast<int>(blockIdx.x) - (GEO == AFFINE ? M.tmaBlock0 : M.stressBlock0);
    stressBlock<float, GEO, VM, E>(M.nx, M.N, M.ice, GEO == AFFINE ? M.aff : M.quad, M.st.u, M.st.v, M.Pw, M.tdiv, rh,
        keep, size_t(b) * E, ex, sums);
}

template <Geometry GEO>
__global__ void __launch_bounds__(kQuadElems) kMevpStress32ThreadBatched(const EnsembleMember* __restrict__ members,
    const uint16_t* __restrict__ blockMember, Rheology<float> rh, float keep)
{
    const EnsembleMember& M = members[blockMember[blockIdx.x]];
    const int b = static_cast<int>(blockIdx.x) - M.stressBlock0;
    stressThread<float, GEO, 3>(M.nx, M.N, M.ice, GEO == AFFINE ? M.aff : M.quad, M.st.u, M.st.v, M.Pw, M.tdiv, rh,
        keep, size_t(b) * kQuadElems + threadIdx.x);
}

size_t blocksOf(size_t n) { return (n + kQuadElems - 1) / kQuadElems; }

} // namespace

cudaError_t launchMevpStress(cudaStream_t s, const DevMesh& m, const FixedGeometry& geo, const double* u,
    const double* v, const double* Pw, double* tdiv, const MevpParams& pIn, bool programmatic)
{
    const MevpParams p = withDerived(pIn);
    const size_t blocks = (m.N + kElems - 1) / kElems;
    auto kernel = geo.rect ? kMevpStress<RECT> : geo.m ? kMevpStress<SPHERE> : kMevpStress<QUAD>;
    return launchAfter(programmatic, s, kernel, blocks, 3 * kElems, 0, m, geo, u, v, Pw, tdiv, p.DeltaMin *
        p.DeltaMin, p.keepd, releaseEarly64(m.N));
}

cudaError_t launchMevpStress32(cudaStream_t s, const DevMesh& m, const StressGeometry<float>& geo, const float* u,
    const float* v, const float2* Pw, float* tdiv, const MevpParams& pIn, bool programmatic)
{
    const MevpParams p = withDerived(pIn);
    const Rheology<float> rh { p.dmin2f, p.dmin2lo, p.DeltaMin };
    if (m.N >= kOneThreadElems)
        return launchAfter(programmatic, s, geo.m ? kMevpStress32Thread<SPHERE> : kMevpStress32Thread<QUAD>,
            blocksOf(m.N), kQuadElems, 0, m, geo, u, v, Pw, tdiv, rh, p.keep);
    auto kernel = geo.m ? kMevpStress32<SPHERE, 3, kQuadElems> : kMevpStress32<QUAD, 3, kQuadElems>;
    return launchAfter(programmatic, s, kernel, (m.N + kQuadElems - 1) / kQuadElems, 3 * kQuadElems, 0, m, geo, u, v,
        Pw, tdiv, rh, p.keep);
}

cudaError_t launchMevpStress32Affine(cudaStream_t s, const DevMesh& m, const StressGeometry<float>& geo,
    const float* u, const float* v, const float2* Pw, float* tdiv, const MevpParams& pIn, int viscosityMode,
    bool programmatic)
{
    const MevpParams p = withDerived(pIn);
    const Rheology<float> rh { p.dmin2f, p.dmin2lo, p.DeltaMin };
    void (*kernels[5])(DevMesh, StressGeometry<float>, const float*, const float*, const float2*, float*,
        Rheology<float>, float)
        = { kMevpStress32<AFFINE, 0, kAffElems>, kMevpStress32<AFFINE, 1, kAffElems>,
              kMevpStress32<AFFINE, 2, kAffElems>, kMevpStress32<AFFINE, 3, kAffElems>,
              kMevpStress32<AFFINE, 4, kAffElems> };
    const int vm = viscosityMode >= 0 && viscosityMode <= 4 ? viscosityMode : 3;
    if (vm == 3 && m.N >= kOneThreadElems)
        return launchAfter(programmatic, s, kMevpStress32Thread<AFFINE>, blocksOf(m.N), kQuadElems, 0, m, geo, u, v,
            Pw, tdiv, rh, p.keep);
    return launchAfter(programmatic, s, kernels[vm], (m.N + kAffElems - 1) / kAffElems, 3 * kAffElems, 0, m, geo, u,
        v, Pw, tdiv, rh, p.keep);
}

cudaError_t launchMevpStress32Batched(cudaStream_t s, const EnsembleMember* members, const uint16_t* blockMember,
    int blocks, size_t elements, const MevpParams& pIn)
{
    const MevpParams p = withDerived(pIn);
    const Rheology<float> rh { p.dmin2f, p.dmin2lo, p.DeltaMin };
    if (elements >= kOneThreadElems)
        return launchAfter(true, s, kMevpStress32ThreadBatched<QUAD>, blocks, kQuadElems, 0, members, blockMember, rh,
            p.keep);
    return launchAfter(true, s, kMevpStress32Batched<QUAD, 3, kQuadElems>, blocks, 3 * kQuadElems, 0, members,
        blockMember, rh, p.keep);
}

cudaError_t launchMevpStress32AffineThreadBatched(cudaStream_t s, const EnsembleMember* members,
    const uint16_t* blockMember, int blocks, const MevpParams& pIn)
{
    const MevpParams p = withDerived(pIn);
    const Rheology<float> rh { p.dmin2f, p.dmin2lo, p.DeltaMin };
    return launchAfter(true, s, kMevpStress32ThreadBatched<AFFINE>, blocks, kQuadElems, 0, members, blockMember, rh,
        p.keep);
}

cudaError_t launchMevpStress32AffineBatched(cudaStream_t s, const EnsembleMember* members,
    const uint16_t* blockMember, int blocks, const MevpParams& pIn, int viscosityMode)
{
    const MevpParams p = withDerived(pIn);
    const Rheology<float> rh { p.dmin2f, p.dmin2lo, p.DeltaMin };
    void (*kernels[5])(const EnsembleMember*, const uint16_t*, Rheology<float>, float)
        = { kMevpStress32Batched<AFFINE, 0, kAffElems>, kMevpStress32Batched<AFFINE, 1, kAffElems>,
              kMevpStress32Batched<AFFINE, 2, kAffElems>, kMevpStress32Batched<AFFINE, 3, kAffElems>,
              kMevpStress32Batched<AFFINE, 4, kAffElems> };
    const int vm = viscosityMode >= 0 && viscosityMode <= 4 ? viscosityMode : 3;
    return launchAfter(true, s, kernels[vm], blocks, 3 * kAffElems, 0, members, blockMember, rh, p.keep);
}

} // namespace nsdg
