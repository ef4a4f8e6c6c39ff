// gravity.cu -- self-gravity with a live potential for sm_103a: the potential's
// starting guess, its ghost fill, the Poisson relaxation sweeps and the gravity
// source term fused with the integrator's combine.
//
// Reference pieces replaced (KennethYeah/HydrodynamicsGPU):
//  * SelfGravitation::resetState (src/Solver/SelfGravitation.cpp:35-98): with
//    useGravity the potential starts as -density, is relaxed, and the starting guess
//    (the host vector, not the relaxed buffer) is added to the total energy;
//  * SelfGravitation::potentialBoundary (:126-140) with the potential's boundary
//    kernels (include/HydroGPU/Equation/SelfGravitationBehavior.h:22-34: PERIODIC ->
//    periodic, MIRROR and FREEFLOW -> free flow) on a stride-1 buffer;
//  * gravityPotentialPoissonRelax (res/SelfGravitation.cl:20-63).  The reference
//    kernel updates the potential in place while its neighbours read it, so a launch
//    has no single result: each order in which a device runs the work-items gives its
//    own.  Here a launch is the red-black order, one of those the reference permits:
//    every interior cell with x + y + z even first (their neighbours are all odd, so
//    these updates do not see each other), then every odd cell (reading the new even
//    values).  It is deterministic and each half is one parallel sweep;
//  * calcGravityDeriv (res/SelfGravitation.cl:65-102) into a deriv that goes straight
//    into the integrator's combine (combinePlanCell), as the flux divergence does.
// Per-cell expressions follow the reference's operation order and types: in FP32 the
// double literals of `4. * M_PI * G * density`, `-2. * (1. / (DX * DX) ...)` and
// `/ (2. * dx[side])` promote those expressions to double.
#include "../../../include/hgpu/hgpu.h"
#include "launch.cuh"
#include "combine_cells.cuh"
#include "gravity.h"

namespace hgpu {
namespace {

constexpr int kThreads = 256;
inline unsigned blocksFor(long long n) { return (unsigned)((n + kThreads - 1) / kThreads); }

// potential = -density (useGravity) or the given channel; total energy += that potential
template <typename real, int D>
__global__ void __launch_bounds__(kThreads) potentialInitKernel(Grid g, int fromDensity, real* state,
                                                                real* pot, long long c0, long long c1) {
    dependentLaunch();
    const long long c = c0 + (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= c1) return;
    real* s = state + (long long)(D + 2) * c;
    const real p = fromDensity ? -s[0] : pot[c];
    pot[c] = p;
    s[D + 1] = s[D + 1] + p;
}

// the potential's ghost fill along one axis: boundaryLine on a one-component buffer
template <typename real>
__global__ void __launch_bounds__(kThreads) potentialBoundaryKernel(Grid g, int axis, int mMin, int mMax,
                                                                    real* pot) {
    dependentLaunch();
    boundaryLine<real>(g, axis, 1, mMin, mMax, pot, (long long)blockIdx.x * blockDim.x + threadIdx.x);
}

// rhs = 4. * M_PI * G * density (double) of every cell, from the stage state: fixed
// while a callback's sweeps run, so it is formed once and the sweeps read 8 bytes a
// cell instead of the state's record
template <typename real, int D>
__global__ void __launch_bounds__(kThreads) relaxRhsKernel(Grid g, GravityConst<real> gc,
                                                           const real* state, double* __restrict__ rhs) {
    dependentLaunch();
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= g.V) return;
    rhs[c] = mulI(gc.fourPiG, (double)state[(long long)(D + 2) * c]);
}

// one colour of a relaxation sweep: blockIdx.y (+ gridDim.y * blockIdx.z) = the interior
// row (y, z), thread x = the k-th cell of that colour along the row.
// skewSum adds phi / dx^2 of the +x, -x, +y, -y, +z, -z neighbours inside [2, S-3]
// (SelfGravitation.cl:39-51).  Each cell's quotients serve all its neighbours of the other
// colour, so the update that makes a cell's phi also stores them (`quot`: one plane when
// the axes' dx^2 are equal (SAME), else one per axis), and a cell costs its own two
// quotients (phi's and the one by diag) instead of 2 D + 1.  FIRST: the colour before has
// no quotients yet; they are formed from its potential.  STORE: the potential itself is
// written too (nothing reads it between sweeps).  1024^2 FP64: 19.2 us a sweep, 23.2 with
// every neighbour's quotient formed in place; bound by the FP64 unit's four sums a cell and
// the quotients' integer work.
template <typename real, int D, bool SAME, bool FIRST>
__global__ void __launch_bounds__(kThreads) relaxKernel(Grid g, GravityConst<real> gc, int colour, bool store,
                                                        const double* rhs, real* quot,
                                                        real* pot) {
    dependentLaunch();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = D > 1 ? (int)blockIdx.y + 2 : 0, z = D > 2 ? (int)blockIdx.z + 2 : 0;
    // x = 2 + 2k + shift, with shift chosen so that x + y + z has the colour's parity
    const int x = 2 + 2 * k + (((y + z) & 1) ^ colour);
    if (x >= g.S[0] - 2) return;
    const long long c = x + (long long)g.S[0] * (y + (long long)g.S[1] * z);
    if (!cellOk(g, c)) return;
    const int at[3] = {x, y, z};
    real skewSum = (real)0;
#pragma unroll
    for (int a = 0; a < D; ++a) {
        const real* q = quot + (SAME ? 0 : a * g.V);
        // a neighbour outside [2, S-3] adds +0, which changes no sum that starts from +0
        const bool up = at[a] < g.S[a] - 3, down = at[a] > 2;
        const long long st = g.step[a];
        real u = (real)0, d = (real)0;
        if (up) u = FIRST ? quotBy(pot[c + st], gc.dxSq[a]) : q[c + st];
        if (down) d = FIRST ? quotBy(pot[c - st], gc.dxSq[a]) : q[c - st];
        skewSum = a == 0 ? zfix(u) : skewSum + u;
        skewSum = skewSum + d;
    }
    // (4. * M_PI * G * density - skewSum) / diag, in double for both precisions
    const double rest = rhs[c] - (double)skewSum;
    if constexpr (sizeof(real) == 8) {
        // ordinary numbers in every lane: the quotients without a branch each
        const double phi = quotPlain(rest, gc.diag);
        if (warpAll(inWindow(rest) & inWindow(phi) & inWindow(gc.diag.b) & inWindow(gc.dxSq[0].b) &
                    inWindow(gc.dxSq[D - 1].b) & inWindow(gc.dxSq[D / 2].b))) {
#pragma unroll
            for (int a = 0; a < (SAME ? 1 : D); ++a) quot[a * g.V + c] = quotPlain(phi, gc.dxSq[a]);
            if (store) pot[c] = phi;
            return;
        }
    }
    const real phi = (real)quotBy(rest, gc.diag);
#pragma unroll
    for (int a = 0; a < (SAME ? 1 : D); ++a) quot[a * g.V + c] = quotBy(phi, gc.dxSq[a]);
    if (store) pot[c] = phi;
}

// calcGravityDeriv of one cell into d (zero outside the interior), then the combine
template <typename real, int D>
__global__ void __launch_bounds__(kThreads) gravityCombineKernel(Grid g, GravityConst<real> gc,
                                                                 const real* stage,
                                                                 const real* pot, CombinePlan<real> plan,
                                                                 const StepConst<real>* sc) {
    dependentLaunch();
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= g.V) return;
    int x, y, z;
    cellCoords(g, c, x, y, z);
    const int N = D + 2, E = D + 1;
    real d[N];
#pragma unroll
    for (int j = 0; j < N; ++j) d[j] = (real)0;
    if (inRange(g, x, y, z, 2, 2)) {
        const real* st = stage + (long long)N * c;
        const real density = st[0];
        real derivEnergyTotal = (real)0;
#pragma unroll
        for (int side = 0; side < D; ++side) {
            const long long sp = g.step[side];
            const real dphi = pot[c + sp] - pot[c - sp];
            // (phi[next] - phi[prev]) / (2. * dx[side]): a double quotient, stored as real
            const real gradient = (real)quotBy((double)dphi, gc.twoDx[side]);
            const real gravity = -gradient;
            const real f = mulI(density, gravity);
            d[1 + side] = zfix(-f);                                  // deriv (+0) -= density * gravity
            const real e = mulI(f, st[1 + side]);
            derivEnergyTotal = side == 0 ? zfix(-e) : derivEnergyTotal - e;
        }
        d[E] = zfix(derivEnergyTotal);                               // deriv[E] (+0) += derivEnergyTotal
    }
    combinePlanCell<real, D>(d, plan, *sc, c, 0);
}

}  // namespace

template <typename real>
GravityConst<real> gravityConst(const double dx[3], double G, int dim) {
    GravityConst<real> gc;
    // ((real)G) as the program's define makes it; 4. * M_PI * G in double, left to right
    gc.fourPiG = (4. * 3.14159265358979323846) * (double)(real)G;
    double invSum = 0.;
    for (int i = 0; i < dim; ++i) {
        const real dxr = (real)dx[i];
        const real sq = dxr * dxr;                                  // DX * DX in the program's type
        hostDivisor(sq, gc.dxSq[i]);
        invSum = i == 0 ? 1. / (double)sq : invSum + 1. / (double)sq;
        hostDivisor(2. * (double)dxr, gc.twoDx[i]);
    }
    for (int i = dim; i < 3; ++i) { hostDivisor((real)1, gc.dxSq[i]); hostDivisor(2., gc.twoDx[i]); }
    hostDivisor((double)(real)(-2. * invSum), gc.diag);              // `const real diag`
    return gc;
}

template <typename real>
void launchPotentialInit(const Grid& g, int fromDensity, real* state, real* pot, cudaStream_t st, long long c0,
                         long long c1) {
    if (c1 < 0 || c1 > g.V) c1 = g.V;
    if (c0 < 0) c0 = 0;
    if (c0 >= c1) return;
    const unsigned b = blocksFor(c1 - c0);
    if (g.dim == 1) launchDependent(potentialInitKernel<real, 1>, b, kThreads, 0, st, g, fromDensity, state, pot, c0, c1);
    else if (g.dim == 2) launchDependent(potentialInitKernel<real, 2>, b, kThreads, 0, st, g, fromDensity, state, pot, c0, c1);
    else launchDependent(potentialInitKernel<real, 3>, b, kThreads, 0, st, g, fromDensity, state, pot, c0, c1);
}

template <typename real>
void launchPotentialBoundary(const Grid& g, const int methods[3][2], real* pot, cudaStream_t st) {
    for (int axis = 0; axis < g.dim; ++axis) {
        int m[2];
        for (int k = 0; k < 2; ++k)
            m[k] = methods[axis][k] == HGPU_BOUNDARY_MIRROR ? HGPU_BOUNDARY_FREEFLOW : methods[axis][k];
        const long long n = g.dim == 1 ? 1 : (long long)g.S[axis == 0 ? 1 : 0] * g.S[axis == 2 ? 1 : 2];
        launchDependent(potentialBoundaryKernel<real>, blocksFor(n), kThreads, 0, st, g, axis, m[0], m[1], pot);
    }
}

template <typename real>
void launchRelaxRhs(const Grid& g, const GravityConst<real>& gc, const real* state, double* rhs, cudaStream_t st) {
    if (g.dim == 1) launchDependent(relaxRhsKernel<real, 1>, blocksFor(g.V), kThreads, 0, st, g, gc, state, rhs);
    else if (g.dim == 2) launchDependent(relaxRhsKernel<real, 2>, blocksFor(g.V), kThreads, 0, st, g, gc, state, rhs);
    else launchDependent(relaxRhsKernel<real, 3>, blocksFor(g.V), kThreads, 0, st, g, gc, state, rhs);
}

template <typename real, int D, bool SAME>
static void relaxSweep(const Grid& g, const GravityConst<real>& gc, const double* rhs, real* quot, real* pot, bool first,
                       bool store, cudaStream_t st) {
    const int nx = g.S[0] - 4, ny = D > 1 ? g.S[1] - 4 : 1, nz = D > 2 ? g.S[2] - 4 : 1;
    if (nx <= 0 || ny <= 0 || nz <= 0) return;
    const dim3 grid((unsigned)((nx + 1) / 2 + kThreads - 1) / kThreads, (unsigned)ny, (unsigned)nz);
    if (first) launchDependent(relaxKernel<real, D, SAME, true>, grid, kThreads, 0, st, g, gc, 0, store, rhs, quot, pot);
    else launchDependent(relaxKernel<real, D, SAME, false>, grid, kThreads, 0, st, g, gc, 0, store, rhs, quot, pot);
    launchDependent(relaxKernel<real, D, SAME, false>, grid, kThreads, 0, st, g, gc, 1, store, rhs, quot, pot);
}

template <typename real>
int relaxQuotPlanes(const Grid& g, const GravityConst<real>& gc) {
    for (int a = 1; a < g.dim; ++a)
        if (gc.dxSq[a].b != gc.dxSq[0].b) return g.dim;
    return 1;
}

template <typename real>
void launchRelaxSweep(const Grid& g, const GravityConst<real>& gc, const double* rhs, real* quot, real* pot, bool first,
                      bool store, cudaStream_t st) {
    const bool same = relaxQuotPlanes(g, gc) == 1;
    if (g.dim == 1) relaxSweep<real, 1, true>(g, gc, rhs, quot, pot, first, store, st);
    else if (g.dim == 2 && same) relaxSweep<real, 2, true>(g, gc, rhs, quot, pot, first, store, st);
    else if (g.dim == 2) relaxSweep<real, 2, false>(g, gc, rhs, quot, pot, first, store, st);
    else if (same) relaxSweep<real, 3, true>(g, gc, rhs, quot, pot, first, store, st);
    else relaxSweep<real, 3, false>(g, gc, rhs, quot, pot, first, store, st);
}

template <typename real>
void launchGravityCombine(const Grid& g, const GravityConst<real>& gc, const real* stage, const real* pot,
                          const CombinePlan<real>& plan, const StepConst<real>* sc, cudaStream_t st) {
    if (g.dim == 1) launchDependent(gravityCombineKernel<real, 1>, blocksFor(g.V), kThreads, 0, st, g, gc, stage, pot, plan, sc);
    else if (g.dim == 2) launchDependent(gravityCombineKernel<real, 2>, blocksFor(g.V), kThreads, 0, st, g, gc,
            stage, pot, plan, sc);
    else launchDependent(gravityCombineKernel<real, 3>, blocksFor(g.V), kThreads, 0, st, g, gc, stage, pot, plan, sc);
}

#define INST(real)                                                                                              \
    template GravityConst<real> gravityConst<real>(const double[3], double, int);                              \
    template void launchPotentialInit<real>(const Grid&, int, real*, real*, cudaStream_t, long long, long long);                      \
    template void launchPotentialBoundary<real>(const Grid&, const int[3][2], real*, cudaStream_t);            \
    template void launchRelaxRhs<real>(const Grid&, const GravityConst<real>&, const real*, double*, cudaStream_t); \
    template int relaxQuotPlanes<real>(const Grid&, const GravityConst<real>&);                                  \
    template void launchRelaxSweep<real>(const Grid&, const GravityConst<real>&, const double*, real*, real*, bool, \
                                         bool, cudaStream_t);                                                   \
    template void launchGravityCombine<real>(const Grid&, const GravityConst<real>&, const real*, const real*,    \
                                             const CombinePlan<real>&, const StepConst<real>*, cudaStream_t);
INST(double)
INST(float)
#undef INST

}  // namespace hgpu
