// combine.cu -- ghost fill, flux divergence + Runge-Kutta stage combine, dt finalisation.
//
// Reference pieces replaced:
//  * Solver::boundary + stateBoundary* kernels (src/Solver/Solver.cpp:448-464,
//    res/Common.cl:49-194): one launch per axis handles every state and both sides;
//  * calcFluxDeriv (res/CalcFluxDeriv.cl:7-44) fused with the integrator's multAdd
//    chain (res/Common.cl:201-210, include/HydroGPU/Integrator/RungeKutta.h:59-125):
//    instead of zero-filling a deriv buffer per stage and re-summing every stage
//    state from buffers, each stage adds its column of the tableau to the running
//    sums of all later rows.  Row m's additions still happen in column order, alpha
//    term before beta term, starting from +0, so every sum is bit-identical;
//  * findMinTimestep's host read and `dt * cfl` (Solver.cpp:466-516): dt is
//    finalised on the device, with dt/dx and beta*dt, for the whole step.
#include <cstring>

#include "combine_cells.cuh"
#include "kernels.h"
#include "launch.cuh"

namespace hgpu {

namespace {
const double kA[12][4][4] = HGPU_TABLE_A;
const double kB[12][4][4] = HGPU_TABLE_B;
const int kOrder[12] = HGPU_TABLE_ORDER;
}  // namespace

int tableauOrder(int integ) { return kOrder[integ]; }
double tableauAlpha(int integ, int m, int k) { return kA[integ][m][k]; }
double tableauBeta(int integ, int m, int k) { return kB[integ][m][k]; }

namespace {

constexpr int kThreads = 256;
inline unsigned blocksFor(long long n) { return (unsigned)((n + kThreads - 1) / kThreads); }

// ---------------- ghost fill ----------------
// one axis, one thread a line: axes of 5 cells, where the reference's fill order shows
// (a ghost is copied from a ghost filled before it)
template <typename real>
__global__ void __launch_bounds__(kThreads) boundaryKernel(Grid g, int axis, int N, int mMin, int mMax,
                                                           real* state, long long t0, long long t1) {
    dependentLaunch();
    const long long t = t0 + (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= t1) return;
    boundaryLine<real>(g, axis, N, mMin, mMax, state, t);
}

// one axis, one thread a ghost cell: thread (line t, k-th of the line's four ghosts)
template <typename real>
__global__ void __launch_bounds__(kThreads) ghostAxisKernel(Grid g, int axis, int N, int mMin, int mMax,
                                                            real* state, long long t0, long long t1) {
    dependentLaunch();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x, t = t0 + i / 4;
    if (t >= t1) return;
    const int k = (int)(i & 3), A = axis == 0 ? 1 : 0, S = g.S[axis];
    const long long nA = g.dim == 1 ? 1 : g.S[A];
    int c[3] = {0, 0, 0};
    c[A] = (int)(t % nA);
    if (g.dim > 1) c[axis == 2 ? 1 : 2] = (int)(t / nA);
    c[axis] = k < 2 ? k : S - 4 + k;
    Methods bc = {{{-1, -1}, {-1, -1}, {-1, -1}}};
    bc.m[axis][0] = mMin;
    bc.m[axis][1] = mMax;
    ghostCell<real>(g, N, bc, state, c[0], c[1], c[2]);
}

// every axis at once, one thread a ghost cell: the ghosts of axis 0 (n0 of them), then those
// of axis 1 inside axis 0's interior (n1), then those of axis 2 inside both.  The
// per-line form (a launch an axis, each thread copying its line's ghosts state by state and
// side by side, every copy after the one before) took 15 us at 133 x 97 and 17 us at
// 2048^2 for the two launches; this one 6 us at both (event-timed, launch included).
template <typename real>
__global__ void __launch_bounds__(kThreads) ghostKernel(Grid g, int N, Methods bc, real* state,
                                                        long long n0, long long n1, long long n) {
    dependentLaunch();
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    auto ghost = [](int k, int S) { return k < 2 ? k : S - 4 + k; };
    int x, y = 0, z = 0;
    if (i < n0) {
        x = ghost((int)(i & 3), g.S[0]);
        i >>= 2;
        y = (int)(i % g.S[1]);
        z = (int)(i / g.S[1]);
    } else if (i < n0 + n1) {
        i -= n0;
        const int w = g.S[0] - 4;
        x = 2 + (int)(i % w);
        i /= w;
        y = ghost((int)(i & 3), g.S[1]);
        z = (int)(i >> 2);
    } else {
        i -= n0 + n1;
        const int w = g.S[0] - 4, h = g.S[1] - 4;
        x = 2 + (int)(i % w);
        i /= w;
        y = 2 + (int)(i % h);
        z = ghost((int)(i / h), g.S[2]);
    }
    ghostCell<real>(g, N, bc, state, x, y, z);
}

// ---------------- flux divergence + stage combine ----------------
// 5 blocks per SM (46 registers, no spills; 52 registers gave 4): KH 2048^2 step -1.1 %
// POST: the zero-potential self-gravity pass of a tableau with fractional alphas, folded into
// the last stage (as a pass of its own over the state: 3D 160x144x136 RungeKutta2TVD 482 us
// of the step, 3D 99x90x86 RungeKutta3TVD 211 us; folded, 60 and 55 us more of combine)
template <typename real, int D, bool POST>
__global__ void __launch_bounds__(kThreads, D < 3 || sizeof(real) == 4 ? 5 : 4) derivCombineKernel(Grid g, Phys<real> ph, const real* flux,
                                                               CombinePlan<real> plan,
                                                               const StepConst<real>* sc, long long c0,
                                                               long long c1) {
    dependentLaunch();
    long long c = c0 + (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= c1) return;
    int x, y, z;
    cellCoords(g, c, x, y, z);
    derivCombineCell<real, D, false, POST>(g, ph, flux, plan, *sc, c, x, y, z, 0);
}

template <typename real>
__global__ void __launch_bounds__(kThreads) alphaOnlyKernel(long long n, int integ, real* state,
                                                            const StepConst<real>* sc) {
    dependentLaunch();
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    state[i] = alphaOnlyElem<real>(integ, state[i], *sc);
}

template <typename real>
__global__ void fixedDtKernel(Phys<real> ph, int integ, double fixedDt, StepConst<real>* sc) {
    dependentLaunch();
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    finalizeOne<real>(ph, integ, 1, fixedDt, nullptr, 0, sc);
}

// Self-gravity pass with ForwardEuler and a zero potential: the (ghost-refreshed)
// state gets `state + deriv * dt` with deriv == +0 (ForwardEuler.cpp:20-32).
template <typename real>
__global__ void __launch_bounds__(kThreads) zeroAddKernel(long long n, real* state,
                                                          const StepConst<real>* sc) {
    dependentLaunch();
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    state[i] = state[i] + (real)0. * sc->dt;
}

}  // namespace

long long boundaryLines(const Grid& g, int axis) {
    return g.dim == 1 ? 1 : (long long)g.S[axis == 0 ? 1 : 0] * g.S[axis == 2 ? 1 : 2];
}

template <typename real>
void launchBoundaryAxis(const Grid& g, const int methods[3][2], real* state, cudaStream_t st, int axis, long long t0,
                        long long t1) {
    const long long n = boundaryLines(g, axis);
    if (t1 < 0 || t1 > n) t1 = n;
    if (t0 < 0) t0 = 0;
    if (t0 >= t1) return;
    if (g.S[axis] < 6)
        launchDependent(boundaryKernel<real>, blocksFor(t1 - t0), kThreads, 0, st, g, axis, g.dim + 2, methods[axis][0],
                        methods[axis][1], state, t0, t1);
    else
        launchDependent(ghostAxisKernel<real>, blocksFor(4 * (t1 - t0)), kThreads, 0, st, g, axis, g.dim + 2,
                        methods[axis][0], methods[axis][1], state, t0, t1);
}

int boundaryLaunches(const Grid& g) {
    for (int a = 0; a < g.dim; ++a)
        if (g.S[a] < 6) return g.dim;
    return 1;
}

template <typename real>
void launchBoundary(const Grid& g, const int methods[3][2], real* state, cudaStream_t st) {
    if (boundaryLaunches(g) > 1 || g.S[0] < 6) {   // an axis whose fill order shows: axis by axis
        for (int axis = 0; axis < g.dim; ++axis) launchBoundaryAxis<real>(g, methods, state, st, axis, 0, -1);
        return;
    }
    Methods bc;
    std::memcpy(bc.m, methods, sizeof bc.m);
    const long long n0 = 4ll * g.S[1] * g.S[2], n1 = g.dim > 1 ? 4ll * (g.S[0] - 4) * g.S[2] : 0,
                    n2 = g.dim > 2 ? 4ll * (g.S[0] - 4) * (g.S[1] - 4) : 0, n = n0 + n1 + n2;
    launchDependent(ghostKernel<real>, blocksFor(n), kThreads, 0, st, g, g.dim + 2, bc, state, n0, n1, n);
}

template <typename real>
void launchDerivCombine(const Grid& g, const Phys<real>& ph, const real* flux, const CombinePlan<real>& plan,
                        const StepConst<real>* sc, cudaStream_t st, long long c0, long long c1) {
    if (c1 < 0 || c1 > g.V) c1 = g.V;
    if (c0 < 0) c0 = 0;
    if (c0 >= c1) return;
    const unsigned b = blocksFor(c1 - c0);
#define L(DD, P) launchDependent(derivCombineKernel<real, DD, P>, b, kThreads, 0, st, g, ph, flux, plan, sc, c0, c1)
    if (plan.alphaAfter >= 0) {
        if (g.dim == 1) L(1, true);
        else if (g.dim == 2) L(2, true);
        else L(3, true);
    } else {
        if (g.dim == 1) L(1, false);
        else if (g.dim == 2) L(2, false);
        else L(3, false);
    }
#undef L
}

template <typename real>
void launchAlphaOnly(const Grid& g, int integrator, real* state, const StepConst<real>* sc, cudaStream_t st) {
    long long n = g.V * (g.dim + 2);
    launchDependent(alphaOnlyKernel<real>, blocksFor(n), kThreads, 0, st, n, integrator, state, sc);
}

template <typename real>
void launchZeroAdd(const Grid& g, real* state, const StepConst<real>* sc, cudaStream_t st) {
    long long n = g.V * (g.dim + 2);
    launchDependent(zeroAddKernel<real>, blocksFor(n), kThreads, 0, st, n, state, sc);
}

template <typename real>
void launchFixedDt(const Phys<real>& ph, int integrator, double fixedDt, StepConst<real>* sc, cudaStream_t st) {
    launchDependent(fixedDtKernel<real>, 1, 32, 0, st, ph, integrator, fixedDt, sc);
}

#define INST(real)                                                                                              \
    template void launchBoundary<real>(const Grid&, const int[3][2], real*, cudaStream_t);                      \
    template void launchBoundaryAxis<real>(const Grid&, const int[3][2], real*, cudaStream_t, int, long long,   \
                                           long long);                                                          \
    template void launchDerivCombine<real>(const Grid&, const Phys<real>&, const real*, const CombinePlan<real>&, \
                                           const StepConst<real>*, cudaStream_t, long long, long long);         \
    template void launchAlphaOnly<real>(const Grid&, int, real*, const StepConst<real>*, cudaStream_t);         \
    template void launchZeroAdd<real>(const Grid&, real*, const StepConst<real>*, cudaStream_t);                \
    template void launchFixedDt<real>(const Phys<real>&, int, double, StepConst<real>*, cudaStream_t);
INST(double)
INST(float)
#undef INST

}  // namespace hgpu
