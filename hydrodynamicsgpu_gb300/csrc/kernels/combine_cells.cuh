// combine_cells.cuh -- per-cell bodies of the ghost fill, flux divergence + RK combine
// and timestep finalisation, shared by combine.cu and the batched kernels (batch.cu).
#pragma once
#include "kernels.h"

namespace hgpu {

// ---------------- tableaus: include/HydroGPU/Integrator/RungeKutta.h:129-294 ----------------
#define HGPU_TABLE_A                                                                                         \
    {{{1}},                                                                                                  \
     {{1, 0}, {1, 0}},                                                                                       \
     {{1, 0}, {1, 0}},                                                                                       \
     {{1, 0}, {1, 0}},                                                                                       \
     {{1, 0, 0}, {1, 0, 0}, {1, 0, 0}},                                                                      \
     {{1, 0, 0, 0}, {1, 0, 0, 0}, {1, 0, 0, 0}, {1, 0, 0, 0}},                                               \
     {{1, 0, 0, 0}, {1, 0, 0, 0}, {1, 0, 0, 0}, {1, 0, 0, 0}},                                               \
     {{1, 0}, {.5, .5}},                                                                                     \
     {{1, 0}, {1, 0}},                                                                                       \
     {{1, 0, 0}, {3. / 4., 1. / 4., 0}, {1. / 3., 2. / 3., 0}},                                              \
     {{1, 0, 0, 0}, {649. / 1600., 951. / 1600., 0, 0},                                                      \
      {53989. / 2500000., 4806213. / 20000000., 23619. / 32000., 0},                                         \
      {1. / 5., 6127. / 30000., 7873. / 30000., 1. / 3.}},                                                   \
     {{1, 0, 0, 0}, {1, 0, 0, 0}, {1, 0, 0, 0}, {-1. / 3., 1. / 3., 2. / 3., 1. / 3.}}}
#define HGPU_TABLE_B                                                                                         \
    {{{1}},                                                                                                  \
     {{.5, 0}, {0, 1}},                                                                                      \
     {{1, 0}, {.5, .5}},                                                                                     \
     {{2. / 3., 0}, {1. / 4., 3. / 4.}},                                                                     \
     {{.5, 0, 0}, {-1, 2, 0}, {1. / 6., 2. / 6., 1. / 6.}},                                                  \
     {{.5, 0, 0, 0}, {0, .5, 0, 0}, {0, 0, 1, 0}, {1. / 6., 2. / 6., 2. / 6., 1. / 6.}},                     \
     {{1. / 3., 0, 0, 0}, {-1. / 3., 0, 0, 0}, {1, -1, 1, 0}, {1. / 8., 3. / 8., 3. / 8., 1. / 8.}},         \
     {{1, 0}, {0, .5}},                                                                                      \
     {{-20, 0}, {41. / 40., -1. / 40.}},                                                                     \
     {{1, 0, 0}, {0, 1. / 4., 0}, {0, 0, 2. / 3.}},                                                          \
     {{.5, 0, 0, 0}, {-10890423. / 25193600., 5000. / 7873, 0, 0},                                           \
      {-102261. / 5000000., -5121. / 20000., 7873. / 10000., 0}, {1. / 10., 1. / 6., 0, 1. / 6.}},          \
     {{.5, 0, 0, 0}, {0, .5, 0, 0}, {0, 0, 1, 0}, {0, 0, 0, 1. / 6.}}}
#define HGPU_TABLE_ORDER {1, 2, 2, 2, 3, 4, 4, 2, 2, 3, 4, 4}

namespace {
__constant__ double cA[12][4][4] = HGPU_TABLE_A;
__constant__ double cB[12][4][4] = HGPU_TABLE_B;
__constant__ int cOrder[12] = HGPU_TABLE_ORDER;
__device__ __forceinline__ int kOrderDev(int i) { return cOrder[i]; }
__device__ __forceinline__ double kAlphaDev(int i, int m, int k) { return cA[i][m][k]; }
__device__ __forceinline__ double kBetaDev(int i, int m, int k) { return cB[i][m][k]; }
}  // namespace

// The boundary methods of a problem ([axis][min, max] of HGPU_BOUNDARY_*).
struct Methods { int m[3][2]; };

// The coordinate along `axis` that the ghost fill copies coordinate k from (k itself for an
// interior coordinate or a side without a method), for an axis of S >= 6 cells, where no
// source is a ghost; `flip`: the copy reflects the normal momentum (MIRROR).
__device__ __forceinline__ int ghostSource(int k, int S, int mMin, int mMax, bool& flip) {
    flip = false;
    const bool low = k < 2, high = k >= S - 2;
    const int m = low ? mMin : mMax;
    if (!(low || high) || m < 0) return k;
    if (m == 0) return low ? k + S - 4 : k - (S - 4);             // periodic
    flip = m == 1;
    if (m == 1) return low ? 3 - k : 2 * S - 5 - k;                // mirror
    return low ? 2 : S - 3;                                        // free flow
}

// The ghost fill of every axis for one ghost cell: the axes' fills run one after another in
// the reference (Solver.cpp:448-464), so a cell that is a ghost of several axes ends up with
// the cell that all its coordinates map to, every MIRROR on the way flipping its axis's
// momentum.  That source is no ghost of a filled side, so no cell of the pass reads what
// another writes.  Axes of S >= 6 cells (Grid::dim of them).
template <typename real>
__device__ __forceinline__ void ghostCell(const Grid& g, int N, const Methods& bc, real* __restrict__ state, int x,
                                          int y, int z) {
    bool f0 = false, f1 = false, f2 = false;
    const int sx = ghostSource(x, g.S[0], bc.m[0][0], bc.m[0][1], f0);
    const int sy = g.dim > 1 ? ghostSource(y, g.S[1], bc.m[1][0], bc.m[1][1], f1) : 0;
    const int sz = g.dim > 2 ? ghostSource(z, g.S[2], bc.m[2][0], bc.m[2][1], f2) : 0;
    const long long c = x + (long long)g.S[0] * (y + (long long)g.S[1] * z);
    const long long s = sx + (long long)g.S[0] * (sy + (long long)g.S[1] * sz);
    if (s == c || !cellOk(g, c) || !cellOk(g, s)) return;
    const bool flip[3] = {f0, f1, f2};
    real v[5];
#pragma unroll
    for (int j = 0; j < 5; ++j)
        if (j < N) v[j] = state[(long long)N * s + j];
#pragma unroll
    for (int j = 0; j < 5; ++j)
        if (j < N) state[(long long)N * c + j] = j >= 1 && j <= 3 && j <= g.dim && flip[j - 1] ? -v[j] : v[j];
}

// One ghost line of the boundary pass along `axis` (thread = transverse line t):
// every state, min side then max side.  In 1D the reference's Mirror/Reflect/FreeFlow
// kernels have no range guard and only work-item 0 addresses the buffer; that
// work-item is what runs here.
template <typename real>
__device__ __forceinline__ void boundaryLine(const Grid& g, int axis, int N, int mMin, int mMax,
                                             real* __restrict__ state, long long t) {
    int A = axis == 0 ? 1 : 0, B = axis == 2 ? 1 : 2;   // transverse axes
    long long nA = g.S[A], nB = g.S[B];
    if (g.dim == 1) { nA = 1; nB = 1; }
    if (t >= nA * nB) return;
    int a = (int)(t % nA), b = (int)(t / nA);
    int c[3];
    c[A] = a; c[B] = b; c[axis] = 0;
    long long base = c[0] + (long long)g.S[0] * (c[1] + (long long)g.S[1] * c[2]);
    long long st = g.step[axis];
    int S = g.S[axis];
    if (!cellOk(g, base) || !cellOk(g, base + (long long)(S - 1) * st)) return;
    for (int j = 0; j < N; ++j) {
        real* p = state + j;
#define AT(k) p[(long long)N * (base + (long long)(k) * st)]
        for (int side = 0; side < 2; ++side) {
            int m = side == 0 ? mMin : mMax;
            if (m < 0) continue;
            // Euler::stateGetBoundaryKernelForBoundaryMethod: MIRROR reflects the normal momentum
            int kern = m == 0 ? 0 : (m == 1 ? ((axis + 1 == j) ? 2 : 1) : 3);
            if (kern == 0) {                                  // periodic
                if (side == 0) { AT(0) = AT(S - 4); AT(1) = AT(S - 3); }
                else { AT(S - 2) = AT(2); AT(S - 1) = AT(3); }
            } else if (kern == 1) {                           // mirror
                if (side == 0) { AT(0) = AT(3); AT(1) = AT(2); }
                else { AT(S - 1) = AT(S - 4); AT(S - 2) = AT(S - 3); }
            } else if (kern == 2) {                           // reflect
                if (side == 0) { AT(0) = -AT(3); AT(1) = -AT(2); }
                else { AT(S - 1) = -AT(S - 4); AT(S - 2) = -AT(S - 3); }
            } else {                                          // free flow
                if (side == 0) { real v = AT(2); AT(1) = v; AT(0) = v; }
                else { real v = AT(S - 3); AT(S - 2) = v; AT(S - 1) = v; }
            }
        }
#undef AT
    }
}

// x * y for an x that is often +-0 (flux differences of piecewise-constant states):
// the signed zero from the bit patterns when x is zero and y finite (what the product
// gives), otherwise mulI, whose zero operands take an out-of-line FP64 call
__device__ __forceinline__ double mulZ(double x, double y) {
    if (isZeroBits(x) && finiteD(y)) return fromBits((bitsOf(x) ^ bitsOf(y)) & (long long)0x8000000000000000ULL);
    return mulI(x, y);
}
__device__ __forceinline__ float mulZ(float x, float y) { return x * y; }

// FLATD: the deriv's products by mulZ (the batched kernels, whose states are mostly flat).
// POST: the new state (the row that slot 0 gets) goes through the self-gravity pass with a
// zero potential, of the tableau plan.alphaAfter, before it is stored.
template <typename real, int D, bool FLATD = false, bool POST = false>
__device__ __forceinline__ void combinePlanCell(const real* d, const CombinePlan<real>& plan,
                                                const StepConst<real>& sc, long long c, long long off);
template <typename real>
__device__ __forceinline__ real alphaOnlyElem(int integ, real u0, const StepConst<real>& sc);

// t = df / dx, without a branch each where the warp's differences are ordinary numbers
template <int N>
__device__ __forceinline__ void quotientsBy(const double* df, const Divisor<double>& dx, double* t) {
    if (warpAll(allInWindow<N>(df) & inWindow(dx.b))) {
#pragma unroll
        for (int j = 0; j < N; ++j) t[j] = quotPlain(df[j], dx);
        return;
    }
#pragma unroll
    for (int j = 0; j < N; ++j) t[j] = quotBy(df[j], dx);
}
template <int N>
__device__ __forceinline__ void quotientsBy(const float* df, const Divisor<float>& dx, float* t) {
#pragma unroll
    for (int j = 0; j < N; ++j) t[j] = df[j] / dx.b;
}

// Flux divergence and Runge-Kutta combine of one cell (res/CalcFluxDeriv.cl:7-44 and
// the multAdd chain).  `off` is the cell offset of this grid inside the slot arrays
// (0 for a single problem; the problem's first cell in a batch).
// deltaFlux / dx with dx's reciprocal bits from the host (quotBy): KH 2048^2 FP64 286 -> 237 us
// a launch against the x quotients by Markstein's two FMAs on the FP64 unit and the rest by
// divI; 216 us with the differences loaded together (below).
template <typename real, int D, bool FLATD = false, bool POST = false>
__device__ __forceinline__ void derivCombineCell(const Grid& g, const Phys<real>& ph, const real* __restrict__ flux,
                                                 const CombinePlan<real>& plan, const StepConst<real>& sc,
                                                 long long c, int x, int y, int z, long long off) {
    const int N = D + 2;
    real d[N];
    if (!cellOk(g, c)) return;
    // calcFluxDeriv: interior cells only, deriv[j] -= (F[i+1] - F[i]) / dx, sides ascending, from 0
    if (inRange(g, x, y, z, 2, 2)) {
#pragma unroll
        for (int side = 0; side < D; ++side)
            if (!cellOk(g, c + g.step[side])) return;
        // every flux difference first, the loads in flight together (KH 2048^2 FP32 104 -> 71 us
        // a launch, FP64 235 -> 216); 3D FP64 axis by axis (its registers spill otherwise)
        constexpr bool ahead = D < 3 || sizeof(real) == 4;
        real df[D][N], t[N];
        auto difference = [&](int side) {
#pragma unroll
            for (int j = 0; j < N; ++j) {
                const real* f = flux + ((long long)side * N + j) * g.V + c;
                df[side][j] = f[g.step[side]] - f[0];
            }
        };
        if (ahead) {
#pragma unroll
            for (int side = 0; side < D; ++side) difference(side);
        }
#pragma unroll
        for (int side = 0; side < D; ++side) {
            if (!ahead) difference(side);
            quotientsBy<N>(df[side], ph.dxDiv[side], t);
#pragma unroll
            for (int j = 0; j < N; ++j) d[j] = side == 0 ? zfix(-t[j]) : d[j] - t[j];
        }
    } else {
#pragma unroll
        for (int j = 0; j < N; ++j) d[j] = (real)0.;
    }
    combinePlanCell<real, D, FLATD, POST>(d, plan, sc, c, off);
}

// The integrator's use of one cell's deriv d: ForwardEuler's state += deriv * dt, or
// this stage's column of the Runge-Kutta rows (see combine.cu).
template <typename real, int D, bool FLATD, bool POST>
__device__ __forceinline__ void combinePlanCell(const real* d, const CombinePlan<real>& plan,
                                                const StepConst<real>& sc, long long c, long long off) {
    const int N = D + 2;
    if (plan.fe) {                                            // ForwardEuler::integrate: state += deriv * dt
        real dt = sc.dt;
        real* s = plan.slot[0] + (long long)N * (off + c);
#pragma unroll
        for (int j = 0; j < N; ++j) s[j] = s[j] + (FLATD ? mulZ(d[j], dt) : mulI(d[j], dt));
        return;
    }
    real u[N];
    const real* in = plan.slot[plan.in] + (long long)N * (off + c);
#pragma unroll
    for (int j = 0; j < N; ++j) u[j] = in[j];
    for (int o = 0; o < plan.nops; ++o) {
        const CombineOp<real>& op = plan.ops[o];
        real v[N];
        bool empty = op.prior < 0;
        if (!empty) {
            const real* p = plan.slot[op.prior] + (long long)N * (off + c);
#pragma unroll
            for (int j = 0; j < N; ++j) v[j] = op.priorAlias ? zfix(p[j]) : p[j];
        }
        if (op.hasAlpha) {
#pragma unroll
            for (int j = 0; j < N; ++j) {
                real t = op.alphaIsOne ? u[j] : mulI(u[j], op.alpha);
                v[j] = empty ? zfix(t) : v[j] + t;
            }
            empty = false;
        }
        if (op.hasBeta) {
            real cf = sc.coef[op.brow][op.bcol];
#pragma unroll
            for (int j = 0; j < N; ++j) {
                real t = FLATD ? mulZ(d[j], cf) : mulI(d[j], cf);
                v[j] = empty ? zfix(t) : v[j] + t;
            }
        }
        real* o_ = plan.slot[op.out] + (long long)N * (off + c);
        if (POST && op.out == 0) {
#pragma unroll
            for (int j = 0; j < N; ++j) v[j] = alphaOnlyElem<real>(plan.alphaAfter, v[j], sc);
        }
#pragma unroll
        for (int j = 0; j < N; ++j) o_[j] = v[j];
    }
}

// dt of one problem from its reduced minimum: `dt * app->cfl` (Solver.cpp:515) or the
// fixed dt; then dt/dx and beta*dt for the step; re-arms the accumulator.
template <typename real>
__device__ __forceinline__ void finalizeOne(const Phys<real>& ph, int integ, int useFixed, double fixedDt,
                                            unsigned long long* acc, unsigned long long accInit, StepConst<real>* sc) {
    real dt;
    if (useFixed) dt = (real)fixedDt;
    else {
        real mn = (real)bitsToDouble(*acc, sizeof(real) == 4);
        dt = (real)(mn * (real)ph.cfl);
        *acc = accInit;
    }
    sc->dt = dt;
    sc->dt_f64 = (double)dt;
    for (int s = 0; s < 3; ++s) sc->dt_dx[s] = dt / ph.dx[s];
    for (int m = 0; m < 4; ++m)
        for (int k = 0; k < 4; ++k) sc->coef[m][k] = (real)kBetaDev(integ, m, k) * dt;
}

// r + t without the FP64 unit where that is exact on the bits: t a zero (r is never -0
// here), or r and t the same normal number whose double is normal
static __device__ __noinline__ double addNative(double r, double t) { return r + t; }
__device__ __forceinline__ double addEqual(double r, double t) {
    if (isZeroBits(t)) return r;
    const unsigned e = (unsigned)__double2hiint(r) & 0x7FF00000u;
    if (bitsOf(r) == bitsOf(t) && e - 0x00100000u < 0x7FD00000u)
        return __hiloint2double(__double2hiint(r) + 0x00100000, __double2loint(r));
    return addNative(r, t);
}
__device__ __forceinline__ float addEqual(float r, float t) { return r + t; }

// The self-gravity pass with a zero potential and a Runge-Kutta integrator, one element:
// every deriv is +0, so the stages are alpha combinations of u0 (the 0 * beta dt terms are
// zeros and change no sum that starts from +0; with a dt that is not finite they are NaN
// and the terms are kept).  Row by row as the integrator adds them; two equal halves
// (RungeKutta2TVD) and zeros need no addition.
template <typename real>
__device__ __forceinline__ real alphaOnlyElem(int integ, real u0, const StepConst<real>& sc) {
    const int order = kOrderDev(integ);
    const bool keepZeros = !finiteBits(sc.dt);
    real u[5];
    u[0] = u0;
    real out = u0;
#pragma unroll
    for (int s = 1; s <= 4; ++s) {
        if (s > order) break;
        real r = (real)0;
#pragma unroll
        for (int k = 0; k < s; ++k) {
            const double a = kAlphaDev(integ, s - 1, k);
            // (the tests on the bits: compares of doubles issue to the FP64 unit)
            if (bitsOf(a) != 0) {
                const real t = bitsOf(a) == 0x3FF0000000000000LL   ? u[k]
                               : bitsOf(a) == 0x3FE0000000000000LL ? halfOf(u[k])
                                                                   : mulZ(u[k], (real)a);
                r = k == 0 ? zfix(t) : addEqual(r, t);
            }
            if (keepZeros && bitsOf(kBetaDev(integ, s - 1, k)) != 0) r = r + (real)0. * sc.coef[s - 1][k];
        }
        out = u[s] = r;
    }
    return out;
}

}  // namespace hgpu
