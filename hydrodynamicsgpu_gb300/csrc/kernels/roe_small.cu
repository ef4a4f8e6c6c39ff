// roe_small.cu -- EulerRoe steps of small grids in few launches (sm_103a).
//
// On a small grid a step's kernels are all latency: a launch holds a few warps on a few
// SMs, and the step pays its chain of launches (12 for a 1D RungeKutta2 step, 39 us at 1028
// cells against 28 here, of which the FP64 unit needs 0.3 us).  Here the step is one prologue kernel, one
// kernel a stage and, for ForwardEuler, one to finish; a block takes a small tile, so that
// a grid of a thousand cells is spread over tens of SMs, and recomputes the faces that its
// neighbours also need instead of waiting for them:
//   * prologue: the ghost fill, the Roe eigenbasis of the tile's faces and of the face past
//     its end on each axis, the wave speeds and, in the last block, the timestep;
//   * stage: Delta-q-tilde of the tile's faces and one more before and two after them, their
//     limited flux, the divergence and the integrator's combine, through shared memory.
// Every value is formed by the operations of the kernels for large grids in their order
// (res/EulerRoe.cl:18-271, res/Roe.cl:4-320, res/CalcFluxDeriv.cl:7-44), so the bits are the
// same.  One thread a face in every phase: 1D tiles of 29 cells and 32 threads (32 faces of
// Delta-q-tilde), 2D tiles of 8 x 8 and 192 (88 faces an axis, a warp never mixes axes); a
// 2D tile forms 1.4x the Delta-q-tilde and 1.13x the fluxes it owns, which the idle SMs of a
// small grid take and a large grid does not (the rule is in Roe::smallGrid, solver.cu).
#include <cstring>
#include <limits>

#include "../../../include/hgpu/hgpu.h"
#include "cfl.cuh"
#include "kernels.h"
#include "launch.cuh"
#include "roe_cells.cuh"

namespace hgpu {
namespace {

template <int D> struct SmallTile;
template <> struct SmallTile<1> { enum { X = 29, Y = 1, G = 32, THREADS = 32 }; };
template <> struct SmallTile<2> { enum { X = 8, Y = 8, G = 96, THREADS = 192 }; };

// the i-th face of `side` among those of the tile's lines that start `before` faces before
// the tile and hold `n` of them: its cell coordinates relative to the tile; false past the end
template <int D>
__device__ __forceinline__ bool smallFace(int side, int i, int before, int extra, int& rx, int& ry) {
    typedef SmallTile<D> T;
    const int nx = side == 0 ? T::X + extra : T::X, ny = side == 0 ? T::Y : T::Y + extra;
    if (i >= nx * ny) return false;
    rx = i % nx - (side == 0 ? before : 0);
    ry = i / nx - (side == 0 ? 0 : before);
    return true;
}

template <typename real, int D>
__global__ void __launch_bounds__(SmallTile<D>::THREADS) smallPrologueKernel(Grid g, Phys<real> ph, Methods bc,
                                                                          real* state, real* __restrict__ basis,
                                                                          int integ, unsigned long long accInit,
                                                                          CflAcc* acc, StepConst<real>* sc,
                                                                          unsigned* health) {
    dependentLaunch();
    typedef SmallTile<D> T;
    typedef RoeRec<D> R_;
    constexpr int N = D + 2, NB = R_::NB, HX = T::X + 2, HY = D > 1 ? T::Y + 2 : 1, oy = D > 1 ? 1 : 0;
    constexpr int FX = T::X + 1, FY = D > 1 ? T::Y + 1 : 1;
    __shared__ RoePrim<real, D> prim[HX * HY];
    __shared__ real lamMin[D][FX * FY], lamMax[D][FX * FY];
    const int x0 = blockIdx.x * T::X, y0 = blockIdx.y * T::Y;
    // the tile's cells and one around them, ghosts read from where the ghost fill copies
    // them; the tile's own ghosts are written (no source is one of them)
    for (int i = threadIdx.x; i < HX * HY; i += T::THREADS) {
        const int x = x0 - 1 + i % HX, y = y0 - oy + i / HX;
        if (x < 0 || x >= g.S[0] || y < 0 || y >= g.S[1]) continue;
        bool fx = false, fy = false;
        const int sx = ghostSource(x, g.S[0], bc.m[0][0], bc.m[0][1], fx);
        const int sy = D > 1 ? ghostSource(y, g.S[1], bc.m[1][0], bc.m[1][1], fy) : y;
        const long long c = x + (long long)g.S[0] * y, src = sx + (long long)g.S[0] * sy;
        if (!cellOk(g, c) || !cellOk(g, src)) continue;
        real s[N];
        loadState<real, D>(state, src, s);
        if (fx) s[1] = -s[1];
        if (D > 1 && fy) s[2] = -s[2];
        const bool own = i % HX >= 1 && i % HX <= T::X && (D == 1 || (i / HX >= 1 && i / HX <= T::Y));
        if (own && src != c) {
#pragma unroll
            for (int j = 0; j < N; ++j) state[(long long)N * c + j] = s[j];
        }
        roePrim<real, D>(s, ph.gamma, prim[i]);
    }
    __syncthreads();
    auto face = [&](auto sideTag) {
        constexpr int SIDE = decltype(sideTag)::value;
        int rx, ry;
        if (!smallFace<D>(SIDE, threadIdx.x % T::G, 0, 1, rx, ry)) return;
        const int x = x0 + rx, y = y0 + ry;
        if (x >= g.S[0] || y >= g.S[1] || !roeFace(g, SIDE, x, y, 0, 2, 1)) return;
        const int self = (ry + oy) * HX + rx + 1;
        real rec[NB];
        roeBasisFromPrim<real, D, SIDE>(prim[self - (SIDE == 0 ? 1 : HX)], prim[self], ph.gamma, rec);
        lamMin[SIDE][ry * FX + rx] = rec[R_::LAM0];
        lamMax[SIDE][ry * FX + rx] = rec[R_::LAME];
        const long long c = x + (long long)g.S[0] * y;
        if (rx < T::X && ry < T::Y && cellOk(g, c)) {
#pragma unroll
            for (int k = 0; k < NB; ++k) basis[((long long)SIDE * NB + k) * g.V + c] = rec[k];
        }
    };
    if (threadIdx.x < T::G) face(std::integral_constant<int, 0>());
    else face(std::integral_constant<int, (D > 1 ? 1 : 0)>());
    __syncthreads();
    unsigned long long s[D] = {};
    const int rx = threadIdx.x % T::X, ry = threadIdx.x / T::X;
    if (ry < T::Y && x0 + rx < g.S[0] && inRange(g, x0 + rx, y0 + ry, 0, 2, 2)) {
#pragma unroll
        for (int a = 0; a < D; ++a) {
            const int f = ry * FX + rx;
            s[a] = realBits((real)fabs(positivePart(lamMax[a][f]) - negativePart(lamMin[a][f + (a == 0 ? 1 : FX)])));
        }
    }
    blockMaxSpeeds<D>(s, acc);
    finishCfl<real, D, true>(ph, integ, accInit, acc, sc, health);
}

template <typename real, int D, int LIM, bool POST>
__global__ void __launch_bounds__(SmallTile<D>::THREADS) smallStageKernel(Grid g, Phys<real> ph, int lim,
                                                                       const StepConst<real>* sc,
                                                                       const real* basis,
                                                                       CombinePlan<real> plan) {
    dependentLaunch();
    typedef SmallTile<D> T;
    constexpr int N = D + 2, NB = RoeRec<D>::NB;
    // Delta-q-tilde lines start one face before the tile, flux lines at it
    constexpr int QX = T::X + 3, QN = D > 1 ? QX * (T::Y + 3) : QX, FX = T::X + 1, FN = D > 1 ? FX * (T::Y + 1) : FX;
    __shared__ real dq[D][N][QN], fl[D][N][FN];
    const int x0 = blockIdx.x * T::X, y0 = blockIdx.y * T::Y;
    const real* stage = plan.slot[plan.in];
    auto deltaQ = [&](auto sideTag) {
        constexpr int SIDE = decltype(sideTag)::value;
        int rx, ry;
        if (!smallFace<D>(SIDE, threadIdx.x % T::G, 1, 3, rx, ry)) return;
        const int x = x0 + rx, y = y0 + ry;
        real q[N];
#pragma unroll
        for (int j = 0; j < N; ++j) q[j] = (real)0;                  // faces the reference never writes
        if (x >= 0 && y >= 0 && x < g.S[0] && y < g.S[1] && roeFace(g, SIDE, x, y, 0, 2, 1)) {
            const long long c = x + (long long)g.S[0] * y;
            if (cellOk(g, c) && cellOk(g, c - g.step[SIDE])) {
                real sL[N], sR[N], rec[NB];
                loadState<real, D>(stage, c - g.step[SIDE], sL);
                loadState<real, D>(stage, c, sR);
#pragma unroll
                for (int k = 0; k < NB; ++k) rec[k] = basis[((long long)SIDE * NB + k) * g.V + c];
#pragma unroll
                for (int j = 0; j < N; ++j) sR[j] = sR[j] - sL[j];
                leftTransform<real, D, SIDE, true>(rec, sR, q);
            }
        }
        const int at = (SIDE == 0 ? ry : ry + 1) * QX + rx + (SIDE == 0 ? 1 : 0);
#pragma unroll
        for (int j = 0; j < N; ++j) dq[SIDE][j][at] = q[j];
    };
    auto flux = [&](auto sideTag) {
        constexpr int SIDE = decltype(sideTag)::value;
        int rx, ry;
        if (!smallFace<D>(SIDE, threadIdx.x % T::G, 0, 1, rx, ry)) return;
        const int x = x0 + rx, y = y0 + ry;
        if (x >= g.S[0] || y >= g.S[1] || !roeFace(g, SIDE, x, y, 0, 2, 1)) return;
        const long long c = x + (long long)g.S[0] * y;
        if (!cellOk(g, c) || !cellOk(g, c - g.step[SIDE])) return;
        constexpr int st = SIDE == 0 ? 1 : QX;
        const int at = (SIDE == 0 ? ry : ry + 1) * QX + rx + (SIDE == 0 ? 1 : 0);
        real sL[N], sR[N], rec[NB], qL[N], q[N], qR[N], F[N];
        loadState<real, D>(stage, c - g.step[SIDE], sL);
        loadState<real, D>(stage, c, sR);
#pragma unroll
        for (int k = 0; k < NB; ++k) rec[k] = basis[((long long)SIDE * NB + k) * g.V + c];
#pragma unroll
        for (int j = 0; j < N; ++j) {
            qL[j] = dq[SIDE][j][at - st];
            q[j] = dq[SIDE][j][at];
            qR[j] = dq[SIDE][j][at + st];
        }
        if constexpr (sizeof(real) == 8) {
            real corr[N];
            roeFluxCorrections<D, SIDE, LIM>(rec, qL, q, qR, sc->dt_dx[SIDE], lim, corr);
            roeFluxTransforms<D, SIDE>(rec, sL, sR, corr, F);
        } else {
            roeFlux<real, D, SIDE, LIM>(rec, sL, sR, qL, q, qR, sc->dt_dx[SIDE], lim, F);
        }
#pragma unroll
        for (int j = 0; j < N; ++j) fl[SIDE][j][ry * FX + rx] = F[j];
    };
    if (threadIdx.x < T::G) deltaQ(std::integral_constant<int, 0>());
    else deltaQ(std::integral_constant<int, (D > 1 ? 1 : 0)>());
    __syncthreads();
    if (threadIdx.x < T::G) flux(std::integral_constant<int, 0>());
    else flux(std::integral_constant<int, (D > 1 ? 1 : 0)>());
    __syncthreads();
    const int rx = threadIdx.x % T::X, ry = threadIdx.x / T::X, x = x0 + rx, y = y0 + ry;
    const long long c = x + (long long)g.S[0] * y;
    if (ry >= T::Y || x >= g.S[0] || y >= g.S[1] || !cellOk(g, c)) return;
    real d[N];
    const bool in = inRange(g, x, y, 0, 2, 2);
#pragma unroll
    for (int j = 0; j < N; ++j) {
        d[j] = (real)0;
        if (in) {
#pragma unroll
            for (int a = 0; a < D; ++a) {
                const real* f = fl[a][j] + ry * FX + rx;
                const real t = quotBy(f[a == 0 ? 1 : FX] - f[0], ph.dxDiv[a]);
                d[j] = a == 0 ? zfix(-t) : d[j] - t;
            }
        }
    }
    combinePlanCell<real, D, false, POST>(d, plan, *sc, c, 0);
}

// ForwardEuler's end (the self-gravity pass with a zero potential): the updated state out of
// `next`, ghosts from where the ghost fill copies them, + 0 * dt
template <typename real>
__global__ void __launch_bounds__(64) smallFinishKernel(Grid g, int N, Methods bc, const real* next,
                                                        real* state,
                                                        const StepConst<real>* sc) {
    dependentLaunch();
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= g.V) return;
    int x, y, z;
    cellCoords(g, c, x, y, z);
    bool fx = false, fy = false;
    const int sx = ghostSource(x, g.S[0], bc.m[0][0], bc.m[0][1], fx);
    const int sy = g.dim > 1 ? ghostSource(y, g.S[1], bc.m[1][0], bc.m[1][1], fy) : 0;
    const long long src = sx + (long long)g.S[0] * sy;
    if (!cellOk(g, src)) return;
    const real zero = (real)0. * sc->dt;
    for (int j = 0; j < N; ++j) {
        const real v = next[(long long)N * src + j];
        state[(long long)N * c + j] = ((j == 1 && fx) || (j == 2 && fy && g.dim > 1) ? -v : v) + zero;
    }
}

template <int D>
dim3 smallGridOf(const Grid& g) {
    typedef SmallTile<D> T;
    return dim3((unsigned)((g.S[0] + T::X - 1) / T::X), (unsigned)((g.S[1] + T::Y - 1) / T::Y));
}

template <typename real, int D, int LIM>
void smallStageLim(const Grid& g, const Phys<real>& ph, int lim, const StepConst<real>* sc, const real* basis,
                   const CombinePlan<real>& plan, cudaStream_t st) {
    const dim3 grid = smallGridOf<D>(g);
    constexpr int threads = SmallTile<D>::THREADS;
    if (plan.alphaAfter >= 0)
        launchDependent(smallStageKernel<real, D, LIM, true>, grid, threads, 0, st, g, ph, lim, sc, basis, plan);
    else launchDependent(smallStageKernel<real, D, LIM, false>, grid, threads, 0, st, g, ph, lim, sc, basis, plan);
}

}  // namespace

template <typename real>
void launchSmallPrologue(const Grid& g, const Phys<real>& ph, const int methods[3][2], real* state, real* basis,
                         int integrator, CflAcc* acc, StepConst<real>* sc, unsigned* health, cudaStream_t st) {
    const real top = std::numeric_limits<real>::infinity();
    unsigned long long accInit = 0;
    std::memcpy(&accInit, &top, sizeof top);
    Methods bc;
    std::memcpy(bc.m, methods, sizeof bc.m);
    if (g.dim == 1)
        launchDependent(smallPrologueKernel<real, 1>, smallGridOf<1>(g), SmallTile<1>::THREADS, 0, st, g, ph, bc, state,
                        basis, integrator, accInit, acc, sc, health);
    else
        launchDependent(smallPrologueKernel<real, 2>, smallGridOf<2>(g), SmallTile<2>::THREADS, 0, st, g, ph, bc, state,
                        basis, integrator, accInit, acc, sc, health);
}

template <typename real>
void launchSmallStage(const Grid& g, const Phys<real>& ph, int limiter, const StepConst<real>* sc, const real* basis,
                      const CombinePlan<real>& plan, cudaStream_t st) {
#define F(LL)                                                                                              \
    if (g.dim == 1) smallStageLim<real, 1, LL>(g, ph, limiter, sc, basis, plan, st);                       \
    else smallStageLim<real, 2, LL>(g, ph, limiter, sc, basis, plan, st)
    switch (limiter) {
    case HGPU_LIMITER_DONORCELL: F(HGPU_LIMITER_DONORCELL); break;
    case HGPU_LIMITER_LAXWENDROFF: F(HGPU_LIMITER_LAXWENDROFF); break;
    case HGPU_LIMITER_MINMOD: F(HGPU_LIMITER_MINMOD); break;
    case HGPU_LIMITER_VANLEER: F(HGPU_LIMITER_VANLEER); break;
    case HGPU_LIMITER_MONOTIZEDCENTRAL: F(HGPU_LIMITER_MONOTIZEDCENTRAL); break;
    case HGPU_LIMITER_SUPERBEE: F(HGPU_LIMITER_SUPERBEE); break;
    default: F(-1); break;
    }
#undef F
}

template <typename real>
void launchSmallFinish(const Grid& g, const int methods[3][2], const real* next, real* state, const StepConst<real>* sc,
                       cudaStream_t st) {
    Methods bc;
    std::memcpy(bc.m, methods, sizeof bc.m);
    launchDependent(smallFinishKernel<real>, (unsigned)((g.V + 63) / 64), 64, 0, st, g, g.dim + 2, bc, next, state, sc);
}

#define INST(real)                                                                                                   \
    template void launchSmallPrologue<real>(const Grid&, const Phys<real>&, const int[3][2], real*, real*, int,      \
                                            CflAcc*, StepConst<real>*, unsigned*, cudaStream_t);                     \
    template void launchSmallStage<real>(const Grid&, const Phys<real>&, int, const StepConst<real>*, const real*,   \
                                         const CombinePlan<real>&, cudaStream_t);                                    \
    template void launchSmallFinish<real>(const Grid&, const int[3][2], const real*, real*, const StepConst<real>*,  \
                                          cudaStream_t);
INST(double)
INST(float)
#undef INST

}  // namespace hgpu
