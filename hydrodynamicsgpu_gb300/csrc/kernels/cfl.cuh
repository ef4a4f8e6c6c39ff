// cfl.cuh -- the CFL timestep of one problem from the largest wave speed difference of
// each axis.
//
// The reference takes the minimum over cells and axes of dx / speed(cell, axis)
// (res/Roe.cl:4-65, res/EulerHLLC.cl:135-168, findMinTimestep Solver.cpp:466-516), a
// quotient per cell and axis.  Rounding is monotone, so the smallest quotient of an axis
// is the quotient of its largest speed: the kernels reduce the speeds (IEEE bits of
// non-negative values order as integers) and the last block to finish forms one quotient
// per axis, the timestep, dt / dx and beta * dt, and clears the accumulator for the next
// step.  KH 2048^2: FP64 60 us and FP32 37 us for the two launches this replaces (a
// quotient per cell and axis, then one thread for the step's constants: 90 + 4 and
// 68 + 4 us).
#pragma once
#include "combine_cells.cuh"
#include "kernels.h"

namespace hgpu {

// max over the block of each axis's speed bits, merged into acc (all threads call)
template <int D>
__device__ __forceinline__ void blockMaxSpeeds(unsigned long long (&s)[D], CflAcc* acc) {
    __shared__ unsigned long long warpMax[D][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int a = 0; a < D; ++a) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long w = __shfl_xor_sync(0xffffffffu, s[a], o);
            s[a] = w > s[a] ? w : s[a];
        }
        if (lane == 0) warpMax[a][warp] = s[a];
    }
    __syncthreads();
    if (threadIdx.x < D) {
        unsigned long long m = 0;
        for (int w = 0; w < nwarps; ++w) m = warpMax[threadIdx.x][w] > m ? warpMax[threadIdx.x][w] : m;
        if (m) atomicMax(&acc->speed[threadIdx.x], m);
    }
}

// The end of a CFL kernel, all threads of the block: the last block of the grid turns the
// maxima into dt = cfl * min (starting from accInit, the bits of the largest value the
// reference's buffer can hold) and the step's constants.  ROE: dx / (speed + 1e-9) in
// double, else dx / speed.  A speed is never NaN and dx is positive, so a cell's quotient is
// NaN where both are infinite, and then that of the axis's largest speed is too: it sets the
// health bit.
template <typename real, int D, bool ROE>
__device__ __forceinline__ void finishCfl(const Phys<real>& ph, int integ, unsigned long long accInit, CflAcc* acc,
                                          StepConst<real>* sc, unsigned* health) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&acc->done, 1u) == gridDim.x * gridDim.y * gridDim.z - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    unsigned long long best = accInit;
    bool nan = false;
#pragma unroll
    for (int a = 0; a < D; ++a) {
        const unsigned long long b = __ldcg(&acc->speed[a]);
        const real speed = (real)bitsToDouble(b, sizeof(real) == 4);
        const real q = ROE ? (real)divI((double)ph.dx[a], (double)speed + 1e-9) : divI(ph.dx[a], speed);
        best = realBits(q) < best ? realBits(q) : best;
        nan |= isNaNBits(q);
    }
    if (nan && threadIdx.x == 0) atomicOr(health, HEALTH_NONFINITE_DT);
    const real dt = (real)((real)bitsToDouble(best, sizeof(real) == 4) * (real)ph.cfl);   // Solver.cpp:515
    __syncthreads();                                       // every thread has read the maxima
    for (int i = threadIdx.x; i < 24; i += blockDim.x) {
        if (i < 16) sc->coef[i >> 2][i & 3] = (real)kBetaDev(integ, i >> 2, i & 3) * dt;
        else if (i < 19) sc->dt_dx[i - 16] = dt / ph.dx[i - 16];
        else if (i == 19) sc->dt = dt;
        else if (i == 20) sc->dt_f64 = (double)dt;
        else if (i == 21) acc->done = 0;
        if (i >= 21) acc->speed[i - 21] = 0;
    }
}

}  // namespace hgpu
