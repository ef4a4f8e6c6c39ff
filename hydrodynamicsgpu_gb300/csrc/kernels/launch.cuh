// launch.cuh -- kernel launches that overlap the start of one kernel with the end of the
// kernel before it in the stream (programmatic dependent launch).
//
// A step is a chain of 10 to 200 kernels, each reading what the one before wrote.  Launched
// plainly, a kernel starts after the previous grid has drained; here it is launched with
// programmatic stream serialization, so its blocks take their places as soon as every block
// of the previous grid is resident or done, and each kernel begins with dependentLaunch():
// let the next grid start in turn, then wait until the previous grid has completed and its
// writes are visible.  Nothing is read or written before that wait, so the order of memory
// operations is that of plain launches.
//
// What keeps the compiler to that order: the wait is a volatile asm with a "memory" clobber,
// which binds every access to memory that may have other names.  A pointer parameter that is
// `__restrict__` is taken to have none, and one that is also `const` lets its loads be issued as
// read-only for the kernel's whole life (ld.global.nc), which starts before the wait while
// earlier kernels still write.  So these kernels declare `__restrict__` only what they write
// and do not read, and the tables that the host fills when a batch is made.  It costs nothing
// measurable: with `const __restrict__` inputs the steps of 2048^2, 1024^2, 160x144x136 and of
// the 1D shock tube took the same within 0.2 %.
#pragma once
#include <cuda_runtime.h>

namespace hgpu {

__device__ __forceinline__ void dependentLaunch() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// kernel<<<grid, block, smem, st>>>(args...), with that attribute while a step is captured
// into a graph, and for grids of at least four blocks per SM (152); every kernel launched
// this way calls dependentLaunch() first.  Launched directly (the adjoint, update_host) the
// attribute costs the host more than it gives a small grid: a 64 x 500 gradient of 20
// RungeKutta4 steps took 20.0 ms with it and 14.0 without, a 512^2 one of 20 RungeKutta2
// steps 23.8 and 24.6.
template <typename... P, typename... A>
inline void launchDependent(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(st, &capture);
    if (capture == cudaStreamCaptureStatusNone && (size_t)grid.x * grid.y * grid.z < 4 * 152) {
        kernel<<<grid, block, smem, st>>>(static_cast<P>(args)...);
        return;
    }
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace hgpu
