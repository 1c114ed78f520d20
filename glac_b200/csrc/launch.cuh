// Launches that may start while the kernel before them on the stream drains.
//
// A step of a small lattice is a chain of kernels of 8-10 us, of which 2-3 us
// are the gap between one kernel's last block and the next one's first load.  A
// chained launch (programmatic dependent launch) goes ahead once every block of
// the kernel before has called chain_release or ended; its blocks then wait in
// chain_wait until that kernel has ended and its writes are visible.  A kernel
// launched this way calls chain_wait before its first access to anything that
// an earlier kernel writes.  Whatever is launched otherwise waits for the whole
// chain.  Flow stages, sub-sweeps and the measurement's parts release late, before
// their last arithmetic: released at their start, the waiting blocks of the next
// kernel crowd onto the SMs that have room and leave it unbalanced (Metropolis sweep
// of 12^3 x 24 in FP32: 177 us, against 132 without chaining).  The trainer's two
// kernels release at their start: their blocks all fit beside one another, and the
// gradient's fetch its rows before they wait.  Combinations and final sums, which are
// short, never release; their end does.
#pragma once

#include <cuda_runtime.h>

namespace glac {

__device__ __forceinline__ void chain_wait() { cudaGridDependencySynchronize(); }
__device__ __forceinline__ void chain_release() { cudaTriggerProgrammaticLaunchCompletion(); }

// `shared`: dynamic shared memory of a block in bytes
template <typename... Params, typename... Args>
void launch_chained_shared(void (*kernel)(Params...), unsigned grid, unsigned threads, size_t shared, cudaStream_t st,
                           Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = shared;
    cfg.stream = st;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}
template <typename... Params, typename... Args>
void launch_chained(void (*kernel)(Params...), unsigned grid, unsigned threads, cudaStream_t st, Args... args) {
    launch_chained_shared(kernel, grid, threads, 0, st, args...);
}

}  // namespace glac
