// pdl.cuh -- programmatic dependent launch: kernels that follow one another
// without the gap of a launch.  The FP32 step kernel waits for its predecessor
// at its start and then lets its successor launch (whose blocks take the places
// that finished blocks leave): 65^2 step 5.1 -> 4.8 us, 1025^2 30.4 us before and
// 30.0 after.  The plain path's kernels do not: with three models
// stepped at once, blocks that wait kept others from running (257 x 129 points
// 8.4 -> 10.0 us a step; 61^2, which leaves places free, gained 8 %).
#pragma once
#include <cuda_runtime.h>

namespace swm {

#ifdef __CUDACC__
// Programmatic dependent launch: a kernel launched with
// cudaLaunchAttributeProgrammaticStreamSerialization may start before its
// predecessor on the stream has finished; grid_dep_wait() returns once the
// predecessor has completed and its writes are visible (at once for a kernel
// launched the ordinary way).  grid_dep_trigger() lets the successor launch.
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dep_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// both, at the start of a kernel that reads nothing its predecessors write
// before this.  The wait first: the other way round a kernel that waits lets
// its successor launch, which waits too, and so on, and the blocks of several
// steps hold places that other streams' kernels could run in (a pass of 63
// steps, three models at once: 61 x 1300 points 415 us that way, 351 this way,
// 395 with ordinary launches; 301 x 401 379, 355, 420).
__device__ __forceinline__ void grid_dep_chain() {
  grid_dep_wait();
  grid_dep_trigger();
}
#endif

// cudaLaunchKernelEx with programmatic stream serialisation (see grid_dep_wait)
template <typename... KArgs, typename... Args>
cudaError_t launch_programmatic(void (*kernel)(KArgs...), dim3 grid, dim3 block, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace swm
