// Programmatic dependent launch: a kernel that starts while the one before it in the stream ends.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace souffle {

// pdl_wait blocks until the kernels that this one depends on have completed (at once without the launch
// attribute); pdl_launch lets the next one start its own set-up.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// A launch whose set-up may overlap the end of the kernel before it; every kernel launched so calls
// pdl_wait, in every thread block, before it touches what earlier kernels write.
template <class... P, class... A>
cudaError_t launch_pdl(void (*k)(P...), int grid, int block, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, std::forward<A>(args)...);
}

}  // namespace souffle
