// Launch helpers: programmatic dependent launch (a kernel that starts while the one before it in the
// stream ends) and the functions' shared-memory limits.
#pragma once
#include <cuda_runtime.h>

#include <map>
#include <mutex>
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

// Lets kernel fn be launched with `bytes` of dynamic shared memory.  The limit belongs to the function
// on its device, for every handle of the process, and a launch above it is refused: it is only ever
// raised, so that a handle that needs less leaves the launches of the others as they are.
inline cudaError_t raise_smem_limit(const void* fn, size_t bytes) {
  static std::mutex lock;
  static std::map<std::pair<const void*, int>, size_t> limits;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> hold(lock);
  size_t& limit = limits[{fn, dev}];
  const size_t most = bytes > limit ? bytes : limit;
  // (set again where it stands, too: a device that was reset has forgotten it)
  e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
  if (e == cudaSuccess) limit = most;
  return e;
}

}  // namespace souffle
