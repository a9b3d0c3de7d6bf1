// Kernel launches with programmatic dependent launch, its device-side calls, and the
// shared-memory limit of a kernel.
#pragma once

#include <mutex>
#include <utility>

#include <cuda_runtime.h>

#include "mg_internal.h"

namespace mg {

// Programmatic dependent launch: wait for the preceding kernel's memory (a no-op
// when there is no programmatic dependency), and let the next kernel be
// scheduled once every CTA of this one has started.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... KArgs, typename... Args>
static cudaError_t launch_smem(bool pdl, void (*kernel)(KArgs...), int grid, int block, size_t smem, cudaStream_t st,
                               Args&&... args)
{
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}
template <typename... KArgs, typename... Args>
static cudaError_t launch_k(bool pdl, void (*kernel)(KArgs...), int grid, int block, cudaStream_t st, Args&&... args)
{
  return launch_smem(pdl, kernel, grid, block, 0, st, std::forward<Args>(args)...);
}
template <typename... KArgs, typename... Args>
static cudaError_t launch_pdl(void (*kernel)(KArgs...), int grid, int block, cudaStream_t st, Args&&... args)
{
  return launch_k(true, kernel, grid, block, st, std::forward<Args>(args)...);
}

// Sets the dynamic shared-memory limit of a kernel once per device, to the most that any
// launch of it takes: the limit belongs to the kernel on the device, so one set to a
// single launch's need would change under the launches of other host threads.
template <typename K>
static mg_status allow_smem(K kernel, size_t bytes, std::once_flag (&once)[64])
{
  int dev = 0;
  MG_CUDA(cudaGetDevice(&dev));
  cudaError_t err = cudaSuccess;
  std::call_once(once[dev & 63],
                 [&] { err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes); });
  MG_CUDA(err);
  return MG_OK;
}

}  // namespace mg
