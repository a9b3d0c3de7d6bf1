/* Preloaded before libcudart: cooperative launches are refused, all of them or all
   after the first, as the runtime refuses a grid that cannot be resident. */
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stdlib.h>
#include <string.h>

#include <cuda_runtime_api.h>

static int cooperative_launches;
int fake_cooperative_launches(void) { return cooperative_launches; }

cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* config, const void* func, void** args)
{
  typedef cudaError_t (*launch_t)(const cudaLaunchConfig_t*, const void*, void**);
  static launch_t real;
  if (!real) {
    void* rt = dlopen(FAKE_CUDART, RTLD_LAZY | RTLD_NOLOAD);
    real = (launch_t)dlsym(rt ? rt : RTLD_NEXT, "cudaLaunchKernelExC");
    if (!real) abort();
  }
  const char* mode = getenv("FAKE_LAUNCH");
  for (unsigned int i = 0; i < config->numAttrs; ++i)
    if (config->attrs[i].id == cudaLaunchAttributeCooperative && config->attrs[i].val.cooperative) {
      ++cooperative_launches;
      if (mode && (!strcmp(mode, "refuse") || (!strcmp(mode, "refuse_later") && cooperative_launches > 1)))
        return cudaErrorCooperativeLaunchTooLarge;
    }
  return real(config, func, args);
}
