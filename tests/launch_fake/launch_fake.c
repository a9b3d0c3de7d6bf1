/* Preloaded before libcudart: cooperative launches are refused as the runtime refuses a
   grid that cannot be resident, or run with another limit on the polls of their waits
   (the resident CG's last argument); all of them, or all after the first. */
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
  const char *mode = getenv("FAKE_LAUNCH"), *spins = getenv("FAKE_SPINS");
  for (unsigned int i = 0; i < config->numAttrs; ++i)
    if (config->attrs[i].id == cudaLaunchAttributeCooperative && config->attrs[i].val.cooperative) {
      ++cooperative_launches;
      const int now = mode && (!strstr(mode, "later") || cooperative_launches > 1);
      if (now && !strncmp(mode, "refuse", 6)) return cudaErrorCooperativeLaunchTooLarge;
      if (now && !strncmp(mode, "give_up", 7)) {
        int limit = spins ? atoi(spins) : 0;
        void* a[17];
        memcpy(a, args, sizeof(a));
        a[16] = &limit;
        return real(config, func, a);
      }
    }
  return real(config, func, args);
}
