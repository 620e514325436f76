/* Preloaded: the RC_FAIL_LAUNCH-th cudaGraphLaunch of the process returns
 * cudaErrorMemoryAllocation and launches nothing. */
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stdlib.h>

typedef int (*launch_fn)(void*, void*);

int cudaGraphLaunch(void* graph, void* stream) {
  static launch_fn real;
  static int calls;
  if (!real) {
    void* lib = dlopen("libcudart.so.13", RTLD_NOW | RTLD_NOLOAD);
    real = lib ? (launch_fn)dlsym(lib, "cudaGraphLaunch") : 0;
  }
  const char* n = getenv("RC_FAIL_LAUNCH");
  if (!real || (n && ++calls == atoi(n))) return 2;
  return real(graph, stream);
}
