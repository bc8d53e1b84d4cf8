// Finds the context's status word for tests/test_gpu_status.py: preloaded, it notes the last word that is asked of
// mapped host memory and passes every call on to the runtime.
#include <dlfcn.h>
#include <cuda_runtime_api.h>

static void* word = nullptr;

extern "C" __attribute__((visibility("default"))) void* status_word() { return word; }

extern "C" __attribute__((visibility("default"))) cudaError_t cudaHostAlloc(void** p, size_t n, unsigned flags) {
  typedef cudaError_t (*Fn)(void**, size_t, unsigned);
  void* runtime = dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD);
  Fn next = runtime ? reinterpret_cast<Fn>(dlsym(runtime, "cudaHostAlloc")) : nullptr;
  if (!next) return cudaErrorUnknown;
  const cudaError_t e = next(p, n, flags);
  if (e == cudaSuccess && n == sizeof(unsigned) && (flags & cudaHostAllocMapped)) word = *p;
  return e;
}
