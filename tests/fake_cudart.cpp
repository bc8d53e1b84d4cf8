// A stand-in for the CUDA runtime, for host-side tests of libkiln_cuda.so without a GPU: device memory is host memory,
// copies and fills happen at once, kernels do nothing. What the library asks for is kept in a list of calls that a test
// reads back, and chosen calls can be made to fail. Preloaded before the library; everything not defined here is the
// real runtime's.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>

namespace {
std::mutex mu;
std::string calls;
size_t fail_above = ~size_t(0);
bool fail_host_only = false;
std::string copied;
unsigned threads = 0;
std::string shapes;

void note(const char* what) {
  std::lock_guard<std::mutex> lk(mu);
  calls += what;
  calls += '\n';
}
cudaError_t alloc(void** p, size_t n, bool host) {
  note(host ? "host" : "malloc");
  if (n > fail_above && (host || !fail_host_only)) return cudaErrorMemoryAllocation;
  *p = aligned_alloc(256, (n + 255) / 256 * 256 + 256);
  return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
CUresult encode(CUtensorMap*, ...) { return CUDA_SUCCESS; }
}  // namespace

#define EXPORT extern "C" __attribute__((visibility("default")))

// what the tests call
EXPORT const char* fake_calls() { return calls.c_str(); }
EXPORT const char* fake_copied(size_t* n) { *n = copied.size(); return copied.data(); }   // the bytes of the last copy
EXPORT unsigned fake_threads() { return threads; }   // a block's, of the last launch in order
EXPORT const char* fake_shapes() { return shapes.c_str(); }   // threads:grid of the launches with attributes
EXPORT void fake_reset() { std::lock_guard<std::mutex> lk(mu); calls.clear(); shapes.clear(); }
EXPORT void fake_fail_above(size_t bytes) { fail_above = bytes; }         // allocations larger than this fail
EXPORT void fake_fail_host_only(int on) { fail_host_only = on != 0; }     // ... of pinned memory only

EXPORT cudaError_t cudaMalloc(void** p, size_t n) { return alloc(p, n, false); }
EXPORT cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return alloc(p, n, true); }
EXPORT cudaError_t cudaMallocHost(void** p, size_t n) { return alloc(p, n, true); }
EXPORT cudaError_t cudaFree(void* p) { note("free"); free(p); return cudaSuccess; }
EXPORT cudaError_t cudaFreeHost(void* p) { note("free"); free(p); return cudaSuccess; }
EXPORT cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) { *d = h; return cudaSuccess; }
EXPORT cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
EXPORT cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  note("copy");
  memcpy(d, s, n);
  copied.assign(static_cast<const char*>(s), n);
  return cudaSuccess;
}
EXPORT cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t) {
  for (size_t i = 0; i < h; ++i) memcpy(static_cast<char*>(d) + i * dp, static_cast<const char*>(s) + i * sp, w);
  return cudaSuccess;
}
EXPORT cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { note("fill"); memset(d, v, n); return cudaSuccess; }
EXPORT cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = reinterpret_cast<cudaStream_t>(malloc(1)); return cudaSuccess; }
EXPORT cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
EXPORT cudaError_t cudaStreamSynchronize(cudaStream_t) { note("sync"); return cudaSuccess; }
EXPORT cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
EXPORT cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = reinterpret_cast<cudaEvent_t>(malloc(1)); return cudaSuccess; }
EXPORT cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
EXPORT cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
EXPORT cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
EXPORT cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
EXPORT cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }
EXPORT cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
EXPORT cudaError_t cudaGetSymbolAddress(void** p, const void*) {
  static char array[256];   // kernels do nothing: only its address is used
  *p = array;
  return cudaSuccess;
}
EXPORT cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
EXPORT cudaError_t cudaSetDevice(int) { return cudaSuccess; }
EXPORT cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
EXPORT cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) {
  memset(p, 0, sizeof *p);
  p->major = 10;
  p->multiProcessorCount = 148;
  return cudaSuccess;
}
EXPORT cudaError_t cudaGetLastError() { return cudaSuccess; }
EXPORT cudaError_t cudaGetDriverEntryPoint(const char*, void** f, unsigned long long, cudaDriverEntryPointQueryResult* q) {
  *f = reinterpret_cast<void*>(&encode);
  if (q) *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
EXPORT cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { note("launch in order"); return cudaSuccess; }
EXPORT cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void*, void**) {
  bool early = false;
  for (unsigned i = 0; i < c->numAttrs; ++i)
    early |= c->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization && c->attrs[i].val.programmaticStreamSerializationAllowed;
  note(early ? "launch early" : "launch in order");
  if (!early) threads = c->blockDim.x;
  shapes += std::to_string(c->blockDim.x) + ':' + std::to_string(c->gridDim.x) + 'x' + std::to_string(c->gridDim.y) + 'x' + std::to_string(c->gridDim.z) + '\n';
  return c->gridDim.y > 65535 || c->gridDim.z > 65535 ? cudaErrorInvalidConfiguration : cudaSuccess;
}
