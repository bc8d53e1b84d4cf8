// All bf16 gates through the gated activation of the library's kernels and through its definition with fp32 division and tanhf; counts where
// the results have other bits. Built and loaded by test_gpu_activation.py.
#include "kc_common.cuh"

using namespace kc;

__device__ float reference(float g, float u, bool gelu) {
  if (!gelu) return bf16_round(bf16_round(g * bf16_round(1.f / (1.f + __expf(-g)))) * u);
  const float gate = bf16_round(1.f + bf16_round(tanhf(gelu_scaled(g))));
  return bf16_round(bf16_round(bf16_round(0.5f * g) * gate) * u);
}
__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b); }

// out: differing results of the one-value form, of the pair form; the first differing gate's bits
__global__ void check(int gelu, const uint16_t* ups, int n_ups, unsigned* out) {
  const unsigned bits = blockIdx.x * blockDim.x + threadIdx.x;
  const float g = __uint_as_float(bits << 16);
  for (int i = 0; i < n_ups; ++i) {
    const float u = __uint_as_float((unsigned)ups[i] << 16), want = reference(g, u, gelu);
    const float one = gelu ? act_gelu_mul(g, u) : act_silu_mul(g, u);
    const unsigned pair = act_pair(bits | 0x3F800000u, ups[i] | 0x40000000u, gelu);   // beside a gate of 1 and an up value of 2
    if (!same(one, want)) { atomicAdd(out, 1u); atomicMin(out + 2, bits); }
    if (!same(__uint_as_float(pair << 16), want)) { atomicAdd(out + 1, 1u); atomicMin(out + 2, bits); }
  }
}

extern "C" __attribute__((visibility("default"))) int run_check(int gelu, const uint16_t* ups, int n_ups, unsigned* out) {
  check<<<256, 256>>>(gelu, ups, n_ups, out);
  const cudaError_t e = cudaGetLastError();
  return e != cudaSuccess ? e : cudaDeviceSynchronize();
}
