// Shared device helpers for the kiln-cuda kernels (sm_100a only).
//
// Everything that waits on the device (mbarrier phases) is bounded: a wait
// that does not complete within KC_SPIN_LIMIT_NS records a code in the
// context's status word and returns false, so a broken pipeline ends as an
// error status on the host instead of a hung GPU.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>
#include <utility>

#ifndef __CUDA_ARCH_FEAT_SM100_ALL
#if defined(__CUDA_ARCH__)
#error "kiln-cuda kernels are written for sm_100a only (compile with -gencode arch=compute_100a,code=sm_100a)"
#endif
#endif

namespace kc {

typedef __nv_bfloat16 bf16;
typedef __nv_bfloat162 bf162;

// Status word codes: (kernel id << 8) | wait id.
enum : uint32_t {
  KC_DEV_QLINEAR = 0x100,
  KC_DEV_ATTN = 0x200,
  KC_DEV_TP = 0x300,
};

constexpr unsigned long long KC_SPIN_LIMIT_NS = 1500ull * 1000ull * 1000ull;  // 1.5 s

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// One lane of a converged warp. Unlike `lane == 0` this keeps the code around it warp-uniform.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}

// ---- mbarrier: by shared address, or by pointer --------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) { mbar_init(smem_u32(bar), count); }
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) { mbar_arrive(smem_u32(bar)); }
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) { mbar_arrive_expect_tx(smem_u32(bar), bytes); }
// One try_wait: the thread may be suspended by the hardware until the phase completes or the hinted time
// (nanoseconds) has passed, so a waiting warp does not burn issue slots spinning.
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(20000u)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_test_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_test_wait(uint64_t* bar, uint32_t parity) { return mbar_test_wait(smem_u32(bar), parity); }
// Bounded wait. On timeout: ORs `code` into *status (if non-null) and returns
// false; the caller must then leave its pipeline loop.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint32_t* status,
                                          uint32_t code) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = globaltimer_ns();
  uint32_t spins = 0;
  while (!mbar_try_wait(bar, parity)) {
    if ((++spins & 0x3f) == 0) {
      if (globaltimer_ns() - t0 > KC_SPIN_LIMIT_NS) {
        if (status) atomicOr(status, code);
        return false;
      }
    }
  }
  return true;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint32_t* status, uint32_t code) {
  return mbar_wait(smem_u32(bar), parity, status, code);
}

// ---- async-proxy fences, bulk copies (TMA) --------------------------------
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// 1-D bulk copy global -> shared, completion counted on an mbarrier.
// Both addresses 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(uint32_t smem_dst, const void* gsrc, uint32_t bytes, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(smem_dst),
      "l"(gsrc), "r"(bytes), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void bulk_g2s(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  bulk_g2s(smem_u32(smem_dst), gsrc, bytes, smem_u32(bar));
}

// 2-D tiled TMA load (no multicast): coordinates {x = innermost, y}.
// x * element size must be a multiple of 16 bytes.
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* tmap, int32_t x,
                                            int32_t y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, "
      "%4}], [%2];" ::"r"(smem_u32(smem_dst)),
      "l"(tmap), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}
// 5-D tiled TMA load (no multicast).
__device__ __forceinline__ void tma_load_5d(void* smem_dst, const CUtensorMap* tmap, int32_t x, int32_t y, int32_t z,
                                            int32_t w, int32_t v, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];" ::
          "r"(smem_u32(smem_dst)),
      "l"(tmap), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(w), "r"(v)
      : "memory");
}
// Encodes a tiled map of `rank` <= 5 dimensions over bf16 elements, 128-byte swizzle; strides in bytes, of dimensions 1 ..
bool encode_tmap_bf16(CUtensorMap* map, int rank, const void* ptr, const uint64_t* dims, const uint64_t* strides,
                      const uint32_t* box, const char** err);
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* tmap) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(tmap) : "memory");
}

// ---- bf16 helpers --------------------------------------------------------
__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

__device__ __forceinline__ uint32_t pack_bf162(float lo, float hi) {
  bf162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float2 unpack_bf162(uint32_t u) {
  bf162 v = *reinterpret_cast<bf162*>(&u);
  return __bfloat1622float2(v);
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// ---- programmatic dependent launch ---------------------------------------
// Every kernel of the step but the first is launched with programmatic stream serialization: it may become resident while
// its predecessor in the stream is still running, executes whatever touches no data that a kernel of the step writes (barrier
// set-up, TMEM allocation, descriptor prefetch, loads of WEIGHTS), and calls pdl_wait() before its first access to memory
// that an earlier kernel of the step writes or reads. The step's first kernel (launch_embed) is launched in plain stream
// order: it starts when everything ahead of it is complete, and the others start after it has, so the copy of the step's
// metadata and all that earlier steps, block copies and resets wrote to the K/V pools is there for each of them. What only
// those wrote may therefore be read before pdl_wait() too: RoPE reads positions and slots, attention units, block tables and
// K/V of keys that the step does not write (AttnUnit::old). Where such a kernel may come first behind such a write it is
// launched in plain stream order itself (in_order). pdl_wait() returns once the
// predecessor grid has completed and its writes are visible; since every kernel calls it before it ends, a
// kernel's completion implies the completion of everything queued before it. pdl_launch_dependents() lets the
// successor start being scheduled; it is issued first thing, so the successor fills SMs as they drain.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// One-time set-up that has to happen once per DEVICE (kernel attributes live in the device's copy of the module, and
// one process may hold contexts on several devices). Host threads of different contexts may race here: the worst
// case is that the set-up runs twice, which is harmless.
struct DeviceOnce {
  unsigned long long done = 0;   // bit d: device d is configured (devices past 63 are configured on every call)
  bool first_on_current_device() {
    int d = 0;
    if (cudaGetDevice(&d) != cudaSuccess || d < 0 || d > 63) return true;
    if (done >> d & 1ull) return false;
    done |= 1ull << d;
    return true;
  }
  void forget_current_device() {
    int d = 0;
    if (cudaGetDevice(&d) == cudaSuccess && d >= 0 && d <= 63) done &= ~(1ull << d);
  }
};

// allow_early = false launches with plain stream order: used for the first kernel after a collective, whose duration
// depends on the OTHER ranks — nothing of this library may be resident and counting down a bounded wait meanwhile.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_k_opt(bool allow_early, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                                Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  if (allow_early) { cfg.attrs = attr; cfg.numAttrs = 1; }
  return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_k(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args&&... args) {
  return launch_k_opt(true, kernel, grid, block, smem, s, std::forward<Args>(args)...);
}

// In clusters of `cluster` CTAs along x.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_k_cluster(int cluster, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Two fp32 operations an instruction.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 r;
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\t"
      "fma.rn.f32x2 x, x, y, z;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return r;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 r;
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmul.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 r;
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tadd.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}

// tanh(y) for |y| < TANH_NEAR: y + y^3 p(y^2), p fitted for the smallest largest relative error; 1.0e-7 at most, 3.5e-8
// root mean square. No special-function operation.
constexpr float TANH_NEAR = 0.75f;
__device__ __forceinline__ float2 tanh_near(float2 y) {
  auto both = [](float x) { return make_float2(x, x); };
  const float2 z = mul2(y, y);
  float2 p = fma2(z, both(-0.0047694784589f), both(0.0196648966521f));
  p = fma2(p, z, both(-0.0533902496099f));
  p = fma2(p, z, both(0.1332652121782f));
  p = fma2(p, z, both(-0.3333306908607f));
  return fma2(mul2(y, z), p, y);
}
// tanh(y) anywhere: further out (1 - u) / (1 + u) with u = e^(-2 |y|), 1.7e-7 at most; 1 and -1 at the infinities, NaN stays
// NaN. Nowhere less exact than tanhf, which is up to 2.0e-7 off.
__device__ __forceinline__ float tanh_any(float y, float near) {
  const float u = ex2(fabsf(y) * -2.8853900817779268f), d = u + 1.f;
  float r = rcp_approx(d);
  r = __fmaf_rn(r, __fmaf_rn(-d, r, 1.f), r);
  const float far = copysignf(__fmaf_rn(-2.f * u, r, 1.f), y);
  return fabsf(y) < TANH_NEAR ? near : far;
}

// Mlp::forward activation (nn.rs:284-294): silu(gate) * up with the three bf16 roundings of the composed ops, or
// gelu_approx(gate) * up op for op (nn.rs:221-235). g and u are bf16 values held in fp32; so is the result.
// 1 / (1 + e^-g), the reciprocal by the hardware's estimate and one step of Newton's iteration, r + r (1 - d r): within 0.501 units
// of fp32's last place of the quotient, where a division is within 0.5, and without a division's branches, which cost a warp 100
// cycles each where others compute; rounded to bf16 it is the quotient's for every bf16 gate. The denominator is taken at 2^-32 of its
// size, so that the reciprocal of a large one (a gate below -87.3) is no subnormal number, which the estimate would flush. An
// infinite denominator is a zero.
__device__ __forceinline__ float act_sigmoid(float g) {
  const float d = fmaf(__expf(-g), 0x1p-32f, 0x1p-32f), r = rcp_approx(d), n = fmaf(r, fmaf(-d, r, 1.f), r);
  return (d > 1e37f ? r : n) * 0x1p-32f;
}
__device__ __forceinline__ float act_silu_mul(float g, float u) {
  const float s = bf16_round(act_sigmoid(g));
  const float t = bf16_round(g * s);
  return bf16_round(t * u);
}
__device__ __forceinline__ float gelu_scaled(float g) {
  const float cube = bf16_round(g * g * g);  // power(x, 3) in fp32, rounded once
  const float inner = bf16_round(g + bf16_round(bf16_round(0.044715f) * cube));
  return bf16_round(bf16_round(0.7978845608028654f) * inner);
}
__device__ __forceinline__ float2 act_gelu_mul(float2 g, float2 u) {
  const float2 y = make_float2(gelu_scaled(g.x), gelu_scaled(g.y)), near = tanh_near(y);   // no branch, as in act_sigmoid
  const float gx = bf16_round(1.f + bf16_round(tanh_any(y.x, near.x))), gy = bf16_round(1.f + bf16_round(tanh_any(y.y, near.y)));
  return make_float2(bf16_round(bf16_round(bf16_round(0.5f * g.x) * gx) * u.x), bf16_round(bf16_round(bf16_round(0.5f * g.y) * gy) * u.y));
}
__device__ __forceinline__ float act_gelu_mul(float g, float u) { return act_gelu_mul(make_float2(g, g), make_float2(u, u)).x; }

// Two of them at once, bf16 pairs in and out: a product of two bf16 numbers rounded to bf16 is what a multiplication of bf16 gives.
__device__ __forceinline__ uint32_t act_pair(uint32_t gate, uint32_t up, bool gelu) {
  const float2 g = unpack_bf162(gate);
  if (gelu) {
    const float2 a = act_gelu_mul(g, unpack_bf162(up));
    return pack_bf162(a.x, a.y);
  }
  const uint32_t s = pack_bf162(act_sigmoid(g.x), act_sigmoid(g.y));
  const bf162 t = __hmul2(*reinterpret_cast<const bf162*>(&gate), *reinterpret_cast<const bf162*>(&s));
  const bf162 r = __hmul2(t, *reinterpret_cast<const bf162*>(&up));
  return *reinterpret_cast<const uint32_t*>(&r);
}

// A ring position: stage index and phase bit, advanced without division.
struct RingPos {
  int stage = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void advance(int n_stages) {
    if (++stage == n_stages) { stage = 0; phase ^= 1u; }
  }
};

}  // namespace kc
