// Greedy sampling and the verify settle walk on the device.
#include "kc_fused.cuh"
#include "kc_umma.cuh"

namespace kc {

namespace {

struct ArgMax { float v; int i; };
__device__ __forceinline__ void load8_bf16(const bf16* p, float (&v)[8]) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const float2 a = unpack_bf162(u.x), b = unpack_bf162(u.y), c = unpack_bf162(u.z), d = unpack_bf162(u.w);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = d.x; v[7] = d.y;
}
__device__ __forceinline__ ArgMax better(ArgMax a, ArgMax b) {
  // larger value wins; on equal values the lower index wins (MLX argmax tie-break as
  // observed in docs/decisions/0004-golden-parity-device-scope-and-dtype-aware-delta.md:53-56)
  if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
  return a;
}

// sample_from_row + Sampler::sample, greedy lane (crates/kiln-engine/src/engine.rs:879-901,
// crates/kiln-engine/src/sampler.rs:100-104): logprobs = logits - logsumexp(logits) in the
// logits dtype, then argmax. The logsumexp accumulates in double and is rounded to bf16 before
// the subtraction; the subtraction result is rounded to bf16, which can merge neighbouring
// logits into ties — hence the explicit lowest-index rule.
// normalize == 0: argmax of the raw row (crates/kiln-models/src/draft.rs:379-381).
__global__ void __launch_bounds__(1024)
greedy_rows_kernel(const bf16* __restrict__ logits, int vocab, int normalize, uint32_t* __restrict__ tokens,
                   uint32_t* __restrict__ tokens_host, const volatile uint32_t* status, uint32_t* __restrict__ status_copy) {
  pdl_launch_dependents();
  pdl_wait();
  const bool notes = status_copy && blockIdx.x == 0 && threadIdx.x == 0;
  const uint32_t st = notes ? *status : 0u;   // host memory: on its way under the passes below
  __shared__ float red_m[32];
  __shared__ double red_s[32];
  __shared__ ArgMax red_a[32];
  __shared__ float s_lse;
  const bf16* row = logits + (size_t)blockIdx.x * vocab;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const bool vec = (vocab & 7) == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0;   // rows start on 16-byte boundaries
  if (normalize) {
    // Pass 1: the row maximum (exact). Pass 2: sum of exp(x - max), every term from the full-precision expf, the
    // running sums in double, so that the logsumexp — max + float(log(sum)), then one rounding to bf16 — lands on
    // the same bf16 value as a double-precision evaluation unless it sits within about 1e-6 of a rounding boundary.
    float m = -INFINITY;
    if (vec) {
      for (int i = threadIdx.x * 8; i < vocab; i += blockDim.x * 8) {
        float x[8];
        load8_bf16(row + i, x);
#pragma unroll
        for (int k = 0; k < 8; ++k) m = fmaxf(m, x[k]);
      }
    } else {
      for (int i = threadIdx.x; i < vocab; i += blockDim.x) m = fmaxf(m, __bfloat162float(row[i]));
    }
    m = warp_max(m);
    if (lane == 0) red_m[warp] = m;
    __syncthreads();
    m = lane < nw ? red_m[lane] : -INFINITY;
    m = warp_max(m);                       // every thread now holds the row maximum
    double sum = 0.0;
    if (vec) {
      for (int i = threadIdx.x * 8; i < vocab; i += blockDim.x * 8) {
        float x[8];
        load8_bf16(row + i, x);
        float part = 0.f;                  // eight terms in fp32 (each at most 1), then into the double sum
#pragma unroll
        for (int k = 0; k < 8; ++k) part += expf(x[k] - m);
        sum += (double)part;
      }
    } else {
      for (int i = threadIdx.x; i < vocab; i += blockDim.x) sum += (double)expf(__bfloat162float(row[i]) - m);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) red_s[warp] = sum;
    __syncthreads();
    if (warp == 0) {
      sum = lane < nw ? red_s[lane] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (lane == 0) s_lse = bf16_round(m + (float)log(sum));
    }
    __syncthreads();
  }
  const float lse = normalize ? s_lse : 0.f;
  ArgMax best{-INFINITY, 0x7fffffff};
  if (vec) {
    for (int i = threadIdx.x * 8; i < vocab; i += blockDim.x * 8) {
      float x[8];
      load8_bf16(row + i, x);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float v = normalize ? bf16_round(x[k] - lse) : x[k];
        if (v > best.v) best = ArgMax{v, i + k};   // indices rise within a thread: strict > keeps the lowest
      }
    }
  } else {
    for (int i = threadIdx.x; i < vocab; i += blockDim.x) {
      float x = __bfloat162float(row[i]);
      if (normalize) x = bf16_round(x - lse);
      best = better(best, ArgMax{x, i});
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgMax b2{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
    best = better(best, b2);
  }
  if (lane == 0) red_a[warp] = best;
  __syncthreads();
  if (warp == 0) {
    best = lane < nw ? red_a[lane] : ArgMax{-INFINITY, 0x7fffffff};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ArgMax b2{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
      best = better(best, b2);
    }
    if (lane == 0) {
      const uint32_t tok = (uint32_t)(best.i == 0x7fffffff ? 0 : best.i);
      tokens[blockIdx.x] = tok;
      if (tokens_host) tokens_host[blockIdx.x] = tok;
      if (notes) *status_copy = st;
    }
  }
}

// The same for rows that start on 16-byte boundaries, of at most GREEDY_CTAS * 256 * NV * 8 values: a row is a cluster's of eight CTAs, a
// thread keeps its share of the row in registers, and the row is read once. What bounds it: for few rows one round trip to L2 and the
// three exchanges between the CTAs, about a microsecond each; for many the exponentials and the exchanges of the clusters that an SM
// holds. The maximum is taken of packed pairs, and a value's rounded difference is the largest when the difference reaches the
// lowest float that rounds to it, so the last pass looks at vectors and only the vector that holds the winner is taken apart.
// 128256 values, in a step: 5 rows 24 -> 10 us, 32 rows 26 to 39 -> 14, 192 rows 44 -> 35; 152064
// values, 320 rows 76 to 86 -> 75.
constexpr int GREEDY_CTAS = 8, GREEDY_THREADS = 256;
__device__ __forceinline__ uint32_t max_bf162(uint32_t a, uint32_t b) {   // a NaN gives way to a number, as with fmaxf
  uint32_t r;
  asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
// The lowest float that bf16_round takes to v, a finite bf16 value or an infinity: half a step of bf16 below it, and that itself where
// v is even (a tie goes to it), else the next float up. Adjacent floats are adjacent integers on either side of zero.
__device__ __forceinline__ float lowest_rounding_to(float v) {
  const uint32_t b = __float_as_uint(v), odd = (b >> 16) & 1;
  if ((b << 1) == 0) return __uint_as_float(0x80008000u);            // zero: half of the smallest bf16 below it
  return __uint_as_float((b >> 31) ? b + 0x8000u - odd : b - 0x8000u + odd);
}
template <int NV>
__global__ void __launch_bounds__(GREEDY_THREADS, NV <= 8 ? 4 : NV <= 10 ? 3 : 2)
greedy_cluster_kernel(const bf16* __restrict__ logits, int vocab, int slice, int normalize, uint32_t* __restrict__ tokens,
                      uint32_t* __restrict__ tokens_host, const volatile uint32_t* status, uint32_t* __restrict__ status_copy) {
  pdl_launch_dependents();
  cluster_arrive();                      // waited for before the first store into another CTA's shared memory: it has started by then
  pdl_wait();
  const bool notes = status_copy && blockIdx.x == 0 && threadIdx.x == 0;
  const uint32_t st = notes ? *status : 0u;   // host memory: on its way under the passes below
  __shared__ float red_m[GREEDY_THREADS / 32], all_m[GREEDY_CTAS];
  __shared__ double red_s[GREEDY_THREADS / 32], all_s[GREEDY_CTAS];
  __shared__ int red_i[GREEDY_THREADS / 32], all_i[GREEDY_CTAS];
  const int row = blockIdx.x / GREEDY_CTAS, rank = blockIdx.x % GREEDY_CTAS;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = GREEDY_THREADS / 32;
  const bf16* values = logits + (size_t)row * vocab;
  const int begin = rank * slice, end = min(vocab, begin + slice), mine = begin + (int)threadIdx.x * 8;
  const uint32_t peer = threadIdx.x < GREEDY_CTAS ? threadIdx.x : 0;
  uint4 x[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int i = mine + k * GREEDY_THREADS * 8;
    x[k] = i < end ? *reinterpret_cast<const uint4*>(values + i) : make_uint4(0xFF80FF80u, 0xFF80FF80u, 0xFF80FF80u, 0xFF80FF80u);   // -infinity
  }
  auto top = [&](int k) { return max_bf162(max_bf162(x[k].x, x[k].y), max_bf162(x[k].z, x[k].w)); };
  uint32_t most = 0xFF80FF80u;
#pragma unroll
  for (int k = 0; k < NV; ++k) most = max_bf162(most, top(k));
  const float2 two = unpack_bf162(most);
  float m = warp_max(fmaxf(two.x, two.y));
  if (lane == 0) red_m[warp] = m;
  __syncthreads();
  cluster_wait();
  if (threadIdx.x < GREEDY_CTAS) {       // this CTA's maximum, to every CTA
    m = red_m[0];
    for (int w = 1; w < nw; ++w) m = fmaxf(m, red_m[w]);
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(cluster_addr(smem_u32(&all_m[rank]), peer)), "f"(m) : "memory");
  }
  cluster_sync();
  m = all_m[0];
#pragma unroll
  for (int c = 1; c < GREEDY_CTAS; ++c) m = fmaxf(m, all_m[c]);
  float lse = 0.f, least = m;
  if (normalize) {
    double sum = 0.0;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      uint32_t u[4] = {x[k].x, x[k].y, x[k].z, x[k].w};
      float part = 0.f;                  // eight terms in fp32 (each at most 1), then into the double sum
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        asm volatile("" : "+r"(u[j]));   // unpacked here: kept as floats from pass to pass the row would take twice the registers
        const float2 v = unpack_bf162(u[j]);
        part += expf(v.x - m);
        part += expf(v.y - m);
      }
      sum += (double)part;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) red_s[warp] = sum;
    __syncthreads();
    if (threadIdx.x < GREEDY_CTAS) {
      sum = red_s[0];
      for (int w = 1; w < nw; ++w) sum += red_s[w];
      asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(cluster_addr(smem_u32(&all_s[rank]), peer)), "d"(sum) : "memory");
    }
    cluster_sync();
    sum = all_s[0];
#pragma unroll
    for (int c = 1; c < GREEDY_CTAS; ++c) sum += all_s[c];
    lse = bf16_round(m + (float)log(sum));
    least = bf16_round(m - lse);         // NaN where the sum is, and then nothing reaches it
    if (least == least) least = lowest_rounding_to(least);
  }
  // a row whose largest value is -infinity has no winner: token 0
  int best = 0x7fffffff;
#pragma unroll
  for (int k = NV - 1; k >= 0; --k) {
    const float2 v = unpack_bf162(top(k));
    if (fmaxf(v.x, v.y) - lse >= least) {
      const uint32_t u[4] = {x[k].x, x[k].y, x[k].z, x[k].w};
#pragma unroll
      for (int j = 3; j >= 0; --j) {
        const float2 e = unpack_bf162(u[j]);
        if (e.y - lse >= least) best = mine + k * GREEDY_THREADS * 8 + 2 * j + 1;
        if (e.x - lse >= least) best = mine + k * GREEDY_THREADS * 8 + 2 * j;
      }
    }
  }
  best = __reduce_min_sync(0xffffffffu, best);
  if (lane == 0) red_i[warp] = best;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < nw; ++w) best = min(best, red_i[w]);
    asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(cluster_addr(smem_u32(&all_i[rank]), 0)), "r"(best) : "memory");
  }
  cluster_sync();
  if (rank == 0 && threadIdx.x == 0) {
    best = all_i[0];
    for (int c = 1; c < GREEDY_CTAS; ++c) best = min(best, all_i[c]);
    const uint32_t tok = (uint32_t)(best == 0x7fffffff || m == -INFINITY ? 0 : best);
    tokens[row] = tok;
    if (tokens_host) tokens_host[row] = tok;
    if (notes) *status_copy = st;
  }
}

// The settle walk (engine.rs:2336-2366): walk rows j = 0..|draft|; row j's token is committed;
// it "agrees" when j < |draft| and equals draft[j]; the walk stops after the first row that
// does not agree. n_committed = rows walked, n_accepted = agreeing rows.
__global__ void verify_accept_kernel(const uint32_t* __restrict__ row_tokens, const int32_t* __restrict__ seq_row_offsets,
                                     const uint32_t* __restrict__ draft, const int32_t* __restrict__ draft_offsets,
                                     const int32_t* __restrict__ draft_len, int n_seqs, int max_commit,
                                     uint32_t* __restrict__ committed, int32_t* __restrict__ n_committed,
                                     int32_t* __restrict__ n_accepted) {
  pdl_launch_dependents();
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_seqs) return;
  const int dl = draft_len[i];
  if (dl < 0) { n_committed[i] = 0; n_accepted[i] = 0; return; }  // segment samples nothing
  const uint32_t* rows = row_tokens + seq_row_offsets[i];
  const uint32_t* d = draft + draft_offsets[i];
  int acc = 0, com = 0;
  for (int j = 0; j <= dl; ++j) {
    const uint32_t tok = rows[j];
    const bool agrees = j < dl && tok == d[j];
    if (agrees) ++acc;
    if (com < max_commit) committed[(size_t)i * max_commit + com] = tok;
    ++com;
    if (!agrees) break;
  }
  n_committed[i] = com;
  n_accepted[i] = acc;
}

// Device-side token feedback of the pipelined decode (StepInput::Lazy, crates/kiln-engine/src/step.rs:45-56;
// engine.rs:1711-1713): row i of the step takes the token that row feed[i] of the previous step sampled.
__global__ void feed_tokens_kernel(uint32_t* __restrict__ tokens, const int32_t* __restrict__ feed,
                                   const uint32_t* __restrict__ prev, int n, int prev_n) {
  pdl_launch_dependents();
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int f = feed[i];
  if (f >= 0 && f < prev_n) tokens[i] = prev[f];
}

}  // namespace

cudaError_t launch_feed_tokens(uint32_t* tokens, const int32_t* feed, const uint32_t* prev, int n, int prev_n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  return launch_k(feed_tokens_kernel, dim3((n + 127) / 128), dim3(128), 0, s, tokens, feed, prev, n, prev_n);
}

cudaError_t launch_greedy_rows(const bf16* logits, int rows, int vocab, int normalize, uint32_t* tokens,
                               cudaStream_t s, uint32_t* tokens_host, const uint32_t* status, uint32_t* status_copy) {
  if (rows <= 0) return cudaSuccess;
  if ((vocab & 7) == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0 && rows <= 0x7fffffff / GREEDY_CTAS) {
    const int vectors = (vocab / 8 + GREEDY_CTAS - 1) / GREEDY_CTAS, slice = vectors * 8, each = (vectors + GREEDY_THREADS - 1) / GREEDY_THREADS;
    auto launch = [&](auto kernel) {
      return launch_k_cluster(GREEDY_CTAS, kernel, dim3(rows * GREEDY_CTAS), dim3(GREEDY_THREADS), 0, s, logits, vocab, slice, normalize, tokens, tokens_host, status, status_copy);
    };
    if (each <= 4) return launch(greedy_cluster_kernel<4>);
    if (each <= 8) return launch(greedy_cluster_kernel<8>);
    if (each <= 10) return launch(greedy_cluster_kernel<10>);
    if (each <= 16) return launch(greedy_cluster_kernel<16>);
  }
  return launch_k(greedy_rows_kernel, dim3(rows), dim3(1024), 0, s, logits, vocab, normalize, tokens, tokens_host, status, status_copy);
}

cudaError_t launch_verify_accept(const uint32_t* row_tokens, const int32_t* seq_row_offsets, const uint32_t* draft,
                                 const int32_t* draft_offsets, const int32_t* draft_len, int n_seqs, int max_commit,
                                 uint32_t* committed, int32_t* n_committed, int32_t* n_accepted, cudaStream_t s) {
  if (n_seqs <= 0) return cudaSuccess;
  return launch_k(verify_accept_kernel, dim3((n_seqs + 127) / 128), dim3(128), 0, s, row_tokens, seq_row_offsets, draft,
                  draft_offsets, draft_len, n_seqs, max_commit, committed, n_committed, n_accepted);
}

}  // namespace kc
