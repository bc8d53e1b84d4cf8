// Quantised weights: re-tiling, the activations' tensor maps, the lanes for few rows of a draft model, the split-K reduction.
// The GEMM on the tensor cores is in kc_qlinear_umma.cu. See kc_qlinear.cuh for the data layout.
#include "kc_qlinear.cuh"

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <cstdlib>

namespace kc {

// ---------------------------------------------------------------------------
// Re-tiling
// ---------------------------------------------------------------------------

__global__ void qweight_retile_kernel(uint8_t* __restrict__ records, const uint32_t* __restrict__ w,
                                      const bf16* __restrict__ scales, const bf16* __restrict__ biases,
                                      int N, int K, int bits, int group, int n_tiles, int kblocks,
                                      int alternate, int gpk, uint32_t packed_bytes, uint32_t record_bytes, int* __restrict__ exponents) {
  int largest = 0, smallest = 0;   // exponents, biased, that this thread has met: of finite scales; from 255, of scales and biases that are not 0
  // alternate: the source has N / 2 gate rows, then N / 2 up rows; 16 of each take turns
  auto source = [&](int n) { return alternate ? (n >> 5 << 4) + (n & 15) + (n & 16 ? N / 2 : 0) : n; };
  const int words_per_row_kb = QL_KB * bits / 32;  // 8 (w4) or 16 (w8)
  const int words_per_rec = QL_TILE_N * words_per_row_kb;
  const int sb_per_rec = QL_TILE_N * gpk;
  const long long per_rec = words_per_rec + sb_per_rec;
  const long long total = (long long)((n_tiles + QL_TILE_GROUP - 1) / QL_TILE_GROUP) * QL_TILE_GROUP * kblocks * per_rec;
  const int src_words_per_row = K * bits / 32;
  const int groups_per_row = K / group;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long rec = i / per_rec;
    const int e = (int)(i % per_rec);
    // record order: [tile group][k-block][tile in group], so the records of 1, 2 or 4 neighbouring tiles for
    // one k-block are contiguous and one bulk copy fetches them
    const int tig = (int)(rec % QL_TILE_GROUP);
    const long long gk = rec / QL_TILE_GROUP;
    const int kb = (int)(gk % kblocks);
    const int tile = (int)(gk / kblocks) * QL_TILE_GROUP + tig;
    uint8_t* base = records + rec * (long long)record_bytes;
    if (e < words_per_rec) {
      const int r = e / words_per_row_kb, c = e % words_per_row_kb;
      const int n = tile * QL_TILE_N + r;
      uint32_t v = 0;
      if (n < N) v = w[(long long)source(n) * src_words_per_row + kb * words_per_row_kb + c];
      if (bits == 4) {
        uint32_t o = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          o |= ((v >> (8 * j)) & 0xFu) << (4 * j);
          o |= ((v >> (8 * j + 4)) & 0xFu) << (16 + 4 * j);
        }
        v = o;
      }
      // 16-byte chunk c / 4 of row r: chunk-major, so that neighbouring rows' chunks are neighbours in shared memory
      reinterpret_cast<uint32_t*>(base)[((c >> 2) * QL_TILE_N + r) * 4 + (c & 3)] = v;
    } else {
      const int e2 = e - words_per_rec;
      const int r = e2 / gpk, gi = e2 % gpk;
      const int n = tile * QL_TILE_N + r;
      bf162 sb = __floats2bfloat162_rn(0.f, 0.f);
      if (n < N) {
        const int g = (kb * QL_KB + gi * group) / group;
        sb.x = scales[(long long)source(n) * groups_per_row + g];
        sb.y = biases[(long long)source(n) * groups_per_row + g];
        const int scale = __bfloat16_as_ushort(sb.x) & 0x7FFF, bias = __bfloat16_as_ushort(sb.y) & 0x7FFF;
        if (scale >> 7 < 255) largest = max(largest, scale >> 7);
        if (scale) smallest = max(smallest, 255 - (scale >> 7));
        if (bias) smallest = max(smallest, 255 - (bias >> 7));
      }
      reinterpret_cast<bf162*>(base + packed_bytes)[e2] = sb;
    }
  }
  largest = __reduce_max_sync(0xffffffffu, largest);   // all threads are here
  smallest = __reduce_max_sync(0xffffffffu, smallest);
  if ((threadIdx.x & 31) == 0) {
    if (largest) atomicMax(exponents, largest);
    if (smallest) atomicMax(exponents + 1, smallest);
  }
}

int qlinear_plan_splits(int n_tiles, int kblocks, int sm_count) {
  // As many k-splits as fill the SMs with a CTA a tile and split, each keeping at least 8 k-blocks; none where the tiles alone keep
  // half of the SMs busy. Splits need not divide the k-blocks evenly (the kernel cuts [K s / S, K (s + 1) / S)).
  if (n_tiles * 2 >= sm_count) return 1;
  int s = sm_count / n_tiles;
  s = std::min(s, std::min(16, kblocks / 8));
  return std::max(s, 1);
}

int qlinear_plan_chains(int n_tiles, int splits, int sm_count) { return (n_tiles + 1) / 2 * splits * 10 >= sm_count * 7 ? 1 : 2; }

cudaError_t qweight_build(QWeight* out, const uint32_t* w, const bf16* scales, const bf16* biases,
                          int N, int K, int bits, int group, int sm_count, cudaStream_t s, bool alternate) {
  QWeight q;
  q.N = N; q.K = K; q.bits = bits; q.group = group;
  q.n_tiles = (N + QL_TILE_N - 1) / QL_TILE_N;
  q.kblocks = K / QL_KB;
  q.gpk = std::max(1, QL_KB / group);
  q.packed_bytes = QL_TILE_N * (QL_KB * bits / 8);
  q.record_bytes = q.packed_bytes + QL_TILE_N * q.gpk * 4;
  q.splits = qlinear_plan_splits(q.n_tiles, q.kblocks, sm_count);
  q.chains = qlinear_plan_chains(q.n_tiles, q.splits, sm_count);
  q.sm_count = sm_count;
  // one allocation: the records, then the exponents that the re-tiling finds
  cudaError_t e = cudaMalloc(&q.records, q.bytes() + 16);
  if (e != cudaSuccess) return e;
  q.exponents = reinterpret_cast<int*>(q.records + q.bytes());
  e = cudaMemsetAsync(q.exponents, 0, 16, s);
  if (e != cudaSuccess) { cudaFree(q.records); return e; }
  const long long total = (long long)(q.bytes() / 4);
  const int threads = 256;
  const int blocks = (int)std::min<long long>((total + threads - 1) / threads, 148LL * 16);
  qweight_retile_kernel<<<blocks, threads, 0, s>>>(q.records, w, scales, biases, N, K, bits, group,
                                                   q.n_tiles, q.kblocks, alternate ? 1 : 0, q.gpk, q.packed_bytes,
                                                   q.record_bytes, q.exponents);
  e = cudaGetLastError();
  if (e != cudaSuccess) { cudaFree(q.records); return e; }
  *out = q;
  return cudaSuccess;
}

cudaError_t qweight_finish(QWeight* w) {
  int exponents[2] = {0, 0};
  cudaError_t e = cudaMemcpy(exponents, w->exponents, sizeof exponents, cudaMemcpyDeviceToHost);
  w->shift = std::max(0, exponents[0] - 121);   // scale * 2^(133 - shift) < 2^(exponent - 126 + 133 - shift) <= 2^128
  // A weight is a multiple of the last place of its scale or bias, and rounded as the shifted one is unless that falls below 2^-126; its product
  // with an activation of 2^-32 or more, and all bits of it, stay above that too where no scale or bias is shifted below 2^-63.
  w->wide = w->shift > 0 && 255 - exponents[1] - w->shift < 127 - 63;
  if (w->wide) w->shift = 0;
  return e;
}

void qweight_free(QWeight* w) {
  if (w && w->records) { cudaFree(w->records); w->records = nullptr; }
}

// ---------------------------------------------------------------------------
// Tensor maps for the activation operand
// ---------------------------------------------------------------------------

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

bool encode_tmap_bf16(CUtensorMap* map, int rank, const void* ptr, const uint64_t* dims, const uint64_t* strides,
                      const uint32_t* box, const char** err) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) { *err = "cuTensorMapEncodeTiled entry point unavailable"; return false; }
  cuuint64_t d[5], st[4];
  cuuint32_t b[5], estr[5];
  for (int i = 0; i < rank; ++i) { d[i] = dims[i]; b[i] = box[i]; estr[i] = 1; }
  for (int i = 0; i + 1 < rank; ++i) st[i] = strides[i];
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(ptr), d, st, b, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  rank > 2 ? CU_TENSOR_MAP_L2_PROMOTION_L2_256B : CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { *err = "cuTensorMapEncodeTiled rejected the tensor geometry"; return false; }
  return true;
}

static bool make_tmap_bf16_2d(CUtensorMap* map, const void* ptr, uint64_t inner, uint64_t outer,
                              uint32_t box_inner, uint32_t box_outer, const char** err) {
  const uint64_t dims[2] = {inner, outer}, strides[1] = {inner * sizeof(bf16)};
  const uint32_t box[2] = {box_inner, box_outer};
  return encode_tmap_bf16(map, 2, ptr, dims, strides, box, err);
}

// The map whose box covers `m_pad` rows (<= 256), so that one TMA operation brings a whole activation k-block.
// Re-encoded only when the row count changes (a host-side encode, no device work).
const CUtensorMap* act_operand_rows_map(const ActOperand* op, int m_pad) {
  if (op->rows_map_n != m_pad) {
    const char* err = "";
    if (!make_tmap_bf16_2d(&op->rows_map, op->ptr, op->K, op->rows, QL_KB, m_pad, &err)) return nullptr;
    op->rows_map_n = m_pad;
  }
  return &op->rows_map;
}

bool act_operand_init(ActOperand* op, const bf16* ptr, int rows, int K, const char** err) {
  op->ptr = ptr; op->rows = rows; op->K = K; op->rows_map_n = 0;
  if (K % QL_KB) { *err = "activation width must be a multiple of 64"; return false; }
  // the first launch's map is encoded here so that a geometry the driver refuses is reported at binding
  const int m_pad = std::min(256, (rows + 15) & ~15);
  if (!make_tmap_bf16_2d(&op->rows_map, ptr, K, rows, QL_KB, m_pad, err)) return false;
  op->rows_map_n = m_pad;
  return true;
}

// ---------------------------------------------------------------------------
// The weight-streaming lane: at most 8 activation rows (the draft model's chained decode forwards,
// crates/kiln-models/src/draft.rs:354-388). Such a launch is bound by the weight bytes alone, and the tensor-core
// kernel above spends most of its time setting up its pipelines. Here the weight is one flat list of units (one
// k-block of one group of four neighbouring tiles: contiguous in memory) that a grid of persistent CTAs cuts into equal
// contiguous runs; a producer warp bulk-copies a CTA's units through a shared-memory ring, and eight consumer warps,
// 16 rows of each of the four tiles apiece, multiply them with mma.sync.m16n8k16, the activation rows riding as the 8
// columns of the B operand (one activation fragment serves the four tiles).
//
// Arithmetic: MLX's row-vector class (its qmv kernels, which serve small batches there too): per quantisation group
// y += scale * sum_k(x_k q_k) + bias * sum_k(x_k) in fp32. The MMA runs on the raw integers (a 4-bit q enters as the
// bf16 value 128 + q, which one OR builds; the 128 is folded into the bias term), so nothing is dequantised per
// element. The 16 k positions of an MMA are assigned to the lanes so that lane (g, t) owns input features
// 32 h + 8 t .. + 7 of each 32-feature half h of the k-block — 4 contiguous bytes of a 4-bit row — and the activation
// fragment is gathered with the same assignment, so the sum runs over the same products.
//
// A run that crosses a group boundary flushes one partial per group it touches. The partials are fp32
// [pieces][M][N]; which CTA writes which piece of which group is a function of the weight's shape and the SM count
// only, and the consumer kernel sums the pieces in index order, so the result does not depend on timing or on M.
// ---------------------------------------------------------------------------

__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                               uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

constexpr int QG_CONSUMER_WARPS = 8;                       // x 16 weight rows = the 128 rows of a tile
constexpr int QG_THREADS = 32 * (QG_CONSUMER_WARPS + 1);   // + the producer warp
#ifndef QG_CTAS
#define QG_CTAS 2
#endif
constexpr int QG_CTAS_PER_SM = QG_CTAS;
constexpr int QG_MAX_PIECES = 40;                          // fp32 partials per output element, at most
constexpr int QG_MIN_UNITS = 4;                            // a CTA's run is at least this long (about 72 KB of 4-bit records)
constexpr int QG_MAX_STAGES = QG_CTAS == 3 ? 3 : 4;
constexpr size_t QG_RING_BYTES = QG_CTAS == 3 ? 60 * 1024 : 80 * 1024;

// One unit of work = the records of one k-block of a whole tile group (QL_TILE_GROUP neighbouring tiles, contiguous in
// memory): one bulk copy, one barrier round, one activation fragment for 4 x 128 weight rows.
struct QgParams {
  const uint8_t* records;
  uint32_t record_bytes;
  int N, n_groups, kblocks, pieces, stages;
  const bf16* x;   // [M, ldx]
  int ldx, M;
  float* partial;  // [pieces][M][N]
  uint32_t* status;
};

// The persistent CTA that owns unit r of T when G CTAs cut the list into runs [T c / G, T (c + 1) / G).
__host__ __device__ inline long long qg_owner(long long r, long long T, long long G) { return ((r + 1) * G + T - 1) / T - 1; }

// Elements (2p, 2p + 1), p = 0..3, of the lane's 8 features as bf16 pairs holding the raw integers.
template <int BITS>
__device__ __forceinline__ void qg_raw_pairs(const uint32_t* u, uint32_t (&e)[4]) {
  if (BITS == 4) {
    // The record's nibble order puts element 2p at bits 4p and element 2p + 1 at bits 16 + 4p. Two masks split the
    // word into bytes (even nibbles: elements 0, 4, 1, 5; odd nibbles: 2, 6, 3, 7), and a byte permute sets each
    // under 0x43: the bf16 value 128 + q, exact.
    const uint32_t lo = u[0] & 0x0F0F0F0Fu, hi = (u[0] >> 4) & 0x0F0F0F0Fu;
    e[0] = __byte_perm(lo, 0x43434343u, 0x4240u);   // elements 0, 1
    e[1] = __byte_perm(hi, 0x43434343u, 0x4240u);   // elements 2, 3
    e[2] = __byte_perm(lo, 0x43434343u, 0x4341u);   // elements 4, 5
    e[3] = __byte_perm(hi, 0x43434343u, 0x4341u);   // elements 6, 7
  } else {
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const uint32_t w = u[p >> 1];
      const int k = (p & 1) * 2;
      // byte k under the exponent of 2^23: the float 8388608 + q, minus 2^23 = q exactly; q < 256 is exact in bf16
      const float lo = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540u | k)) - 8388608.f;
      const float hi = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540u | (k + 1))) - 8388608.f;
      e[p] = pack_bf162(lo, hi);
    }
  }
}

// Byte offset in a record of the 8 features 8 t .. 8 t + 7 of a row's first 32-feature half: with 16-byte chunks
// chunk-major, the four lanes of a 4-bit row read one chunk and those of an 8-bit row two.
template <int BITS>
__device__ __forceinline__ uint32_t lane_offset(int row, int t) {
  return BITS == 4 ? (uint32_t)row * 16 + t * 4 : (uint32_t)((t >> 1) * QL_TILE_N + row) * 16 + (t & 1) * 8;
}

template <int BITS, int GPK>
__global__ void __launch_bounds__(QG_THREADS, QG_CTAS_PER_SM) qlinear_stream_kernel(const QgParams p) {
  constexpr int ROW_BYTES = QL_KB * BITS / 8;          // bytes of one weight row in one k-block: 32 or 64
  constexpr int PACKED = QL_TILE_N * ROW_BYTES;
  constexpr int HALF_BYTES = QL_TILE_N * ROW_BYTES / 2;   // one 32-feature half of all rows (chunk-major order)
  constexpr int LANE_WORDS = BITS / 4;                 // 32-bit words holding the lane's 8 features of a half
  constexpr int NT = QL_TILE_GROUP;
  extern __shared__ __align__(128) uint8_t smem[];
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = p.stages;
  const uint32_t unit_bytes = NT * p.record_bytes;
  uint8_t* ring = smem;
  float* xs = reinterpret_cast<float*>(smem + (size_t)S * unit_bytes);               // [kblocks][GPK][8]
  uint64_t* full = reinterpret_cast<uint64_t*>(xs + (size_t)p.kblocks * GPK * 8);
  uint64_t* empty = full + S;
  const long long T = (long long)p.n_groups * p.kblocks, G = gridDim.x;
  const long long R0 = T * blockIdx.x / G, R1 = T * (blockIdx.x + 1) / G;
  const int n_units = (int)(R1 - R0);
  if (threadIdx.x == 0) {
    for (int i = 0; i < S; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], QG_CONSUMER_WARPS); }
    mbar_fence_init();
  }
  __syncthreads();

  if (warp == QG_CONSUMER_WARPS) {
    // ---- producer: the weights do not depend on the kernels before this one, so it never waits for them ----
    if (lane == 0) {
      RingPos rp;
      int issued = 0;
      bool ok = true;
      const uint8_t* src = p.records + (size_t)R0 * unit_bytes;   // units are contiguous: [group][k-block][tile in group]
      for (int i = 0; i < n_units; ++i, rp.advance(S), src += unit_bytes) {
        if (!mbar_wait(&empty[rp.stage], rp.phase ^ 1, p.status, KC_DEV_QLINEAR | 0x11)) { ok = false; break; }
        mbar_arrive_expect_tx(&full[rp.stage], unit_bytes);
        bulk_g2s(ring + (size_t)rp.stage * unit_bytes, src, unit_bytes, &full[rp.stage]);
        ++issued;
      }
      if (!ok) {
        // gave up: the copies already issued still land in this CTA's shared memory; wait for them (bounded) before leaving
        RingPos dp;
        for (int i = 0; i < issued; ++i, dp.advance(S))
          if (i >= issued - S) mbar_wait(&full[dp.stage], dp.phase, p.status, KC_DEV_QLINEAR | 0x12);
      }
    }
  } else {
    // ---- consumers ----
    const int g = lane >> 2, t = lane & 3;
    const int r0 = warp * 16 + g;                      // this lane's weight rows in each tile: r0 and r0 + 8
    const bool x_live = g < p.M;
    const bf16* xr = p.x + (size_t)(x_live ? g : 0) * p.ldx + 8 * t;
    pdl_wait();   // x comes from the kernel before; the partials below may still be read by it
    // sum_k x_k per (k-block, group half, activation row) for the k-blocks of this CTA's run
    {
      const int n_kb = n_units < p.kblocks ? n_units : p.kblocks;
      for (int i = warp; i < n_kb; i += QG_CONSUMER_WARPS) {
        const int kb = (int)((R0 + i) % p.kblocks);
        float sh[2] = {0.f, 0.f};
        if (x_live) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint4 v = *reinterpret_cast<const uint4*>(xr + (size_t)kb * QL_KB + 32 * h);
            const float2 a = unpack_bf162(v.x), b = unpack_bf162(v.y), c = unpack_bf162(v.z), d = unpack_bf162(v.w);
            sh[h] = ((a.x + a.y) + (b.x + b.y)) + ((c.x + c.y) + (d.x + d.y));
          }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          sh[h] += __shfl_xor_sync(0xffffffffu, sh[h], 1);
          sh[h] += __shfl_xor_sync(0xffffffffu, sh[h], 2);
        }
        if (t == 0) {
          if (GPK == 2) { xs[((size_t)kb * 2 + 0) * 8 + g] = sh[0]; xs[((size_t)kb * 2 + 1) * 8 + g] = sh[1]; }
          else xs[(size_t)kb * 8 + g] = sh[0] + sh[1];
        }
      }
      asm volatile("bar.sync 1, %0;" ::"n"(QG_CONSUMER_WARPS * 32) : "memory");
    }
    float acc[NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    int grp = (int)(R0 / p.kblocks), kb = (int)(R0 % p.kblocks);
    long long seg0 = R0;   // first unit of the current group's segment
    bool ok = true;
    RingPos rp;
    auto flush = [&](long long seg_end) {
      // acc[j][0], [1] = weight row r0 of tile j against activation rows 2t, 2t + 1; [2], [3] = row r0 + 8
      const long long t_first = (long long)grp * p.kblocks, t_last = t_first + p.kblocks - 1;
      const int c_first = (int)qg_owner(t_first, T, G);
      const int piece = (int)blockIdx.x - c_first;
      const int n_pieces = (int)qg_owner(t_last, T, G) - c_first + 1;
      const bool closes = seg_end == t_last + 1;       // the CTA holding a group's last unit also clears its unused slots
#pragma unroll
      for (int j = 0; j < NT; ++j) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int n = (grp * NT + j) * QL_TILE_N + r0 + 8 * h;
          if (n < p.N) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int m = 2 * t + e;
              if (m < p.M) {
                p.partial[((size_t)piece * p.M + m) * p.N + n] = acc[j][2 * h + e];
                if (closes)
                  for (int q = n_pieces; q < p.pieces; ++q) p.partial[((size_t)q * p.M + m) * p.N + n] = 0.f;
              }
            }
          }
        }
        acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
      }
    };
    const uint32_t lane_off = lane_offset<BITS>(r0, t);
    const uint32_t sb_off = PACKED + (uint32_t)r0 * GPK * 4;
    // the activation fragment and the row sums of a unit are fetched one unit ahead
    uint4 xa[2], xa_next[2];
    float2 xsum[GPK], xsum_next[GPK];
    auto fetch_x = [&](int kbn, uint4 (&xv)[2], float2 (&sv)[GPK]) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        xv[h] = make_uint4(0, 0, 0, 0);
        if (x_live) xv[h] = *reinterpret_cast<const uint4*>(xr + (size_t)kbn * QL_KB + 32 * h);
      }
#pragma unroll
      for (int q = 0; q < GPK; ++q) sv[q] = *reinterpret_cast<const float2*>(xs + ((size_t)kbn * GPK + q) * 8 + 2 * t);
    };
    fetch_x(kb, xa_next, xsum_next);
    for (int i = 0; i < n_units; ++i, rp.advance(S)) {
      xa[0] = xa_next[0]; xa[1] = xa_next[1];
#pragma unroll
      for (int q = 0; q < GPK; ++q) xsum[q] = xsum_next[q];
      if (i + 1 < n_units) fetch_x(kb + 1 == p.kblocks ? 0 : kb + 1, xa_next, xsum_next);
      ok = __all_sync(0xffffffffu, mbar_wait(&full[rp.stage], rp.phase, p.status, KC_DEV_QLINEAR | 0x13));
      if (!ok) break;
      const uint8_t* unit = ring + (size_t)rp.stage * unit_bytes;
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const uint8_t* rec = unit + (size_t)j * p.record_bytes;
        uint32_t u[2][2][LANE_WORDS];   // [half][row r0 / r0 + 8][words]
        uint32_t sbw[2][GPK];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const uint8_t* src = rec + lane_off + r * 8 * 16 + h * HALF_BYTES;
            if (LANE_WORDS == 1) u[h][r][0] = *reinterpret_cast<const uint32_t*>(src);
            else { const uint2 v = *reinterpret_cast<const uint2*>(src); u[h][r][0] = v.x; u[h][r][LANE_WORDS - 1] = v.y; }
          }
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
          for (int q = 0; q < GPK; ++q) sbw[r][q] = *reinterpret_cast<const uint32_t*>(rec + sb_off + r * 8 * GPK * 4 + q * 4);
        float raw[2][4];   // one accumulator per 32-feature half: the two MMA chains are independent
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          raw[h][0] = raw[h][1] = raw[h][2] = raw[h][3] = 0.f;
          uint32_t e0[4], e1[4];
          qg_raw_pairs<BITS>(u[h][0], e0);
          qg_raw_pairs<BITS>(u[h][1], e1);
          mma_bf16_16816(raw[h], e0[0], e1[0], e0[2], e1[2], xa[h].x, xa[h].z);
          mma_bf16_16816(raw[h], e0[1], e1[1], e0[3], e1[3], xa[h].y, xa[h].w);
        }
        if (GPK == 1) {
#pragma unroll
          for (int c = 0; c < 4; ++c) raw[0][c] += raw[1][c];
        }
#pragma unroll
        for (int q = 0; q < GPK; ++q) {
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const float sc = __uint_as_float(sbw[r][q] << 16), bi = __uint_as_float(sbw[r][q] & 0xFFFF0000u);
            const float bc = BITS == 4 ? fmaf(-128.f, sc, bi) : bi;   // the 128 every 4-bit q carries
            acc[j][2 * r + 0] = fmaf(sc, raw[q][2 * r + 0], fmaf(bc, xsum[q].x, acc[j][2 * r + 0]));
            acc[j][2 * r + 1] = fmaf(sc, raw[q][2 * r + 1], fmaf(bc, xsum[q].y, acc[j][2 * r + 1]));
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[rp.stage]);   // the unit has been read: its slot can refill
      if (++kb == p.kblocks) {
        flush(R0 + i + 1);
        kb = 0; ++grp; seg0 = R0 + i + 1;
      }
    }
    if (ok && seg0 < R1) flush(R1);
  }
}

static int qg_groups(const QWeight& w) { return (w.n_tiles + QL_TILE_GROUP - 1) / QL_TILE_GROUP; }

// Persistent CTAs of the weight-streaming lane: a function of the weight's shape and the SM count only.
static int qg_ctas(const QWeight& w) {
  const long long T = (long long)qg_groups(w) * w.kblocks;
  // a run is at least QG_MIN_UNITS units, and long enough that a group's k-blocks spread over at most QG_MAX_PIECES
  // runs (each piece is one more fp32 partial the consumer kernel has to read)
  const long long run = std::max<long long>(QG_MIN_UNITS, (w.kblocks + QG_MAX_PIECES - 2) / (QG_MAX_PIECES - 1));
  return (int)std::max<long long>(1, std::min<long long>(T / run, (long long)QG_CTAS_PER_SM * w.sm_count));
}

int qlinear_stream_pieces(const QWeight& w) {
  const long long T = (long long)qg_groups(w) * w.kblocks, G = qg_ctas(w);
  int most = 1;
  for (int grp = 0; grp < qg_groups(w); ++grp) {
    const long long first = (long long)grp * w.kblocks;
    most = std::max(most, (int)(qg_owner(first + w.kblocks - 1, T, G) - qg_owner(first, T, G)) + 1);
  }
  return most;
}

template <int BITS, int GPK>
static cudaError_t launch_stream(const QgParams& p, int ctas, size_t smem, cudaStream_t s) {
  static DeviceOnce configured;
  if (configured.first_on_current_device()) {
    cudaError_t e = cudaFuncSetAttribute(qlinear_stream_kernel<BITS, GPK>, cudaFuncAttributeMaxDynamicSharedMemorySize, 110 * 1024);
    if (e != cudaSuccess) { configured.forget_current_device(); return e; }
  }
  return launch_k(qlinear_stream_kernel<BITS, GPK>, dim3(ctas), dim3(QG_THREADS), smem, s, p);
}

cudaError_t qlinear_stream(const QWeight& w, const bf16* x, int ldx, int M, float* partial, uint32_t* status, cudaStream_t s) {
  if (M < 1 || M > QL_STREAM_MAX_M || !partial) return cudaErrorInvalidValue;
  if ((ldx & 7) || (reinterpret_cast<uintptr_t>(x) & 15)) return cudaErrorInvalidValue;   // 16-byte activation loads
  QgParams p;
  p.records = w.records; p.record_bytes = w.record_bytes;
  p.N = w.N; p.n_groups = qg_groups(w); p.kblocks = w.kblocks; p.pieces = qlinear_stream_pieces(w);
  const size_t unit_bytes = (size_t)QL_TILE_GROUP * w.record_bytes;
  p.stages = (int)std::max<size_t>(2, std::min<size_t>(QG_MAX_STAGES, QG_RING_BYTES / unit_bytes));
  p.x = x; p.ldx = ldx; p.M = M; p.partial = partial; p.status = status;
  const size_t smem = (size_t)p.stages * unit_bytes + (size_t)w.kblocks * w.gpk * 8 * sizeof(float) + 2 * p.stages * sizeof(uint64_t);
  if (smem > 110 * 1024) return cudaErrorInvalidValue;
  const int ctas = qg_ctas(w);
  if (w.bits == 4) return w.gpk == 2 ? launch_stream<4, 2>(p, ctas, smem, s) : launch_stream<4, 1>(p, ctas, smem, s);
  return w.gpk == 2 ? launch_stream<8, 2>(p, ctas, smem, s) : launch_stream<8, 1>(p, ctas, smem, s);
}

// ---------------------------------------------------------------------------
// The small-weight lane of the same arithmetic: at most 8 rows against a weight of a few MB (the layers of a 1B-class
// draft model), where a launch is a chain of latencies and not a stream. One CTA = (tile, run of k-blocks); thread 0
// asks for ALL of the CTA's records with bulk copies onto one barrier before the kernel waits for its predecessor
// (weights depend on nothing), the activation slice of the run is staged once, and the eight warps (16 weight rows
// of the tile each) then work through records that are all resident, four at a time, with no ring and no hand-over.
// The k-blocks of a tile are cut into at most QV_MAX_PIECES runs — a function of the weight's shape and the SM count
// only — and leave fp32 partials [pieces][M][N] like the streaming kernel's, for the consumer kernel to sum in order.
// ---------------------------------------------------------------------------
constexpr int QV_WARPS = 8;
constexpr int QV_THREADS = QV_WARPS * 32;
constexpr int QV_MAX_PIECES = 8;
constexpr size_t QV_SMEM_BUDGET = 96 * 1024;   // two CTAs per SM

struct QvParams {
  const uint8_t* records;
  uint32_t record_bytes;
  int N, n_tiles, kblocks, c_used, kbper;
  const bf16* x;   // [M, ldx]
  int ldx, M;
  float* partial;  // [c_used][M][N]
  uint32_t* status;
  // Optional gated-activation operand: x is then not read; the activations are silu(gate) * up (gelu_approx for
  // glu == 2) of a gate_up output still in its fp32 partial form [gu_pieces][M][2 K] (K = this weight's input width).
  const float* gu;
  int gu_pieces, glu, gu_interleaved;
};

template <int BITS, int GPK>
__global__ void __launch_bounds__(QV_THREADS) qlinear_gemv_kernel(const QvParams p) {
  constexpr int ROW_BYTES = QL_KB * BITS / 8;
  constexpr int PACKED = QL_TILE_N * ROW_BYTES;
  constexpr int HALF_BYTES = QL_TILE_N * ROW_BYTES / 2;
  constexpr int LANE_WORDS = BITS / 4;
  constexpr int RB = BITS == 4 ? 4 : 2;               // records whose loads and MMA chains overlap
  extern __shared__ __align__(128) uint8_t smem[];
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = blockIdx.x / p.c_used, part = blockIdx.x - tile * p.c_used;
  const int kb0 = part * p.kbper, kb1 = min(p.kblocks, kb0 + p.kbper), nkb = kb1 - kb0;
  uint8_t* recs = smem;                                                     // [nkb][record_bytes]
  bf16* xs = reinterpret_cast<bf16*>(recs + (size_t)p.kbper * p.record_bytes);      // [8][kbper * 64]
  float* xsum = reinterpret_cast<float*>(xs + (size_t)8 * p.kbper * QL_KB);         // [kbper][GPK][8]
  uint64_t* bar = reinterpret_cast<uint64_t*>(xsum + (size_t)p.kbper * GPK * 8);   // one per batch of RB records
  const int n_batches = (nkb + RB - 1) / RB;
  if (threadIdx.x == 0) {
    for (int b = 0; b < n_batches; ++b) mbar_init(&bar[b], 1);
    mbar_fence_init();
    const uint8_t* src = p.records + ((size_t)(tile >> 2) * p.kblocks + kb0) * QL_TILE_GROUP * p.record_bytes + (size_t)(tile & 3) * p.record_bytes;
    for (int b = 0; b < n_batches; ++b) {
      const int in_batch = min(RB, nkb - b * RB);
      mbar_arrive_expect_tx(&bar[b], (uint32_t)in_batch * p.record_bytes);
      for (int i = b * RB; i < b * RB + in_batch; ++i, src += (size_t)QL_TILE_GROUP * p.record_bytes)
        bulk_g2s(recs + (size_t)i * p.record_bytes, src, p.record_bytes, &bar[b]);
    }
  }
  __syncthreads();
  pdl_wait();   // x comes from the kernel before; the partials below may still be read by it
  // the activation slice of this run, rows past M as zeros
  const int row_elems = p.kbper * QL_KB;
  for (int i = threadIdx.x; i < 8 * nkb * 8; i += QV_THREADS) {
    const int m = i / (nkb * 8), c8 = i - m * (nkb * 8);
    uint4 v = make_uint4(0, 0, 0, 0);
    if (m < p.M) {
      if (!p.gu) {
        v = *reinterpret_cast<const uint4*>(p.x + (size_t)m * p.ldx + (size_t)kb0 * QL_KB + c8 * 8);
      } else {
        // Mlp::forward's activation (nn.rs:284-294) on the way in: the arithmetic of glu_from_kernel
        const int F = p.kblocks * QL_KB, col = kb0 * QL_KB + c8 * 8;
        const int gcol = p.gu_interleaved ? (col >> 4) * 32 + (col & 15) : col;
        const int ucol = p.gu_interleaved ? gcol + 16 : F + col;
        const float* base = p.gu + (size_t)m * 2 * F;
        float4 g0 = *reinterpret_cast<const float4*>(base + gcol), g1 = *reinterpret_cast<const float4*>(base + gcol + 4);
        float4 u0 = *reinterpret_cast<const float4*>(base + ucol), u1 = *reinterpret_cast<const float4*>(base + ucol + 4);
        for (int k = 1; k < p.gu_pieces; ++k) {
          const float* pk = base + (size_t)k * p.M * 2 * F;
          const float4 a = *reinterpret_cast<const float4*>(pk + gcol), b = *reinterpret_cast<const float4*>(pk + gcol + 4);
          const float4 c = *reinterpret_cast<const float4*>(pk + ucol), d = *reinterpret_cast<const float4*>(pk + ucol + 4);
          g0.x += a.x; g0.y += a.y; g0.z += a.z; g0.w += a.w; g1.x += b.x; g1.y += b.y; g1.z += b.z; g1.w += b.w;
          u0.x += c.x; u0.y += c.y; u0.z += c.z; u0.w += c.w; u1.x += d.x; u1.y += d.y; u1.z += d.z; u1.w += d.w;
        }
        const float gv[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w}, uv[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
        float a[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
          a[k] = p.glu == 2 ? act_gelu_mul(bf16_round(gv[k]), bf16_round(uv[k])) : act_silu_mul(bf16_round(gv[k]), bf16_round(uv[k]));
        v = make_uint4(pack_bf162(a[0], a[1]), pack_bf162(a[2], a[3]), pack_bf162(a[4], a[5]), pack_bf162(a[6], a[7]));
      }
    }
    *reinterpret_cast<uint4*>(xs + (size_t)m * row_elems + c8 * 8) = v;
    // the sum of x per (k-block, scale group, row) in the same pass: the 64 / GPK features of a group are the chunks of
    // 8 / GPK neighbouring threads (the loop's trip count is a multiple of 64, so a warp is in it whole or not at all)
    const float2 e0 = unpack_bf162(v.x), e1 = unpack_bf162(v.y), e2 = unpack_bf162(v.z), e3 = unpack_bf162(v.w);
    float sx = ((e0.x + e0.y) + (e1.x + e1.y)) + ((e2.x + e2.y) + (e3.x + e3.y));
    sx += __shfl_xor_sync(0xffffffffu, sx, 1);
    sx += __shfl_xor_sync(0xffffffffu, sx, 2);
    if (GPK == 1) sx += __shfl_xor_sync(0xffffffffu, sx, 4);
    if ((c8 & (8 / GPK - 1)) == 0) xsum[(size_t)((c8 >> 3) * GPK + ((c8 & 7) >> (GPK == 1 ? 3 : 2))) * 8 + m] = sx;
  }
  __syncthreads();
  const int g = lane >> 2, t = lane & 3;
  const int r0 = warp * 16 + g;
  const uint32_t lane_off = lane_offset<BITS>(r0, t);
  const uint32_t sb_off = PACKED + (uint32_t)r0 * GPK * 4;
  const bf16* xrow = xs + (size_t)g * row_elems + 8 * t;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  for (int kbl = 0; kbl < nkb; kbl += RB) {
    const int nb = nkb - kbl < RB ? nkb - kbl : RB;
    // the batch's records have landed (the later batches are still on their way: copy and arithmetic overlap)
    if (!__all_sync(0xffffffffu, mbar_wait(&bar[kbl / RB], 0, p.status, KC_DEV_QLINEAR | 0x21))) {
      // gave up: the copies may still land in this CTA's shared memory; one more bounded wait for each of them
      for (int b = kbl / RB; b < n_batches; ++b) mbar_wait(&bar[b], 0, nullptr, 0);
      return;
    }
    uint4 xa[RB][2];
    float2 xsv[RB][GPK];
    uint32_t u[RB][2][2][LANE_WORDS];
    uint32_t sbw[RB][2][GPK];
#pragma unroll
    for (int i = 0; i < RB; ++i) {
      const int kk = kbl + (i < nb ? i : 0);
      const uint8_t* rc = recs + (size_t)kk * p.record_bytes;
#pragma unroll
      for (int h = 0; h < 2; ++h) xa[i][h] = *reinterpret_cast<const uint4*>(xrow + kk * QL_KB + 32 * h);
#pragma unroll
      for (int q = 0; q < GPK; ++q) xsv[i][q] = *reinterpret_cast<const float2*>(xsum + (size_t)(kk * GPK + q) * 8 + 2 * t);
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const uint8_t* src = rc + lane_off + r * 8 * 16 + h * HALF_BYTES;
          if (LANE_WORDS == 1) u[i][h][r][0] = *reinterpret_cast<const uint32_t*>(src);
          else { const uint2 v = *reinterpret_cast<const uint2*>(src); u[i][h][r][0] = v.x; u[i][h][r][LANE_WORDS - 1] = v.y; }
        }
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int q = 0; q < GPK; ++q) sbw[i][r][q] = *reinterpret_cast<const uint32_t*>(rc + sb_off + r * 8 * GPK * 4 + q * 4);
    }
    float raw[RB][2][4];
#pragma unroll
    for (int i = 0; i < RB; ++i) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        raw[i][h][0] = raw[i][h][1] = raw[i][h][2] = raw[i][h][3] = 0.f;
        uint32_t e0[4], e1[4];
        qg_raw_pairs<BITS>(u[i][h][0], e0);
        qg_raw_pairs<BITS>(u[i][h][1], e1);
        mma_bf16_16816(raw[i][h], e0[0], e1[0], e0[2], e1[2], xa[i][h].x, xa[i][h].z);
        mma_bf16_16816(raw[i][h], e0[1], e1[1], e0[3], e1[3], xa[i][h].y, xa[i][h].w);
      }
    }
    // the sums join the accumulator in k-block order: the result does not depend on RB
#pragma unroll
    for (int i = 0; i < RB; ++i) {
      if (i < nb) {
        if (GPK == 1) {
#pragma unroll
          for (int k = 0; k < 4; ++k) raw[i][0][k] += raw[i][1][k];
        }
#pragma unroll
        for (int q = 0; q < GPK; ++q) {
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const float sc = __uint_as_float(sbw[i][r][q] << 16), bi = __uint_as_float(sbw[i][r][q] & 0xFFFF0000u);
            const float bc = BITS == 4 ? fmaf(-128.f, sc, bi) : bi;   // the 128 every 4-bit q carries
            acc[2 * r + 0] = fmaf(sc, raw[i][q][2 * r + 0], fmaf(bc, xsv[i][q].x, acc[2 * r + 0]));
            acc[2 * r + 1] = fmaf(sc, raw[i][q][2 * r + 1], fmaf(bc, xsv[i][q].y, acc[2 * r + 1]));
          }
        }
      }
    }
  }
  // acc[0], [1] = weight row r0 against activation rows 2t, 2t + 1; [2], [3] = row r0 + 8
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int n = tile * QL_TILE_N + r0 + 8 * r;
    if (n < p.N) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int m = 2 * t + e;
        if (m < p.M) p.partial[((size_t)part * p.M + m) * p.N + n] = acc[2 * r + e];
      }
    }
  }
}

// The cut of a weight for the small-weight lane: runs of kbper k-blocks, c_used of them per tile.
struct QvPlan { bool ok; int c_used, kbper; size_t smem; };
static QvPlan qv_plan(const QWeight& w) {
  QvPlan q{false, 0, 0, 0};
  if (w.n_tiles < 1 || w.kblocks < 1) return q;
  const size_t per_kb = (size_t)w.record_bytes + 8 * QL_KB * sizeof(bf16) + (size_t)w.gpk * 8 * sizeof(float) + 8;   // + a barrier
  const int cap_kb = (int)((QV_SMEM_BUDGET - 64) / per_kb);
  if (cap_kb < 1) return q;
  // runs of about 8 k-blocks (a few microseconds of copy and arithmetic), fewer runs where the tiles alone fill the
  // SMs: every run is one more fp32 partial for the consumer kernel to read
  int c = std::max(1, std::min(QV_MAX_PIECES, w.kblocks / 8));
  c = std::min(c, std::max(1, 2 * w.sm_count / w.n_tiles));
  int kbper = std::min((w.kblocks + c - 1) / c, cap_kb);
  q.kbper = kbper;
  q.c_used = (w.kblocks + kbper - 1) / kbper;
  q.smem = (size_t)kbper * per_kb + 64;
  q.ok = q.c_used <= QV_MAX_PIECES;
  return q;
}

int qlinear_gemv_pieces(const QWeight& w) {
  const QvPlan q = qv_plan(w);
  return q.ok ? q.c_used : 0;
}

template <int BITS, int GPK>
static cudaError_t launch_gemv(const QvParams& p, int ctas, size_t smem, cudaStream_t s) {
  static DeviceOnce configured;
  if (configured.first_on_current_device()) {
    cudaError_t e = cudaFuncSetAttribute(qlinear_gemv_kernel<BITS, GPK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)QV_SMEM_BUDGET);
    if (e != cudaSuccess) { configured.forget_current_device(); return e; }
  }
  return launch_k(qlinear_gemv_kernel<BITS, GPK>, dim3(ctas), dim3(QV_THREADS), smem, s, p);
}

cudaError_t qlinear_gemv(const QWeight& w, const bf16* x, int ldx, int M, float* partial, uint32_t* status, cudaStream_t s,
                         const QvGatedInput* gated) {
  const QvPlan q = qv_plan(w);
  if (!q.ok || M < 1 || M > QL_STREAM_MAX_M || !partial) return cudaErrorInvalidValue;
  if (!gated && ((ldx & 7) || (reinterpret_cast<uintptr_t>(x) & 15))) return cudaErrorInvalidValue;   // 16-byte activation loads
  if (gated && (!gated->partial || gated->pieces < 1 || (reinterpret_cast<uintptr_t>(gated->partial) & 15) || (w.K & 127)))
    return cudaErrorInvalidValue;
  QvParams p;
  p.gu = gated ? gated->partial : nullptr; p.gu_pieces = gated ? gated->pieces : 0;
  p.glu = gated ? (gated->gelu ? 2 : 1) : 0; p.gu_interleaved = gated && gated->interleaved ? 1 : 0;
  p.records = w.records; p.record_bytes = w.record_bytes;
  p.N = w.N; p.n_tiles = w.n_tiles; p.kblocks = w.kblocks; p.c_used = q.c_used; p.kbper = q.kbper;
  p.x = x; p.ldx = ldx; p.M = M; p.partial = partial; p.status = status;
  const int ctas = w.n_tiles * q.c_used;
  if (w.bits == 4) return w.gpk == 2 ? launch_gemv<4, 2>(p, ctas, q.smem, s) : launch_gemv<4, 1>(p, ctas, q.smem, s);
  return w.gpk == 2 ? launch_gemv<8, 2>(p, ctas, q.smem, s) : launch_gemv<8, 1>(p, ctas, q.smem, s);
}

// ---------------------------------------------------------------------------
// Split-K reduction
// ---------------------------------------------------------------------------

// Pairs of neighbouring features go through 8-byte loads when every row of the partials and of y starts on the
// matching boundary (N, ldy even, bases aligned); otherwise one element per thread. The additions of an element are
// the same on both paths.
__global__ void qlinear_reduce_kernel(const float* __restrict__ partial, int splits, int M, int N,
                                      bf16* __restrict__ y, int ldy, int vec) {
  pdl_launch_dependents();
  pdl_wait();
  const long long stride = (long long)gridDim.x * blockDim.x;
  const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const size_t split_stride = (size_t)M * N;
  if (vec) {
    const long long total = (long long)M * N / 2;
    for (long long i = first; i < total; i += stride) {
      const long long e = i * 2;
      const int m = (int)(e / N), n = (int)(e % N);
      float2 acc = *reinterpret_cast<const float2*>(partial + e);
      for (int s = 1; s < splits; ++s) {
        const float2 v = *reinterpret_cast<const float2*>(partial + s * split_stride + e);
        acc.x += v.x; acc.y += v.y;
      }
      *reinterpret_cast<bf162*>(y + (size_t)m * ldy + n) = __floats2bfloat162_rn(acc.x, acc.y);
    }
  } else {
    const long long total = (long long)M * N;
    for (long long e = first; e < total; e += stride) {
      const int m = (int)(e / N), n = (int)(e % N);
      float acc = partial[e];
      for (int s = 1; s < splits; ++s) acc += partial[s * split_stride + e];
      y[(size_t)m * ldy + n] = __float2bfloat16_rn(acc);
    }
  }
}

// The reduction of ONE row fused with its raw arg-max (the head of a draft model's chained step, draft.rs:379-381:
// argmax of the logits row, lowest index on ties): every CTA sums its slice of the pieces in index order, rounds to
// bf16 (the head's output, also stored to y), keeps the best of its slice, and the CTA that finishes last — counted
// with one atomic per CTA, nobody waits — takes the best over the CTAs and stores the token. scratch: 2 floats per
// CTA followed by one counter word that is zero between launches (the last CTA resets it).
__global__ void __launch_bounds__(256) qlinear_reduce_argmax_kernel(const float* __restrict__ partial, int splits, int N,
                                                                    bf16* __restrict__ y, float* __restrict__ scratch,
                                                                    uint32_t* __restrict__ token, uint32_t* __restrict__ token_host) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float s_v[8];
  __shared__ int s_i[8];
  __shared__ bool s_last;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto better = [](float av, int ai, float bv, int bi) { return bv > av || (bv == av && bi < ai); };
  float best_v = -INFINITY;
  int best_i = 0x7fffffff;
  for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < N; n += gridDim.x * blockDim.x) {
    float acc = partial[n];
    for (int k = 1; k < splits; ++k) acc += partial[(size_t)k * N + n];
    const bf16 r = __float2bfloat16_rn(acc);
    y[n] = r;
    const float v = __bfloat162float(r);
    if (better(best_v, best_i, v, n)) { best_v = v; best_i = n; }
  }
  auto reduce_block = [&]() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best_v, o);
      const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
      if (better(best_v, best_i, ov, oi)) { best_v = ov; best_i = oi; }
    }
    if (lane == 0) { s_v[warp] = best_v; s_i[warp] = best_i; }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
        if (better(best_v, best_i, s_v[w], s_i[w])) { best_v = s_v[w]; best_i = s_i[w]; }
    }
  };
  reduce_block();
  uint32_t* counter = reinterpret_cast<uint32_t*>(scratch + 2 * gridDim.x);
  if (threadIdx.x == 0) {
    scratch[2 * blockIdx.x] = best_v;
    scratch[2 * blockIdx.x + 1] = __int_as_float(best_i);
    __threadfence();
    s_last = atomicAdd(counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  best_v = -INFINITY; best_i = 0x7fffffff;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) {
    const float v = __ldcg(scratch + 2 * b);
    const int i = __float_as_int(__ldcg(scratch + 2 * b + 1));
    if (better(best_v, best_i, v, i)) { best_v = v; best_i = i; }
  }
  __syncthreads();   // s_v / s_i are reused
  reduce_block();
  if (threadIdx.x == 0) {
    const uint32_t tok = (uint32_t)best_i < (uint32_t)N ? (uint32_t)best_i : 0u;   // a row of NaNs has no maximum
    *token = tok;
    if (token_host) *token_host = tok;
    *counter = 0u;
  }
}

int qlinear_reduce_argmax_ctas(int N) { return std::max(1, std::min((N + 511) / 512, 296)); }

cudaError_t qlinear_reduce_argmax(const float* partial, int splits, int N, bf16* y, float* scratch, uint32_t* token, uint32_t* token_host,
                                  cudaStream_t s) {
  if (!partial || !y || !scratch || !token || splits < 1 || N < 1) return cudaErrorInvalidValue;
  return launch_k(qlinear_reduce_argmax_kernel, dim3(qlinear_reduce_argmax_ctas(N)), dim3(256), 0, s, partial, splits, N, y, scratch, token, token_host);
}

cudaError_t qlinear_reduce_splits(const float* partial, int splits, int M, int N, bf16* y, int ldy,
                                  cudaStream_t s) {
  const int vec = (N % 2 == 0 && ldy % 2 == 0 && (reinterpret_cast<uintptr_t>(partial) & 7) == 0 &&
                   (reinterpret_cast<uintptr_t>(y) & 3) == 0) ? 1 : 0;
  const long long total = vec ? (long long)M * N / 2 : (long long)M * N;
  const int threads = 256;
  const int blocks = (int)std::max<long long>(1, std::min<long long>((total + threads - 1) / threads, 148LL * 8));
  return launch_k(qlinear_reduce_kernel, dim3(blocks), dim3(threads), 0, s, partial, splits, M, N, y, ldy, vec);
}

}  // namespace kc

