// Affine-dequant GEMM for sm_100a. See kc_qlinear.cuh for the data layout.
//
// qlinear_umma_ta_kernel — one CTA per (one or two 128-row weight tiles, k-split), 20 warps:
//   warp 0      bulk-copies the weight records (cp.async.bulk, mbarrier tx)
//   warp 1      TMA-loads the activation k-blocks (cp.async.bulk.tensor, 128B swizzle)
//   warps 2-3   allocate TMEM, issue tcgen05.mma (weights = A/M side from TENSOR MEMORY, activations = B/N side
//               from shared memory), each into an accumulator of its own: nothing orders them to each other
//   warps 4-19  unpack the 4/8-bit words, apply scale/bias in registers and write the bf16 A operand into tensor
//               memory with tcgen05.st; afterwards drain the accumulators (tcgen05.ld) into y, the split-K
//               partials or the gated activation.
// The accumulator D[n, m] lives in TMEM: lane = weight row n, column = activation row m.
// Every output element depends only on its own activation row and on a k order
// fixed by (N, K), which is what lets verify rows share a step with other rows
// and still reproduce the bits of a one-row decode. More rows than one accumulator set holds are cut into chunks of
// rows (blockIdx.z): rows are independent, so no bit changes.
#include "kc_qlinear.cuh"
#include "kc_umma.cuh"

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <cstdlib>

namespace kc {

// ---------------------------------------------------------------------------
// Re-tiling
// ---------------------------------------------------------------------------

// Scales below this limit can be multiplied by 2^129 (4-bit) or 2^133 (8-bit) within bf16: see dequant_row.
__host__ __device__ constexpr float ql_scale_limit(int bits) { return bits == 4 ? 0.5f : 0.03125f; }

__global__ void qweight_retile_kernel(uint8_t* __restrict__ records, const uint32_t* __restrict__ w,
                                      const bf16* __restrict__ scales, const bf16* __restrict__ biases,
                                      int N, int K, int bits, int group, int n_tiles, int kblocks,
                                      int gpk, uint32_t packed_bytes, uint32_t record_bytes, int* __restrict__ wide) {
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
      if (n < N) v = w[(long long)n * src_words_per_row + kb * words_per_row_kb + c];
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
        sb.x = scales[(long long)n * groups_per_row + g];
        sb.y = biases[(long long)n * groups_per_row + g];
        if (!(fabsf(__bfloat162float(sb.x)) < ql_scale_limit(bits))) *wide = 1;
      }
      reinterpret_cast<bf162*>(base + packed_bytes)[e2] = sb;
    }
  }
}

int qlinear_plan_splits(int n_tiles, int kblocks, int sm_count) {
  // As many k-splits as fill the SMs with one-tile CTAs, each keeping at least 8 k-blocks; none when two-tile CTAs
  // already fill them. Splits need not divide the k-blocks evenly (the kernel cuts [K s / S, K (s + 1) / S)).
  if (n_tiles * 2 >= sm_count) return 1;
  int s = sm_count / n_tiles;
  s = std::min(s, std::min(16, kblocks / 8));
  return std::max(s, 1);
}

cudaError_t qweight_build(QWeight* out, const uint32_t* w, const bf16* scales, const bf16* biases,
                          int N, int K, int bits, int group, int sm_count, cudaStream_t s) {
  QWeight q;
  q.N = N; q.K = K; q.bits = bits; q.group = group;
  q.n_tiles = (N + QL_TILE_N - 1) / QL_TILE_N;
  q.kblocks = K / QL_KB;
  q.gpk = std::max(1, QL_KB / group);
  q.packed_bytes = QL_TILE_N * (QL_KB * bits / 8);
  q.record_bytes = q.packed_bytes + QL_TILE_N * q.gpk * 4;
  q.splits = qlinear_plan_splits(q.n_tiles, q.kblocks, sm_count);
  q.sm_count = sm_count;
  // one allocation: the records, then a flag that the re-tiling raises
  cudaError_t e = cudaMalloc(&q.records, q.bytes() + 16);
  if (e != cudaSuccess) return e;
  q.wide = reinterpret_cast<int*>(q.records + q.bytes());
  e = cudaMemsetAsync(q.wide, 0, 16, s);
  if (e != cudaSuccess) { cudaFree(q.records); return e; }
  const long long total = (long long)(q.bytes() / 4);
  const int threads = 256;
  const int blocks = (int)std::min<long long>((total + threads - 1) / threads, 148LL * 16);
  qweight_retile_kernel<<<blocks, threads, 0, s>>>(q.records, w, scales, biases, N, K, bits, group,
                                                   q.n_tiles, q.kblocks, q.gpk, q.packed_bytes,
                                                   q.record_bytes, q.wide);
  e = cudaGetLastError();
  if (e != cudaSuccess) { cudaFree(q.records); return e; }
  *out = q;
  return cudaSuccess;
}

cudaError_t qweight_finish(QWeight* w) {
  return cudaMemcpy(&w->wide_scale, w->wide, sizeof(int), cudaMemcpyDeviceToHost);
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
static const CUtensorMap* act_operand_rows_map(const ActOperand* op, int m_pad) {
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
// Dequantisation of one weight row of one k-block: 64 values -> 32 bf16 pairs, w = bf16(q * scale + bias), one rounding.
//
// The dequantisers' instruction issue is what bounds a launch of few rows, so the integers become bf16 operands of the
// multiply-add without a conversion: the bf16 with bit pattern N < 256 is N * 2^-133 (subnormals and the first binade
// have the same spacing), so a nibble masked into bits 4..7 of a half-word IS q * 2^-129 and a byte in bits 0..7 IS
// q * 2^-133. One fused multiply-add with the scale times 2^129 (2^133: exact, a power of two) gives q * scale + bias
// rounded once — the value that converting q first gives. 11 instructions for 8 weights instead of 15 (4 bits), 2 for
// 2 instead of 7 (8 bits). The scaled scale must stay below 2^128: a weight with a scale of ql_scale_limit or more
// (its `wide` flag, raised when it is re-tiled) takes the conversion.
// ---------------------------------------------------------------------------

__device__ __forceinline__ uint32_t bf2_fma(uint32_t a, bf162 s, bf162 b) {
  const bf162 r = __hfma2(*reinterpret_cast<const bf162*>(&a), s, b);
  return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ bf162 bf2_bits(uint32_t u) { return *reinterpret_cast<const bf162*>(&u); }
// (scale, scale) times 2^129 or 2^133, in two exact steps (neither power of two is a bf16)
template <int BITS>
__device__ __forceinline__ bf162 scaled_scale(bf162 sb) {
  const bf162 s = __hmul2(__bfloat162bfloat162(sb.x), bf2_bits(0x7F007F00u));              // 2^127
  return __hmul2(s, BITS == 4 ? bf2_bits(0x40804080u) : bf2_bits(0x42804280u));            // 2^2, 2^6
}

// Packed words of a row (chunk c = 16 bytes at row_base + c * QL_TILE_N * 16) -> v[32].
template <int BITS, int GPK>
__device__ __forceinline__ void dequant_row(const uint8_t* row_base, const bf162 (&sb)[GPK], uint32_t (&v)[32]) {
  constexpr int CHUNKS = BITS / 2;
  bf162 s2[GPK], b2[GPK];
#pragma unroll
  for (int g = 0; g < GPK; ++g) { s2[g] = scaled_scale<BITS>(sb[g]); b2[g] = __bfloat162bfloat162(sb[g].y); }
#pragma unroll
  for (int h = 0; h < CHUNKS; ++h) {
    const uint4 q = *reinterpret_cast<const uint4*>(row_base + h * (QL_TILE_N * 16));
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
    const int g = GPK == 2 ? h * 2 / CHUNKS : 0;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (BITS == 4) {
        // the record's nibble order: element 2j at bits 4j, element 2j + 1 at bits 16 + 4j
        uint32_t* o = v + (h * 4 + c) * 4;
        o[0] = bf2_fma((w[c] << 4) & 0x00F000F0u, s2[g], b2[g]);
        o[1] = bf2_fma(w[c] & 0x00F000F0u, s2[g], b2[g]);
        o[2] = bf2_fma((w[c] >> 4) & 0x00F000F0u, s2[g], b2[g]);
        o[3] = bf2_fma((w[c] >> 8) & 0x00F000F0u, s2[g], b2[g]);
      } else {
        uint32_t* o = v + (h * 4 + c) * 2;
        o[0] = bf2_fma(__byte_perm(w[c], 0u, 0x4140u), s2[g], b2[g]);
        o[1] = bf2_fma(__byte_perm(w[c], 0u, 0x4342u), s2[g], b2[g]);
      }
    }
  }
}

// The same for a weight with a scale past the limit: the integers are converted first (exact: at most 8 bits), the
// multiply-add is the same one with its one rounding.
template <int BITS, int GPK>
__device__ __forceinline__ void dequant_row_wide(const uint8_t* row_base, const bf162 (&sb)[GPK], uint32_t (&v)[32]) {
  constexpr int CHUNKS = BITS / 2;
#pragma unroll
  for (int h = 0; h < CHUNKS; ++h) {
    const uint4 q = *reinterpret_cast<const uint4*>(row_base + h * (QL_TILE_N * 16));
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
    const int g = GPK == 2 ? h * 2 / CHUNKS : 0;
    const bf162 s2 = __bfloat162bfloat162(sb[g].x), b2 = __bfloat162bfloat162(sb[g].y);
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int j = 0; j < 16 / BITS; ++j) {
        const uint32_t lo = BITS == 4 ? (w[c] >> (4 * j)) & 0xFu : (w[c] >> (16 * j)) & 0xFFu;
        const uint32_t hi = BITS == 4 ? (w[c] >> (16 + 4 * j)) & 0xFu : (w[c] >> (16 * j + 8)) & 0xFFu;
        v[(h * 4 + c) * (16 / BITS) + j] = bf2_fma(pack_bf162((float)lo, (float)hi), s2, b2);
      }
  }
}

// ---------------------------------------------------------------------------
// tcgen05 helpers (the others are in kc_umma.cuh)
// ---------------------------------------------------------------------------

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  tmem_ld16_issue(taddr, r);
  tmem_wait_ld();
}

// ---------------------------------------------------------------------------
// The kernel
// ---------------------------------------------------------------------------

constexpr int QL_DQ_WARP0 = 4;         // first dequant/epilogue warp
constexpr int QL_DQ_GROUPS = 4;        // dequant groups of four warps (the four TMEM lane quarters)
constexpr int QL_DQ_WARPS = QL_DQ_GROUPS * 4;
constexpr int QL_THREADS = (QL_DQ_WARP0 + QL_DQ_WARPS) * 32;   // 20 warps
constexpr int QL_EPI_STAGE_BYTES = 32 * 32 * 4;   // per-warp transpose buffer of the epilogue

struct QlKernelParams {
  const uint8_t* records;
  uint32_t record_bytes;
  int N, n_tiles, kblocks;
  int M, m_pad;          // live rows of the launch; rows of a chunk (blockIdx.z), a multiple of 16
  int row0;              // first activation row
  int splits;
  int a_stages, r_stages, b_stages;   // ring depths: stages in TMEM, k-blocks of records and stages of activations in shared memory
  int glu;               // 0, or 1 (silu) / 2 (gelu_approx): the epilogue writes act = activation(gate tile) * up tile
  bf16* act; int ld_act;
  uint32_t tmem_cols;    // columns allocated: a power of two
  bf16* y; int ldy;
  float* partial;        // [splits][M][N]
  int chunks;            // of rows (qlinear_umma_rows_kernel)
  uint32_t* status;
};

// The epilogue shared by the GEMM kernels: every epilogue warp drains its TMEM lane quarter, 32 columns (rows of the
// step) at a time, transposes through a private 4 KB shared buffer and stores row-contiguous vectors: bf16 y, fp32
// split-K partials, or — when the CTA owns (gate, up) tile pairs — the gated activation.
template <int NT>
__device__ __forceinline__ void ql_epilogue(const QlKernelParams& p, uint8_t* smem, int warp, int lane, uint32_t tmem_base,
                                            int tile0, int nt_live, int split, int chunk0, bool two_sums) {
  tc_fence_after();
  // every MMA has completed and every copy into the rings has been consumed: the ring memory is free
  float* stage = reinterpret_cast<float*>(smem + (size_t)(warp - QL_DQ_WARP0) * QL_EPI_STAGE_BYTES);
  const int q = warp & 3;                        // TMEM lane quarter this warp may read
  const int eg = (warp - QL_DQ_WARP0) >> 2;      // warps of one quarter split the 32-column chunks
  const int chunks = (p.m_pad + 31) >> 5;
  const int col_stride = (p.m_pad + 31) & ~31;
  const bool vec_ok = p.splits == 1 ? ((p.ldy & 3) == 0 && (reinterpret_cast<uintptr_t>(p.y) & 7) == 0)
                                    : ((p.N & 3) == 0 && (reinterpret_cast<uintptr_t>(p.partial) & 15) == 0);
  const int nl = 4 * (lane & 7), mr0 = lane >> 3;
  if (NT >= 2 && p.glu) {
    // tiles (2 pr, 2 pr + 1) of this CTA are the gate and up halves of features 128 * (tile0 / 2 + pr) ..:
    // both accumulators' values of a (feature, row) sit in the same thread, 16 rows at a time
    const int chunks16 = p.m_pad >> 4;
    for (int item = eg; item < (nt_live >> 1) * chunks16; item += QL_DQ_WARPS / 4) {
      const int pr = item / chunks16, ch = item - pr * chunks16;
      uint32_t g[16], u[16];
      tmem_ld16(tmem_base + ((uint32_t)(q * 32) << 16) + (2 * pr) * col_stride + ch * 16, g);
      tmem_ld16(tmem_base + ((uint32_t)(q * 32) << 16) + (2 * pr + 1) * col_stride + ch * 16, u);
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float gv = bf16_round(__uint_as_float(g[j])), uv = bf16_round(__uint_as_float(u[j]));
        stage[j * 32 + lane] = p.glu == 2 ? act_gelu_mul(gv, uv) : act_silu_mul(gv, uv);
      }
      __syncwarp();
      const int f = ((tile0 >> 1) + pr) * QL_TILE_N + q * 32 + nl;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int mr = 4 * k + mr0;
        const int m = chunk0 + ch * 16 + mr;
        if (m >= p.M) continue;
        const float4 v4 = *reinterpret_cast<const float4*>(stage + mr * 32 + nl);
        *reinterpret_cast<uint2*>(p.act + (size_t)(p.row0 + m) * p.ld_act + f) =
            make_uint2(pack_bf162(v4.x, v4.y), pack_bf162(v4.z, v4.w));
      }
    }
  } else
  for (int item = eg; item < nt_live * chunks; item += QL_DQ_WARPS / 4) {
    const int t = item / chunks, ch = item - t * chunks;
    const int col = t * col_stride + ch * 32;
    uint32_t v[32];
    tmem_ld32(tmem_base + ((uint32_t)(q * 32) << 16) + col, v);
    if (NT == 1 && two_sums) {                   // even plus odd k-blocks
      uint32_t w[32];
      tmem_ld32(tmem_base + ((uint32_t)(q * 32) << 16) + col + col_stride, w);
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(w[j]));
    }
    __syncwarp();                                // the previous item's reads of the buffer are done
#pragma unroll
    for (int j = 0; j < 32; ++j) stage[j * 32 + lane] = __uint_as_float(v[j]);   // stage[m][n]
    __syncwarp();
    const int n = (tile0 + t) * QL_TILE_N + q * 32 + nl;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int mr = 4 * k + mr0;
      const int mc = ch * 32 + mr, m = chunk0 + mc;
      if (mc >= p.m_pad || m >= p.M || n >= p.N) continue;
      const float4 f = *reinterpret_cast<const float4*>(stage + mr * 32 + nl);
      if (p.splits == 1) {
        bf16* dst = p.y + (size_t)(p.row0 + m) * p.ldy + n;
        if (vec_ok && n + 3 < p.N) {
          *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf162(f.x, f.y), pack_bf162(f.z, f.w));
        } else {
          const float e[4] = {f.x, f.y, f.z, f.w};
          for (int c = 0; c < 4 && n + c < p.N; ++c) dst[c] = __float2bfloat16_rn(e[c]);
        }
      } else {
        float* dst = p.partial + ((size_t)split * p.M + m) * p.N + n;
        if (vec_ok && n + 3 < p.N) {
          *reinterpret_cast<float4*>(dst) = f;
        } else {
          const float e[4] = {f.x, f.y, f.z, f.w};
          for (int c = 0; c < 4 && n + c < p.N; ++c) dst[c] = e[c];
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// The kernel. The dequantised weights reach the tensor core through TENSOR MEMORY (tcgen05.mma with the A operand in
// TMEM), not through shared memory: an M = 128, N = 192 MMA needs 97 cycles when run alone, but a kernel that staged the
// bf16 weights in shared memory took about 1140 cycles per k-block of eight of them, the time its 154 KB of
// shared-memory traffic takes. A dequantiser thread owns one weight row (= one TMEM lane) of one UNIT — one 128-row tile
// of one 64-feature k-block —, expands its 64 weights in registers and writes them with one tcgen05.st (column c =
// weights 2c and 2c + 1), so the MMAs read only the activation k-block from shared memory.
//
// What bounds it: at few rows (an MMA then takes 46 cycles whatever its N) the dequantisers' instruction issue and the
// hand-overs; from about 128 rows on the tensor pipe, 4 * N / 2 cycles per unit. Hence: four groups of four warps, each
// converting every fourth unit on its own; and two accumulators, each with an issuing WARP and a ring of A slots of its
// own — the CTA's two tiles, or the even and the odd k-blocks of its one tile, summed in the epilogue. A stage is one
// unit of each. An issuing warp runs its loop converged with one elected lane around the MMAs: with `if (lane == 0)`
// around the loop the operands of each MMA went through vector registers and eight MMAs took 700 cycles to issue.
// 28672 x 4096 in 4 bits, 112 CTAs, every launch from HBM: 35.7 us -> 21 us at 1 row, 40.7 -> 37 us at 192 rows.
//
// The order in which an element's k-blocks are accumulated is a function of the weight's shape only.
//
// TMEM columns: [2 accumulators of round32(m_pad)] [a_stages x 2 units x 32 columns of bf16 pairs].
// ---------------------------------------------------------------------------
template <int BITS, int GPK, int NT, int P, bool WIDE>
__global__ void __launch_bounds__(QL_THREADS, 1)
qlinear_umma_ta_kernel(const __grid_constant__ CUtensorMap map_rows, const QlKernelParams p) {
  constexpr int KC = NT == 1 ? 2 : 1;                   // slots of records and activations in a stage (see below)
  constexpr uint32_t PACKED = QL_TILE_N * (QL_KB * BITS / 8);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int SA = p.a_stages, SB = p.b_stages;
  const uint32_t b_bytes = (uint32_t)p.m_pad * 128u;    // one activation k-block
  const uint32_t r_bytes = NT * p.record_bytes;         // the records of one k-block
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int tile0 = blockIdx.x * NT, split = blockIdx.y, chunk0 = blockIdx.z * p.m_pad;
  const int nt_live = min(NT, p.n_tiles - tile0);
  // splits may be uneven: split s takes k-blocks [K s / S, K (s + 1) / S) — a fixed function of the weight's shape
  const int kb0 = (int)((long long)p.kblocks * split / p.splits);
  const int nkb = (int)((long long)p.kblocks * (split + 1) / p.splits) - kb0;
  // Ring depths: a group visits every second stage, and it must meet every fill of the slots it waits on (a wait names a
  // fill by its parity only), so r_stages is a multiple of 2 * KC k-blocks and a_stages of 2.
  const int RS = p.r_stages;
  // A slot holds the P k-blocks of one unit per tile: two tiles: slot n has k-blocks P n ..; one tile: slot 2 j + u has
  // k-blocks 2 P j + u, 2 P j + u + 2, .. of accumulator u. own(u): k-blocks of accumulator u.
  auto own = [&](int u) { return NT == 2 ? nkb : (nkb + 1 - u) / 2; };
  const int n_slots = NT == 2 ? (nkb + P - 1) / P : (own(0) + P - 1) / P + (own(1) + P - 1) / P;
  auto slot_kb = [&](int n) { return NT == 2 ? P * n : 2 * P * (n >> 1) + (n & 1); };
  auto slot_live = [&](int n) { return NT == 2 ? min(P, nkb - P * n) : min(P, own(n & 1) - P * (n >> 1)); };
  const uint32_t col_stride = (uint32_t)(p.m_pad + 31) & ~31u;
  const uint32_t a_col0 = 2 * col_stride;               // first column of the A ring

  uint8_t* sB = smem;
  uint8_t* sR = sB + (size_t)SB * P * b_bytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sR + (size_t)RS * P * r_bytes);
  uint64_t* raw_full = bars;
  uint64_t* raw_empty = raw_full + RS;
  uint64_t* b_full = raw_empty + RS;
  uint64_t* b_empty = b_full + SB;
  uint64_t* a_ready = b_empty + SB;
  uint64_t* a_empty = a_ready + 2 * SA;                 // [stage][unit], like a_ready
  uint64_t* acc_full = a_empty + 2 * SA;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);

  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int i = 0; i < RS; ++i) { mbar_init(&raw_full[i], 1); mbar_init(&raw_empty[i], 4 * nt_live); }
    for (int i = 0; i < SB; ++i) { mbar_init(&b_full[i], 1); mbar_init(&b_empty[i], nt_live); }
    for (int i = 0; i < 2 * SA; ++i) { mbar_init(&a_ready[i], 4); mbar_init(&a_empty[i], 1); }
    mbar_init(acc_full, NT == 1 ? 2 : nt_live);   // each issuer commits to it after its last MMA
    mbar_fence_init();
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(p.tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (warp == 1 && lane == 0) tma_prefetch_desc(&map_rows);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ---- weight record producer: weights depend on no kernel before this one ----
    if (lane == 0) {
      RingPos rp;
      const uint8_t* src = p.records + (((size_t)(tile0 / QL_TILE_GROUP) * p.kblocks + kb0) * QL_TILE_GROUP + tile0 % QL_TILE_GROUP) * p.record_bytes;
      const uint32_t bytes = p.record_bytes * nt_live;
      const size_t kb_pitch = (size_t)QL_TILE_GROUP * p.record_bytes;
      for (int i = 0; i < n_slots; ++i, rp.advance(RS)) {
        if (!mbar_wait(&raw_empty[rp.stage], rp.phase ^ 1, p.status, KC_DEV_QLINEAR | 1)) break;
        const int live = slot_live(i);
        const uint8_t* from = src + slot_kb(i) * kb_pitch;
        mbar_arrive_expect_tx(&raw_full[rp.stage], bytes * live);
#pragma unroll
        for (int q = 0; q < P; ++q)
          if (q < live) bulk_g2s(sR + (size_t)(rp.stage * P + q) * r_bytes, from + q * KC * kb_pitch, bytes, &raw_full[rp.stage]);
      }
    }
  } else if (warp == 1) {
    // ---- activation producer: the first access of this kernel to memory written by earlier kernels ----
    if (lane == 0) {
      pdl_wait();
      RingPos bp;
      for (int i = 0; i < n_slots; ++i, bp.advance(SB)) {
        if (!mbar_wait(&b_empty[bp.stage], bp.phase ^ 1, p.status, KC_DEV_QLINEAR | 2)) break;
        const int live = slot_live(i), kb = kb0 + slot_kb(i);
        mbar_arrive_expect_tx(&b_full[bp.stage], b_bytes * live);
#pragma unroll
        for (int q = 0; q < P; ++q)
          if (q < live)
            tma_load_2d(sB + (size_t)(bp.stage * P + q) * b_bytes, &map_rows, (kb + q * KC) * QL_KB, p.row0 + chunk0, &b_full[bp.stage]);
      }
    }
  } else if (warp < QL_DQ_WARP0) {
    // ---- MMA issuers: warp 2 + u issues the MMAs of unit u of every stage into accumulator u. The whole warp runs the
    // loop, one elected lane issues. The two never touch the same accumulator, so nothing orders them to each other.
    // A barrier test takes about 130 cycles from issue to branch, as long as the issue of four MMAs: the next stage's
    // barriers are tested before this stage's MMAs issue, and only a stage that was not ready then waits.
    pdl_wait();
    const int u = warp - 2;
    if (NT == 1 || u < nt_live) {
      const uint32_t idesc = umma_idesc_bf16(QL_TILE_N, p.m_pad);
      const uint64_t proto = umma_smem_desc(0, 1024);
      const uint32_t d_hi = (uint32_t)(proto >> 32), b_lo0 = (uint32_t)proto | ((smem_u32(sB) >> 4) & 0x3FFF);
      const uint32_t d_t = tmem_base + u * col_stride, a_t0 = tmem_base + a_col0 + u * 32 * P;
      const int left0 = own(u), n_own = (left0 + P - 1) / P;   // k-blocks and units of this accumulator
      int as = 0, bs = NT == 2 ? 0 : u;                     // ring positions of the next one
      uint32_t aphase = 0, bphase = 0, acc = 0;
      bool ok = true, ready = false;
      for (int i = 0; i < n_own; ++i) {
        if (!__all_sync(0xffffffffu, ready)) {
          ok = warp_wait(&b_full[bs], bphase, p.status, KC_DEV_QLINEAR | 4) &&
               warp_wait(&a_ready[2 * as + u], aphase, p.status, KC_DEV_QLINEAR | 3);
          if (!ok) break;
        }
        tc_fence_after();   // the A operand was written with tcgen05.st by other threads
        const uint32_t b_lo = b_lo0 + bs * P * (b_bytes >> 4), a_t = a_t0 + as * (64 * P);
        uint64_t *a_done = &a_empty[2 * as + u], *b_done = &b_empty[bs];
        if (++as == SA) { as = 0; aphase ^= 1u; }
        bs += KC;
        if (bs >= SB) { bs -= SB; bphase ^= 1u; }
        ready = i + 1 < n_own && (mbar_test_wait(&b_full[bs], bphase) & mbar_test_wait(&a_ready[2 * as + u], aphase));
        const int live = left0 - P * i;
        if (elect_one()) {
#pragma unroll
          for (int q = 0; q < P; ++q) {
            if (q > 0 && q >= live) break;
#pragma unroll
            for (int ks = 0; ks < QL_KB / 16; ++ks)
              umma_bf16_ts(d_t, a_t + 32 * q + 8 * ks, b_lo + q * (b_bytes >> 4) + 2 * ks, d_hi, idesc, q == 0 && ks == 0 ? acc : 1u);
          }
          umma_commit(a_done);
          umma_commit(b_done);
        }
        __syncwarp();
        acc = 1;
      }
      if (ok && elect_one()) umma_commit(acc_full);
      __syncwarp();
    }
  } else if (warp >= QL_DQ_WARP0) {
    // ---- dequantisers: thread = one weight row (TMEM lane 32 * (warp % 4) + lane) of every fourth unit ----
    // Group g converts unit g & 1 of the stages g >> 1, (g >> 1) + 2, ...
    const int grp = (warp - QL_DQ_WARP0) >> 2, unit = grp & 1;
    const int row = (warp & 3) * 32 + lane;
    const uint32_t a_addr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + a_col0 + unit * 32 * P;
    const int tile = NT == 2 ? unit : 0;
    const uint8_t* row_raw = sR + (size_t)tile * p.record_bytes + row * 16;
    const uint8_t* row_sb = sR + (size_t)tile * p.record_bytes + PACKED + row * (GPK * 4);
    int rs = NT == 2 ? grp >> 1 : (grp >> 1) * 2 + unit, as = grp >> 1;   // ring positions of the group's next unit
    constexpr int R_STEP = 2 * KC;                      // slots between a group's units
    uint32_t rphase = 0, aphase = 0;
    const int left0 = NT == 2 && unit >= nt_live ? 0 : own(unit), units = (left0 + P - 1) / P;   // units: one per stage
    bool ok = true, released = false, raw_ready = false;
    for (int i = grp >> 1; i < units; i += 2) {
      // the first SA stages are dequantised under the tail of the previous kernel; a slot that is being reused is freed
      // by an MMA, which needs activations, which need the previous kernel: the bounded wait for it counts from there
      if (!released && i >= SA) { pdl_wait(); released = true; }
      if (!__all_sync(0xffffffffu, raw_ready)) {
        ok = warp_wait(&raw_full[rs], rphase, p.status, KC_DEV_QLINEAR | 5);
        if (!ok) break;
      }
      // the slot's barrier is tested under the arithmetic, the next record's under the store (see the issuers)
      const bool a_free = mbar_test_wait(&a_empty[2 * as + unit], aphase ^ 1);
      const uint32_t a_slot = a_addr + as * (64 * P);
      const int live = left0 - P * i;
#pragma unroll
      for (int q = 0; q < P; ++q) {
        if (q > 0 && q >= live) break;
        const size_t at = (size_t)(rs * P + q) * r_bytes;
        uint32_t v[32];
        bf162 sb[GPK];
        if (GPK == 1) {
          sb[0] = *reinterpret_cast<const bf162*>(row_sb + at);
        } else {
          const uint2 s = *reinterpret_cast<const uint2*>(row_sb + at);
          sb[0] = bf2_bits(s.x); sb[GPK - 1] = bf2_bits(s.y);
        }
        if (!WIDE) dequant_row<BITS, GPK>(row_raw + at, sb, v);
        else dequant_row_wide<BITS, GPK>(row_raw + at, sb, v);
        if (q == 0) {
          if (!__all_sync(0xffffffffu, a_free)) ok = warp_wait(&a_empty[2 * as + unit], aphase ^ 1, p.status, KC_DEV_QLINEAR | 6);
          if (!ok) break;
          tc_fence_after();
        }
        tmem_st32(a_slot + 32 * q, v);
      }
      if (!ok) break;
      __syncwarp();
      if (lane == 0) mbar_arrive(&raw_empty[rs]);       // the records are in registers: their slot can refill
      rs += R_STEP;
      if (rs >= RS) { rs -= RS; rphase ^= 1u; }
      raw_ready = i + 2 < units && mbar_test_wait(&raw_full[rs], rphase);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&a_ready[2 * as + unit]);
      as += 2;
      if (as >= SA) { as -= SA; aphase ^= 1u; }
    }
    // ---- epilogue ----
    pdl_wait();   // the stores below may overwrite what an earlier kernel still reads
    if (ok) ok = warp_wait(acc_full, 0, p.status, KC_DEV_QLINEAR | 7);
    if (ok) ql_epilogue<NT>(p, smem, warp, lane, tmem_base, tile0, nt_live, split, chunk0, nkb > 1);
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(p.tmem_cols)
                 : "memory");
  }
}

// Ring depths and shared memory of one launch geometry; ok == false when it does not fit tensor or shared memory.
struct TaPlan { bool ok; int sa, sb, rs; uint32_t tmem_cols; size_t smem; };
static TaPlan plan_ta(int nt, int per, int m_pad, uint32_t record_bytes) {
  TaPlan t{};
  const int acc_cols = 2 * ((m_pad + 31) & ~31);
  int sa = std::min(6 / per, (512 - acc_cols) / (64 * per)) & ~1;
  if (sa < 2 || m_pad > 256) return t;
  uint32_t cols = 32;
  while ((int)cols < acc_cols + sa * 64 * per) cols <<= 1;
  const size_t budget = (size_t)212 * 1024;
  const size_t b_stage = (size_t)per * m_pad * 128;
  const size_t r_stage = (size_t)per * nt * record_bytes;
  // activations arrive from L2 (about 2000 cycles): up to 16 k-blocks ahead where they are small, 6 of 192 rows
  int sb = (int)std::min<size_t>(16 / per, std::max<size_t>(per == 1 ? 6 : 4, (size_t)(64 * 1024) / b_stage));
  while (sb > 4 && (size_t)sb * b_stage + (nt == 2 ? 6 : 8) * r_stage > budget) --sb;
  sb &= nt == 1 ? ~1 : ~0;   // one tile per CTA: an issuer takes every second k-block and must meet every fill of its slots
  if ((size_t)sb * b_stage + 4 * r_stage > budget) return t;
  // a multiple of the k-blocks between a group's units (see the kernel), so that a slot always serves the same groups
  int rs = (int)std::min<size_t>(32, (budget - (size_t)sb * b_stage) / r_stage) & (nt == 2 ? ~1 : ~3);
  if (rs < 4) return t;
  // the epilogue's per-warp transpose buffers reuse the ring memory from its start
  while ((size_t)sb * b_stage + (size_t)rs * r_stage < (size_t)QL_DQ_WARPS * QL_EPI_STAGE_BYTES) rs += 4;
  const size_t smem = 1024 + (size_t)sb * b_stage + (size_t)rs * r_stage + (2 * rs + 2 * sb + 4 * sa + 1) * 8 + 16;
  if (smem > 227 * 1024) return t;
  t.ok = true; t.sa = sa; t.sb = sb; t.rs = rs; t.tmem_cols = cols; t.smem = smem;
  return t;
}

// ---------------------------------------------------------------------------
// Many rows against a weight that is split along K: qlinear_umma_rows_kernel. The splits are there to fill the SMs at few rows;
// with many, chunks of rows do, and a CTA takes all splits of its tile and rows one after the other, so that no partial goes
// through memory and nothing is left to reduce. Persistent: a CTA walks over (tile, chunk) items, weights and activations of
// the next split or item arriving under the last one.
//
// The sums are those of the launches with a split a CTA: the even and the odd k-blocks of a split in an accumulator each, the
// split's sum of the two, and the splits' sums added in order, which lie in shared memory meanwhile.
//
// Roles as in qlinear_umma_ta_kernel. A segment is one split of one item. A stage is two k-blocks, one for each accumulator;
// where a segment ends on an odd one the stage's second unit passes through the rings empty. At a segment's end the
// dequantisers, who have the next segment's first stages in tensor memory by then, read the accumulators.
//
// What bounds it: the hand-over of the dequantised weights as in qlinear_umma_ta_kernel (about 500 cycles a k-block up to 112
// rows), then the activations: every CTA reads its own, 24 KB a k-block of 192 rows, 45 bytes a cycle and SM of L2. A form with
// two tiles a CTA sharing them, four accumulators of 96 rows, took 980 cycles a pair of k-blocks, 349 us where this takes 231.
// 4096 x 14336 at 2048 rows: tensor pipe 51 % active, HBM at 6 % of its rate. The 8-bit instantiations for large scales spill
// (40 and 48 bytes at 96 registers, the most that 640 threads leave).
// TMEM columns: [even, odd: round32(m_pad) each] [a_stages x 2 units x 32 columns].
// ---------------------------------------------------------------------------
template <int BITS, int GPK, bool WIDE>
__global__ void __launch_bounds__(QL_THREADS, 1)
qlinear_umma_rows_kernel(const __grid_constant__ CUtensorMap map_rows, const QlKernelParams p) {
  constexpr uint32_t PACKED = QL_TILE_N * (QL_KB * BITS / 8);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int SA = p.a_stages, SB = p.b_stages, RS = p.r_stages;   // SB, RS: k-blocks
  const uint32_t b_bytes = (uint32_t)p.m_pad * 128u;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int items = p.n_tiles * p.chunks;
  const uint32_t cs = (uint32_t)(p.m_pad + 31) & ~31u, a_col0 = 2 * cs;
  auto first_kb = [&](int split) { return (int)((long long)p.kblocks * split / p.splits); };

  uint8_t* sB = smem;
  uint8_t* sR = sB + (size_t)SB * b_bytes;
  float* sums = reinterpret_cast<float*>(sR + (size_t)RS * p.record_bytes);   // [row][128] of the splits so far
  uint64_t* bars = reinterpret_cast<uint64_t*>(sums + p.m_pad * QL_TILE_N);
  uint64_t* raw_full = bars;
  uint64_t* raw_empty = raw_full + RS;
  uint64_t* b_full = raw_empty + RS;
  uint64_t* b_empty = b_full + SB;
  uint64_t* a_ready = b_empty + SB;       // [stage][unit]
  uint64_t* a_empty = a_ready + 2 * SA;
  uint64_t* acc_full = a_empty + 2 * SA;  // a segment's products are in
  uint64_t* acc_free = acc_full + 1;      // .. and read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_free + 1);

  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int i = 0; i < RS; ++i) { mbar_init(&raw_full[i], 1); mbar_init(&raw_empty[i], 4); }
    for (int i = 0; i < SB; ++i) { mbar_init(&b_full[i], 1); mbar_init(&b_empty[i], 1); }
    for (int i = 0; i < 2 * SA; ++i) { mbar_init(&a_ready[i], 4); mbar_init(&a_empty[i], 1); }
    mbar_init(acc_full, 2); mbar_init(acc_free, QL_DQ_WARPS);
    mbar_fence_init();
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(p.tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (warp == 1 && lane == 0) tma_prefetch_desc(&map_rows);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp < 2) {
    // ---- producers: warp 0 the weight records, warp 1 the activations, the first access of this kernel to memory written by
    // earlier kernels. Both walk the same k-blocks; an empty unit's barrier is completed without a copy. ----
    if (lane == 0) {
      if (warp == 1) pdl_wait();
      RingPos rp;
      const int depth = warp == 0 ? RS : SB;
      uint64_t *full = warp == 0 ? raw_full : b_full, *empty = warp == 0 ? raw_empty : b_empty;
      bool ok = true;
      for (int item = blockIdx.x; ok && item < items; item += gridDim.x) {
        const int tile = item % p.n_tiles, row = p.row0 + item / p.n_tiles * p.m_pad;
        const uint8_t* src = p.records + ((size_t)(tile / QL_TILE_GROUP) * p.kblocks * QL_TILE_GROUP + tile % QL_TILE_GROUP) * p.record_bytes;
        for (int split = 0; ok && split < p.splits; ++split) {
          const int kb1 = first_kb(split + 1);
          int kb = first_kb(split);
          for (int left = (kb1 - kb + 1) & ~1; left > 0; --left, ++kb, rp.advance(depth)) {
            ok = mbar_wait(&empty[rp.stage], rp.phase ^ 1, p.status, KC_DEV_QLINEAR | (1 + warp));
            if (!ok) break;
            if (kb >= kb1) {
              mbar_arrive(&full[rp.stage]);
            } else if (warp == 0) {
              mbar_arrive_expect_tx(&full[rp.stage], p.record_bytes);
              bulk_g2s(sR + (size_t)rp.stage * p.record_bytes, src + (size_t)kb * QL_TILE_GROUP * p.record_bytes, p.record_bytes, &full[rp.stage]);
            } else {
              mbar_arrive_expect_tx(&full[rp.stage], b_bytes);
              tma_load_2d(sB + (size_t)rp.stage * b_bytes, &map_rows, kb * QL_KB, row, &full[rp.stage]);
            }
          }
        }
      }
    }
  } else if (warp < QL_DQ_WARP0) {
    // ---- MMA issuers: warp 2 + u has accumulator u, the k-blocks u, u + 2, .. of a segment ----
    pdl_wait();
    const int u = warp - 2;
    const uint32_t idesc = umma_idesc_bf16(QL_TILE_N, p.m_pad);
    const uint64_t proto = umma_smem_desc(0, 1024);
    const uint32_t d_hi = (uint32_t)(proto >> 32), b_lo0 = (uint32_t)proto | ((smem_u32(sB) >> 4) & 0x3FFF);
    const uint32_t d = tmem_base + u * cs, a_t0 = tmem_base + a_col0 + u * 32;
    int as = 0, bs = u, seg = 0;
    uint32_t aphase = 0, bphase = 0;
    bool ok = true, ready = false;
    for (int item = blockIdx.x; ok && item < items; item += gridDim.x) {
      for (int split = 0; ok && split < p.splits; ++split, ++seg) {
        const int nkb = first_kb(split + 1) - first_kb(split), stages = (nkb + 1) >> 1;
        if (seg > 0) ok = warp_wait(acc_free, (seg - 1) & 1, p.status, KC_DEV_QLINEAR | 8);
        for (int j = 0; ok && j < stages; ++j) {
          if (!__all_sync(0xffffffffu, ready)) {
            ok = warp_wait(&b_full[bs], bphase, p.status, KC_DEV_QLINEAR | 4) &&
                 warp_wait(&a_ready[2 * as + u], aphase, p.status, KC_DEV_QLINEAR | 3);
            if (!ok) break;
          }
          tc_fence_after();
          const uint32_t b_lo = b_lo0 + bs * (b_bytes >> 4), a_t = a_t0 + as * 64;
          uint64_t *a_done = &a_empty[2 * as + u], *b_done = &b_empty[bs];
          if (++as == SA) { as = 0; aphase ^= 1u; }
          bs += 2;
          if (bs >= SB) { bs -= SB; bphase ^= 1u; }
          ready = j + 1 < stages && (mbar_test_wait(&b_full[bs], bphase) & mbar_test_wait(&a_ready[2 * as + u], aphase));
          if (elect_one()) {
            if (2 * j + u < nkb) {
#pragma unroll
              for (int ks = 0; ks < QL_KB / 16; ++ks)
                umma_bf16_ts(d, a_t + 8 * ks, b_lo + 2 * ks, d_hi, idesc, j == 0 && ks == 0 ? 0u : 1u);
            }
            umma_commit(a_done);
            umma_commit(b_done);
          }
          __syncwarp();
        }
        if (ok && elect_one()) umma_commit(acc_full);
        __syncwarp();
      }
    }
  } else {
    // ---- dequantisers: group g converts unit g & 1 of the stages g >> 1, (g >> 1) + 2, .. over all segments ----
    const int grp = (warp - QL_DQ_WARP0) >> 2, unit = grp & 1, q = warp & 3;
    const int n_in = q * 32 + lane;
    const uint32_t lanes = (uint32_t)(q * 32) << 16;
    const uint32_t a_addr = tmem_base + lanes + a_col0 + unit * 32;
    const uint8_t *row_raw = sR + n_in * 16, *row_sb = sR + PACKED + n_in * (GPK * 4);
    int rs = (grp >> 1) * 2 + unit, as = grp >> 1, seg = 0, stage0 = 0;   // stage0: parity of the segment's first stage
    uint32_t rphase = 0, aphase = 0;
    int done = 0;
    bool ok = true, released = false, raw_ready = false;
    int waiting_item = -1, waiting_split = 0;   // the segment whose accumulators are still to be read
    // eight columns (rows of the step) at a time: the split's sum, added to those before it or written out
    auto drain = [&]() {
      if (!released) { pdl_wait(); released = true; }   // the stores may overwrite what an earlier kernel still reads
      ok = warp_wait(acc_full, (seg - 1) & 1, p.status, KC_DEV_QLINEAR | 7);
      if (!ok) return;
      tc_fence_after();
      const bool odd = first_kb(waiting_split + 1) - first_kb(waiting_split) > 1, last = waiting_split == p.splits - 1;
      const int n = waiting_item % p.n_tiles * QL_TILE_N + n_in, row0 = waiting_item / p.n_tiles * p.m_pad;
#pragma unroll 1
      for (int c = grp * 8; c < p.m_pad; c += QL_DQ_GROUPS * 8) {
        const uint32_t at = tmem_base + lanes + c;
        uint32_t e[8], o[8];
        tmem_ld8_issue(at, e);
        tmem_ld8_issue(odd ? at + cs : at, o);
        float* sum = sums + c * QL_TILE_N + n_in;
        float before[8];
        if (waiting_split > 0) {
#pragma unroll
          for (int j = 0; j < 8; ++j) before[j] = sum[j * QL_TILE_N];
        }
        tmem_wait_ld();
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          asm volatile("" : "+r"(e[j]), "+r"(o[j]));   // no use before the wait
          v[j] = odd ? __uint_as_float(e[j]) + __uint_as_float(o[j]) : __uint_as_float(e[j]);
          if (waiting_split > 0) v[j] = before[j] + v[j];
        }
        if (!last) {
#pragma unroll
          for (int j = 0; j < 8; ++j) sum[j * QL_TILE_N] = v[j];
        } else if (n < p.N) {
          const int m = row0 + c;
          bf16* dst = p.y + (size_t)(p.row0 + m) * p.ldy + n;
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (m + j < p.M) dst[(size_t)j * p.ldy] = __float2bfloat16_rn(v[j]);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_free);
      waiting_item = -1;
    };
    for (int item = blockIdx.x; ok && item < items; item += gridDim.x) {
      for (int split = 0; ok && split < p.splits; ++split) {
        const int nkb = first_kb(split + 1) - first_kb(split), stages = (nkb + 1) >> 1;
        for (int j = (grp >> 1) ^ stage0; ok && j < stages; j += 2) {
          // the first stages are dequantised under the tail of the previous kernel: see qlinear_umma_ta_kernel
          if (!released && 2 * done >= SA) { pdl_wait(); released = true; }
          ++done;
          if (!__all_sync(0xffffffffu, raw_ready)) {
            ok = warp_wait(&raw_full[rs], rphase, p.status, KC_DEV_QLINEAR | 5);
            if (!ok) break;
          }
          const bool a_free = mbar_test_wait(&a_empty[2 * as + unit], aphase ^ 1);
          const size_t at = (size_t)rs * p.record_bytes;
          uint32_t v[32];   // of an empty unit: whatever its slot holds, which no product takes
          bf162 sb[GPK];
          if (GPK == 1) {
            sb[0] = *reinterpret_cast<const bf162*>(row_sb + at);
          } else {
            const uint2 s = *reinterpret_cast<const uint2*>(row_sb + at);
            sb[0] = bf2_bits(s.x); sb[GPK - 1] = bf2_bits(s.y);
          }
          if (!WIDE) dequant_row<BITS, GPK>(row_raw + at, sb, v);
          else dequant_row_wide<BITS, GPK>(row_raw + at, sb, v);
          if (!__all_sync(0xffffffffu, a_free)) ok = warp_wait(&a_empty[2 * as + unit], aphase ^ 1, p.status, KC_DEV_QLINEAR | 6);
          if (!ok) break;
          tc_fence_after();
          tmem_st32(a_addr + as * 64, v);
          __syncwarp();
          if (lane == 0) mbar_arrive(&raw_empty[rs]);
          rs += 4;
          if (rs >= RS) { rs -= RS; rphase ^= 1u; }
          raw_ready = mbar_test_wait(&raw_full[rs], rphase);
          tmem_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&a_ready[2 * as + unit]);
          as += 2;
          if (as >= SA) { as -= SA; aphase ^= 1u; }
          if (waiting_item >= 0) drain();
        }
        if (ok && waiting_item >= 0) drain();   // a segment without a stage of this group
        waiting_item = item; waiting_split = split;
        ++seg;
        stage0 ^= stages & 1;
      }
    }
    if (ok && waiting_item >= 0) drain();
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(p.tmem_cols) : "memory");
  }
}

// Ring depths and shared memory of qlinear_umma_rows_kernel.
static TaPlan plan_rows(const QWeight& w, int m_pad) {
  TaPlan t{};
  const int acc_cols = 2 * ((m_pad + 31) & ~31);
  t.sa = std::min(6, (512 - acc_cols) / 64) & ~1;
  t.tmem_cols = 512;
  const size_t sums = (size_t)m_pad * QL_TILE_N * 4, budget = (size_t)224 * 1024 - sums;
  const size_t b_stage = (size_t)m_pad * 128, r_stage = w.record_bytes;
  t.rs = 4; t.sb = 4;
  if (t.sb * b_stage + t.rs * r_stage > budget) return t;
  // Deeper as far as there is room, activations by stages of two k-blocks, records by two stages (see the kernel). Three stages
  // of activations come first: with two a k-block of 160 rows took 690 cycles, with three one of 144 took 517.
  for (bool more = true; more;) {
    more = false;
    if (t.sb < 12 && (t.sb + 2) * b_stage + t.rs * r_stage <= budget) { t.sb += 2; more = true; }
    if (t.rs < 16 && t.sb * b_stage + (t.rs + 4) * r_stage <= budget) { t.rs += 4; more = true; }
  }
  t.smem = 1024 + t.sb * b_stage + t.rs * r_stage + sums + (2 * t.rs + 2 * t.sb + 4 * t.sa + 2) * 8 + 16;
  t.ok = t.sa >= 2 && t.smem <= 227 * 1024;
  return t;
}

template <int BITS, int GPK, bool WIDE>
static cudaError_t launch_umma_rows_as(const QLinearLaunch& l, QlKernelParams& p, cudaStream_t s) {
  const QWeight& w = *l.w;
  const TaPlan t = plan_rows(w, p.m_pad);
  if (!t.ok) return cudaErrorInvalidValue;
  p.tmem_cols = t.tmem_cols;
  p.a_stages = t.sa; p.b_stages = t.sb; p.r_stages = t.rs;
  static DeviceOnce configured;   // the attribute belongs to the device's copy of the kernel
  if (configured.first_on_current_device()) {
    cudaError_t e = cudaFuncSetAttribute(qlinear_umma_rows_kernel<BITS, GPK, WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) { configured.forget_current_device(); return e; }
  }
  const CUtensorMap* rows = act_operand_rows_map(l.x, p.m_pad);
  if (!rows) return cudaErrorInvalidValue;
  return launch_k(qlinear_umma_rows_kernel<BITS, GPK, WIDE>, dim3(std::min(w.n_tiles * p.chunks, w.sm_count)), dim3(QL_THREADS), t.smem, s, *rows, p);
}
template <int BITS, int GPK>
static cudaError_t launch_umma_rows(const QLinearLaunch& l, QlKernelParams& p, cudaStream_t s) {
  return l.w->wide_scale ? launch_umma_rows_as<BITS, GPK, true>(l, p, s) : launch_umma_rows_as<BITS, GPK, false>(l, p, s);
}

template <int BITS, int GPK, int NT, int P, bool WIDE>
static cudaError_t launch_umma_ta(const QLinearLaunch& l, QlKernelParams& p, cudaStream_t s) {
  const QWeight& w = *l.w;
  const TaPlan t = plan_ta(NT, P, p.m_pad, p.record_bytes);
  if (!t.ok) return cudaErrorInvalidValue;   // the caller sized the row chunk with plan_ta
  p.tmem_cols = t.tmem_cols;
  p.a_stages = t.sa; p.b_stages = t.sb; p.r_stages = t.rs;
  static DeviceOnce configured;   // the attribute belongs to the device's copy of the kernel
  if (configured.first_on_current_device()) {
    cudaError_t e = cudaFuncSetAttribute(qlinear_umma_ta_kernel<BITS, GPK, NT, P, WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) { configured.forget_current_device(); return e; }
  }
  const CUtensorMap* rows = act_operand_rows_map(l.x, p.m_pad);
  if (!rows) return cudaErrorInvalidValue;
  dim3 grid((w.n_tiles + NT - 1) / NT, w.splits, (p.M + p.m_pad - 1) / p.m_pad);
  return launch_k(qlinear_umma_ta_kernel<BITS, GPK, NT, P, WIDE>, grid, dim3(QL_THREADS), t.smem, s, *rows, p);
}

template <int BITS, int GPK>
static cudaError_t launch_umma_nt(const QLinearLaunch& l, QlKernelParams& p, int nt, cudaStream_t s) {
  // a scale of the weight is past ql_scale_limit: kernels of its own, so that the others don't carry the conversion
  if (l.w->wide_scale) return nt == 2 ? launch_umma_ta<BITS, GPK, 2, 1, true>(l, p, s) : launch_umma_ta<BITS, GPK, 1, 1, true>(l, p, s);
  if (plan_ta(nt, 2, p.m_pad, p.record_bytes).ok)
    return nt == 2 ? launch_umma_ta<BITS, GPK, 2, 2, false>(l, p, s) : launch_umma_ta<BITS, GPK, 1, 2, false>(l, p, s);
  return nt == 2 ? launch_umma_ta<BITS, GPK, 2, 1, false>(l, p, s) : launch_umma_ta<BITS, GPK, 1, 1, false>(l, p, s);
}

// Weight tiles per CTA: two when the grid then still has about 0.7 CTAs per SM (measured: 112 CTAs of two tiles beat
// 224 CTAs of one on 148 SMs — the activation k-block is read from L2 once per CTA), else one.
static int plan_tiles_per_cta(const QWeight& w, int sm_count) {
  return ((w.n_tiles + 1) / 2) * w.splits * 10 >= sm_count * 7 ? 2 : 1;
}

// The most rows one CTA takes: what the two accumulators (192 columns each) and the rings of the weight's record size
// leave room for. With one tile per CTA and one accumulator it was 256 rows; the two accumulators of that form (even and
// odd k-blocks) take 10 to 30 % off launches of up to 192 rows and of more than 256, and the second chunk that 193 to 256
// rows need costs up to 25 % (4096 x 4096, L2 flushed: 23.6 -> 27.6 us at 193 rows, 25.6 -> 29.7 at 256; 21.5 at 192,
// 33.8 -> 31.7 at 257). One accumulator for these rows alone would give them other bits than fewer rows have.
static int plan_row_cap(int nt, uint32_t record_bytes) {
  static const int caps[] = {192, 128, 64, 32, 16};
  for (int c : caps)
    if (plan_ta(nt, 1, c, record_bytes).ok) return c;
  return 0;
}

// Rows of a chunk (one CTA's share of the rows) for M rows. All chunks are one launch, CTAs of the next filling the SMs
// that the last wave of one leaves idle; the chunk size is the one whose waves take the least time, counted in MMA
// cycles: a unit of 128 x 64 weights takes 2 cycles per row, not less than 184, and a CTA about 6000 around them. Chunks of
// fewer than 96 rows are not looked at: a unit takes its 184 cycles then, whatever the rows, so more chunks are only more
// waves.
// 28672 x 4096, 2048 rows: 13 chunks of 160 rows are 10 waves, 368 us; 11 chunks of 192, a launch each, took 450.
static int plan_chunk_rows(const QWeight& w, int nt, int cap, int M) {
  const int ctas = ((w.n_tiles + nt - 1) / nt) * w.splits;
  const long long units = (long long)w.kblocks * nt / w.splits;
  int best = 0;
  long long best_cost = 0;
  for (int chunks = (M + cap - 1) / cap; best == 0 || chunks * 96 <= M; ++chunks) {
    const int per = ((M + chunks - 1) / chunks + 15) & ~15;
    const int n = (M + per - 1) / per;
    const long long waves = ((long long)ctas * n + w.sm_count - 1) / w.sm_count;
    const long long cost = waves * (units * std::max(184, 2 * per) + 6000);
    if (best == 0 || cost < best_cost) { best = per; best_cost = cost; }
  }
  return best;
}

constexpr int QL_ROWS_MIN = 257;   // below, a chunk or two of rows never fill the SMs
// With more k-blocks all splits in turn are the slower way at most row counts: 7000 x 28672 (448) 499 -> 564 us at 1200 rows, 805
// -> 885 at 2048; 8192 x 28672 316 -> 334 at 640, 757 -> 780 at 1500, though 265 -> 251 at 513. 3584 x 18944 (296): the same
// within a fiftieth up to 2048 rows, a tenth faster from there.
constexpr int QL_ROWS_MAX_KBLOCKS = 300;
// Whether a weight's rows are taken by qlinear_umma_rows_kernel, and how many a chunk: 0 where a split a CTA takes about as long
// or less. In cycles, fitted to launches of 264 to 2048 rows against eight weights of 16 to 64 tiles and 56 to 448 k-blocks, the
// fit within a tenth of them: a k-block there takes 330 and 1.55 a row, a CTA's start and end 9500; here 330 and 1.9 a row, 2.3
// where two stages of activations only have room, a segment's end 600. A reduction of their own costs partials 2150 bytes a
// cycle over all SMs where there are more than QL_MAX_M rows, else 6500. Summed by the kernel that reads the result anyway
// they cost that next to nothing, and of the two ways the one with a launch of its own size has to be faster by a seventh:
// a layer of a step, splits apart -> in turn, us: 1B (2048 features) 96 -> 100 at 257 rows, 142 -> 147 at 448; 9B (3584) 201 -> 206 at
// 333; 8B (4096) 289 -> 284 at 448, 300 -> 293 at 512; 7B (3584, 8 bits) 335 -> 330 at 448. More than eight splits are short ones, whose ends
// lie less under the next one's start, 900: at 600 a call of 1024 x 8192 (16 splits) and 768 rows went from 48.5 to 56.1 us.
// The choice against both ways at 23 row counts from 257 to 4096 and 26 weights: 22 % ahead of a split a CTA on average and
// within 1 % of the best choice of way and chunk; behind a split a CTA by more than 2 % at two of the 598, 6000 x 12288 of 8
// bits and 768 rows (3 %) and 3584 x 18944 of 8 bits and 2048 rows (1 % in three runs, 9 % in one).
// At 2048 rows, split a CTA -> this: 4096 x 4096 156 -> 96 us, 4096 x 14336 281 -> 231, 6144 x 4096 185 -> 131, 8192 x 8192
// 310 -> 262. At 366: 24 -> 27 (and 2 us less in the consumer), 46 -> 67, 28 -> 29: not taken.
static int plan_rows_chunk(const QWeight& w, int M, bool summed) {
  if (w.splits == 1 || plan_tiles_per_cta(w, w.sm_count) != 1 || M < QL_ROWS_MIN || w.kblocks > QL_ROWS_MAX_KBLOCKS) return 0;
  const int cap = plan_row_cap(1, w.record_bytes);
  if (cap == 0) return 0;
  auto apart_cost = [&](int rows) -> long long {
    if (rows == 0) return 0;
    const int per = plan_chunk_rows(w, 1, cap, rows);
    const long long ctas = (long long)w.n_tiles * w.splits * ((rows + per - 1) / per), waves = (ctas + w.sm_count - 1) / w.sm_count;
    const long long values = (long long)rows * w.N;
    return waves * (w.kblocks * (330 + per * 31 / 20) / w.splits + 9500) +
           (summed ? 0 : M > QL_MAX_M ? values * (4 * w.splits + 2) / 2150 : values * 4 * w.splits / 6500);
  };
  const long long apart = M / QL_MAX_M * apart_cost(QL_MAX_M) + apart_cost(M % QL_MAX_M);
  int best = 0;
  long long best_cost = apart / 100 * (summed ? 86 : 92);
  const int ends = w.splits * (w.splits > 8 ? 900 : 600);
  if (w.kblocks * (330 + 96 * 19 / 10) + ends + 8000 >= best_cost) return 0;   // one wave of the smallest chunks
  for (int per = 192; per >= 96; per -= 16) {
    const TaPlan t = plan_rows(w, per);
    if (!t.ok) continue;
    const long long items = (long long)w.n_tiles * ((M + per - 1) / per), waves = (items + w.sm_count - 1) / w.sm_count;
    const long long cost = waves * (w.kblocks * (330 + per * (t.sb >= 6 ? 19 : 23) / 10) + ends) + 8000;
    if (cost < best_cost) { best = per; best_cost = cost; }
  }
  return best;
}
bool qlinear_in_turn(const QWeight& w, int M, bool summed) { return plan_rows_chunk(w, M, summed) > 0; }

cudaError_t qlinear_umma(const QLinearLaunch& l, cudaStream_t s) {
  const QWeight& w = *l.w;
  if (l.M < 1 || l.M > qlinear_slab_rows(w, l.M)) return cudaErrorInvalidValue;
  if (l.row0 % 16 || l.row0 + l.M > l.x->rows) return cudaErrorInvalidValue;   // rows past the operand's end read as zeros
  const int nt = plan_tiles_per_cta(w, w.sm_count);
  const int cap = plan_row_cap(nt, w.record_bytes);
  if (cap == 0) return cudaErrorInvalidValue;
  // the gated activation is fused when a CTA owns whole (gate, up) tile pairs and writes final values
  const bool glu = l.glu && nt == 2 && w.splits == 1 && (w.n_tiles & 1) == 0 && (w.N % (2 * QL_TILE_N)) == 0 && l.act &&
                   (l.ld_act & 3) == 0 && (reinterpret_cast<uintptr_t>(l.act) & 7) == 0;
  if (l.glu_done) *l.glu_done = glu ? 1 : 0;
  QlKernelParams p;
  p.records = w.records; p.record_bytes = w.record_bytes;
  p.N = w.N; p.n_tiles = w.n_tiles; p.kblocks = w.kblocks;
  p.M = l.M; p.m_pad = plan_chunk_rows(w, nt, cap, l.M); p.row0 = l.row0;
  p.splits = w.splits; p.chunks = 0;
  p.y = l.y; p.ldy = l.ldy; p.partial = l.partial; p.status = l.status;
  p.glu = glu ? l.glu : 0; p.act = l.act; p.ld_act = l.ld_act;
  if (const int rows = plan_rows_chunk(w, l.M, l.summed)) {
    p.m_pad = rows; p.chunks = (l.M + rows - 1) / rows;
    if (w.bits == 4) return w.gpk == 2 ? launch_umma_rows<4, 2>(l, p, s) : launch_umma_rows<4, 1>(l, p, s);
    return w.gpk == 2 ? launch_umma_rows<8, 2>(l, p, s) : launch_umma_rows<8, 1>(l, p, s);
  }
  if (w.bits == 4) return w.gpk == 2 ? launch_umma_nt<4, 2>(l, p, nt, s) : launch_umma_nt<4, 1>(l, p, nt, s);
  return w.gpk == 2 ? launch_umma_nt<8, 2>(l, p, nt, s) : launch_umma_nt<8, 1>(l, p, nt, s);
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
        const int gcol = p.gu_interleaved ? (col >> 7) * 256 + (col & 127) : col;
        const int ucol = p.gu_interleaved ? gcol + 128 : F + col;
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

