// The affine-dequant GEMM on the tensor cores. See kc_qlinear.cuh for the data layout.
//
// qlinear_umma_kernel — teams of two CTAs. A team has a PAIR of neighbouring 128-row weight tiles at a time, one tile a CTA,
// and the same k-blocks of both. Up to solo_rows activation rows its CTAs know nothing of each other; with more they are a cluster
// whose two SMs work on one M = 256 product (tcgen05 cta_group::2), each holding half of the activations. 20 warps:
//   warp 0        bulk-copies the weight records (cp.async.bulk, mbarrier tx)
//   warp 1        TMA-loads the activation k-blocks (cp.async.bulk.tensor, 128B swizzle), of a cluster its CTA's half of the rows
//   warp 2        allocates TMEM; issues tcgen05.mma (weights = A/M side from TENSOR MEMORY, activations = B/N side from shared
//                 memory), of a cluster the first CTA's for both
//   warps 4-19    four groups of four warps. Three dequantise: they unpack the 4/8-bit words, apply scale and bias in registers and
//                 write the bf16 A operand into tensor memory (tcgen05.st). The first drains accumulators (tcgen05.ld) under the
//                 next task's products; the last task is drained by all.
// The accumulator D[n, m] lives in TMEM: lane = weight row n, column = activation row m.
//
// Every output element depends only on its own activation row and on an order of sums fixed by (N, K) and the SM count: a
// pair's k-blocks are cut into parts at fixed places, a part is one chain of products or two (its even and its odd k-blocks,
// QWeight::chains, added at its end), and the parts are added in order. That is what lets verify rows share a step with other
// rows and still reproduce the bits of a one-row decode. More rows than one accumulator holds are chunks of rows: rows are
// independent, so no bit changes.
#include "kc_qlinear.cuh"
#include "kc_umma.cuh"

#include <algorithm>
#include <cmath>

namespace kc {

// ---------------------------------------------------------------------------
// Dequantisation of one weight row of one k-block: 64 values -> 32 bf16 pairs, w = bf16(q * scale + bias), one rounding.
//
// The integers become bf16 operands of the multiply-add without a conversion: the bf16 with bit pattern N < 256 is N * 2^-133
// (subnormals and the first binade have the same spacing), so a nibble masked into bits 0..3 or a byte in bits 0..7 of a
// half-word IS q * 2^-133, a nibble in bits 4..7 q * 2^-129. One fused multiply-add with the scale times 2^133 (2^129: exact,
// powers of two) gives q * scale + bias rounded once — the value that converting q first gives. 9 instructions for 8 weights
// of 4 bits (two nibbles of a half-word in place, two behind one shift), 4 for 4 of 8 bits. The scaled scale must stay below
// 2^128: a weight with larger scales (2^-5 and more) is taken at 2^-shift of its size, QWeight::shift, and its sums are
// multiplied back, both exact as long as nothing falls below the normal numbers on the way. Where scales are so far apart that
// something would (2^57 and more between the smallest and 2^-6 of the largest), WIDE brings the integers to size instead, two
// multiplications a pair.
// ---------------------------------------------------------------------------

__device__ __forceinline__ bf162 bf2_bits(uint32_t u) { return *reinterpret_cast<const bf162*>(&u); }
__device__ __forceinline__ uint32_t bf2_fma(uint32_t a, bf162 s, bf162 b) {
  const bf162 r = __hfma2(*reinterpret_cast<const bf162*>(&a), s, b);
  return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t bf2_raw(bf162 v) { return *reinterpret_cast<const uint32_t*>(&v); }
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}

// The factors of a weight's scales and biases: scale * s0 * s1 = scale * 2^(133 - shift), bias * b = bias * 2^-shift.
struct QlFactors { uint32_t s0, s1, b; };

// Packed words of a row (16-byte chunk c at row + c * QL_TILE_N * 16), its scale and bias pairs at sb -> v[32].
template <bool WIDE>
__device__ __forceinline__ uint32_t dequant_pair(uint32_t q, uint32_t size, bf162 s, bf162 b) {   // size: 2^-127 of what makes q the integers
  if (!WIDE) return bf2_fma(q, s, b);
  return bf2_fma(bf2_raw(__hmul2(__hmul2(bf2_bits(q), bf2_bits(0x7F007F00u)), bf2_bits(size))), s, b);
}
template <int BITS, int GPK, bool WIDE>
__device__ __forceinline__ void dequant_row(uint32_t row, uint32_t sb, const QlFactors& f, uint32_t (&v)[32]) {
  constexpr int CHUNKS = BITS / 2;
  bf162 s_lo[GPK], s_hi[GPK], bias[GPK];
  uint32_t raw[GPK];
  if (GPK == 1) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(raw[0]) : "r"(sb));
  else asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(raw[0]), "=r"(raw[GPK - 1]) : "r"(sb));
  uint4 w[CHUNKS];
#pragma unroll
  for (int h = 0; h < CHUNKS; ++h) w[h] = lds128(row + h * (QL_TILE_N * 16));
#pragma unroll
  for (int g = 0; g < GPK; ++g) {
    const bf162 pair = bf2_bits(raw[g]);
    s_lo[g] = __bfloat162bfloat162(pair.x);
    bias[g] = __bfloat162bfloat162(pair.y);
    if (!WIDE) {
      s_lo[g] = __hmul2(__hmul2(s_lo[g], bf2_bits(f.s0)), bf2_bits(f.s1));
      bias[g] = __hmul2(bias[g], bf2_bits(f.b));
    }
    if (BITS == 4) s_hi[g] = WIDE ? s_lo[g] : __hmul2(s_lo[g], bf2_bits(0x3D803D80u));   // 2^-4
  }
#pragma unroll
  for (int h = 0; h < CHUNKS; ++h) {
    const uint32_t word[4] = {w[h].x, w[h].y, w[h].z, w[h].w};
    const int g = GPK == 2 ? h * 2 / CHUNKS : 0;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (BITS == 4) {
        // the record's nibble order: element 2j at bits 4j, element 2j + 1 at bits 16 + 4j
        uint32_t* o = v + (h * 4 + c) * 4;
        const uint32_t up = word[c] >> 8;
        o[0] = dequant_pair<WIDE>(word[c] & 0x000F000Fu, 0x42804280u, s_lo[g], bias[g]);   // 2^6
        o[1] = dequant_pair<WIDE>(word[c] & 0x00F000F0u, 0x40804080u, s_hi[g], bias[g]);   // 2^2
        o[2] = dequant_pair<WIDE>(up & 0x000F000Fu, 0x42804280u, s_lo[g], bias[g]);
        o[3] = dequant_pair<WIDE>(up & 0x00F000F0u, 0x40804080u, s_hi[g], bias[g]);
      } else {
        uint32_t* o = v + (h * 4 + c) * 2;
        o[0] = dequant_pair<WIDE>(__byte_perm(word[c], 0u, 0x4140u), 0x42804280u, s_lo[g], bias[g]);
        o[1] = dequant_pair<WIDE>(__byte_perm(word[c], 0u, 0x4342u), 0x42804280u, s_lo[g], bias[g]);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Tasks
// ---------------------------------------------------------------------------

constexpr int QL_GROUP0 = 4;                                   // first warp of the four groups
constexpr int QL_GROUPS = 4;
constexpr int QL_THREADS = (QL_GROUP0 + 4 * QL_GROUPS) * 32;   // 20 warps
constexpr int QL_STAGE_BYTES = 1280;                           // a warp's buffer on the way out: 16 rows of 32 bf16, or 8 of fp32, with padding
// k-blocks of a unit: two where a unit's products take few cycles a k-block, one where two accumulators of many rows leave tensor
// memory for four k-blocks only.
__host__ __device__ constexpr int ql_unit(int cg) { return cg == 1 ? 2 : 1; }

// How a launch's teams share the work:
//   APART    a team a (pair, split, chunk of rows); the splits are left to the kernel that reads the result, or there is one
//   RUNS     (of one chain) the k-blocks of all pairs, one after the other, in as many equal runs as the SMs have teams, each at least a pair's:
//            where a run ends inside a pair, its sums so far go through global memory to the team with the pair's end, which goes
//            on from them: the same chain of products as one team's. A team waits for the one before it only, having left its own sums
//            first, so all that it takes is that CTAs start in the order of their indices, or that all are resident: then a waiting
//            CTA's predecessor runs. CUDA promises neither; the hardware hands CTAs out in order, and a grid has one a SM. With both
//            broken (another process's waiting kernel on the SMs that are missing) the wait gives up by its limit and the call fails.
//            Numbers taken from a counter as CTAs start need no such order; they cost the start a round trip: 28672 x 4096 at 1 row 16.1
//            -> 16.5 us, the one-row step of the 8B model 2025 -> 2053. A cooperative launch: 16.1 -> 20.0, 2025 -> 2143
//   IN_TURN  a team takes a (pair, chunk) at a time, its splits one after the other, their sums in shared memory
constexpr int QL_MAX_SPLITS = 16;
constexpr uint32_t QL_NOTHING = 0xFFFFFFFFu;
enum : int { QL_APART = 0, QL_RUNS = 1, QL_IN_TURN = 2 };

struct QlKernelParams {
  const uint8_t* records;
  uint32_t record_bytes;
  int N, kblocks, n_pairs;
  int splits;            // parts of a pair (split s has k-blocks [K s / S, K (s + 1) / S)), added in order
  int chains;            // of a part: one, or its even and its odd k-blocks apart
  int teams;             // of the grid
  int M, m_pad, chunks;  // live rows of the launch; rows of a chunk, a multiple of 16, of 32 in a cluster
  int row0;              // first activation row
  int way;
  int a_slots, b_slots, r_slots, accs;   // ring depths, in units: dequantised weights, activations, records; accumulators with a barrier
  uint32_t tmem_cols;    // columns allocated: a power of two
  QlFactors factors;
  float back0, back1;    // the products' sums times back0 * back1 = 2^shift
  int glu;               // 0, or 1 (silu) / 2 (gelu_approx): act = activation(gate) * up, see ql_drain
  bf16* act; int ld_act;
  int vec;               // rows of y, or of the partials, start on 16 bytes, and whole groups of 8 (4) features
  bf16* y; int ldy;
  float* partial;        // APART with several splits: [splits][M][N]
  uint4* fix;            // RUNS: [chunk][team][CTA][m_pad / 4][128], see ql_fix_slot
  uint32_t* status;
};

// first, last: whether it has its pair's first split or k-block, its last; acc: the accumulator, its wait's parity above; of a
// cluster's second chain: acc1
struct QlTask { int pair, chunk, split, kb0, nkb; bool first, last; uint32_t acc, acc1; };

// Where the work of a CTA is cut, in shared memory: a division takes one of the single-thread roles a microsecond between the
// arithmetic of the dequantisers, so one idle warp does them all before the roles start.
struct QlCuts {
  int r0, r1, p0, segments;            // RUNS: the run (in a pair it starts at an even k-block: only a pair's end makes half a unit), its first pair, its pairs
  int pair, chunk;                     // IN_TURN: the team's first item
  int units;                           // of all tasks
  int split[QL_MAX_SPLITS + 1];        // k-blocks where the splits of a pair start
};
template <int UNIT>
__device__ __forceinline__ void ql_cut(const QlKernelParams& p, QlCuts* c, int lane) {
  const unsigned team = blockIdx.x >> 1, K = p.kblocks;
  auto of = [](int k) { return (k + UNIT - 1) / UNIT; };
  if (lane <= p.splits) c->split[lane] = K * lane / p.splits;
  __syncwarp();
  if (lane) return;
  int n = 0;
  if (p.way == QL_RUNS) {
    auto start = [&](unsigned t) {
      const int at = (int)((unsigned long long)p.n_pairs * K * t / p.teams);
      return at - (at % (int)K & 1);
    };
    c->r0 = start(team); c->r1 = start(team + 1);
    c->p0 = c->r0 / (int)K;
    int pairs = 0;
    for (int a = c->r0, e = (c->p0 + 1) * K; a < c->r1; a = e, e += K, ++pairs) n += of(min(c->r1, e) - a);
    c->segments = pairs;
    n *= p.chunks;
  } else if (p.way == QL_APART) {
    n = of(c->split[blockIdx.y + 1] - c->split[blockIdx.y]);
  } else {
    for (int i = 0; i < p.splits; ++i) n += of(c->split[i + 1] - c->split[i]);
    n *= (p.n_pairs * p.chunks - team + p.teams - 1) / p.teams;
    c->pair = team % p.n_pairs; c->chunk = team / p.n_pairs;
  }
  c->units = n;
}

// The tasks of a team, in order.
struct QlTasks {
  const QlKernelParams& p;
  const QlCuts& c;
  int at = 0, chunk = 0;      // APART: done; RUNS: segment of the run, chunk; IN_TURN: the item's pair, chunk
  int split = 0;              // IN_TURN: of the item, the next one
  __device__ QlTasks(const QlKernelParams& params, const QlCuts& cuts) : p(params), c(cuts) {
    if (p.way == QL_IN_TURN) { at = c.pair; chunk = c.chunk; }
  }
  // Segments of a run: what another team waits for comes first, what waits for another team last: the run's last pair, of which
  // it may hold a part without the end; the whole pairs; its first pair, whose start may be another's.
  __device__ bool next(QlTask& t) {
    const int K = p.kblocks;
    if (p.way == QL_RUNS) {
      if (chunk >= p.chunks) return false;
      const int n = c.segments, pair = c.p0 + (at == 0 ? n - 1 : at == n - 1 ? 0 : at);
      const int a = max(c.r0, pair * K), b = min(c.r1, (pair + 1) * K);
      t = QlTask{pair, chunk, 0, a - pair * K, b - a, a == pair * K, b == (pair + 1) * K, 0, 0};
      if (++at == n) { at = 0; ++chunk; }
      return true;
    }
    if (p.way == QL_APART) {
      if (at++) return false;
      const int s = blockIdx.y;
      t = QlTask{(int)(blockIdx.x >> 1), (int)blockIdx.z, s, c.split[s], c.split[s + 1] - c.split[s], s == 0, s == p.splits - 1, 0, 0};
      return true;
    }
    if (chunk >= p.chunks) return false;
    t = QlTask{at, chunk, split, c.split[split], c.split[split + 1] - c.split[split], split == 0, split == p.splits - 1, 0, 0};
    if (++split == p.splits) {
      split = 0; at += p.teams;
      while (at >= p.n_pairs) { at -= p.n_pairs; ++chunk; }
    }
    return true;
  }
  // A task that goes on from another team's sums.
  __device__ bool goes_on(const QlTask& t) const { return p.way == QL_RUNS && !t.first; }
  // The part has an odd k-block: a second chain that is no chain of nothing.
  __device__ bool second(const QlTask& t) const { return p.chains == 2 && t.nkb > 1; }
};

// The sums that a run leaves of a pair whose end it does not hold: [row / 4][128][4], of a CTA. Between launches every word is
// QL_NOTHING, and a word that is something else is there: the reader polls the sums themselves and puts QL_NOTHING back. A word
// that says so needs a fence before it, which took 4 us beside the copies that are under way. Relaxed accesses on both sides: a plain store beside
// a load of the same word would be a race.
__device__ __forceinline__ uint4* ql_fix_slot(const QlKernelParams& p, int chunk, int team, int row) {
  return p.fix + (((size_t)chunk * p.teams + team) * 2 + (blockIdx.x & 1)) * (p.m_pad / 4) * QL_TILE_N + row;
}
__device__ __forceinline__ bool ql_fix_load(const uint4* src, uint4& v) {
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(src) : "memory");
  return v.x != QL_NOTHING && v.y != QL_NOTHING && v.z != QL_NOTHING && v.w != QL_NOTHING;
}

__device__ __forceinline__ void ql_fix_store(uint4* dst, uint4 v) {
  asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// Puts another team's sums into a task's accumulator: one group's warps, a lane quarter each.
__device__ __forceinline__ bool ql_go_on(const QlKernelParams& p, const QlTask& t, uint32_t acc, int q, int lane) {
  uint4* src = ql_fix_slot(p, t.chunk, (blockIdx.x >> 1) - 1, q * 32 + lane);
  const uint4 nothing = make_uint4(QL_NOTHING, QL_NOTHING, QL_NOTHING, QL_NOTHING);
  const int last = p.m_pad / 4 - 1;
  for (int s = 0; s < p.m_pad; s += 32) {   // a round trip to L2 each; the last 16 rows may be past the chunk's, in columns that nothing else has
    uint4 f[8];
    unsigned long long t0 = 0;
    while (true) {
      bool there = true;
#pragma unroll
      for (int j = 0; j < 8; ++j) there &= ql_fix_load(src + min(s / 4 + j, last) * QL_TILE_N, f[j]);
      if (__all_sync(0xffffffffu, there)) break;
      const unsigned long long now = globaltimer_ns();
      if (t0 == 0) t0 = now;
      if (__any_sync(0xffffffffu, now - t0 > KC_SPIN_LIMIT_NS)) {
        if (p.status) atomicOr(p.status, KC_DEV_QLINEAR | 9u);
        return false;
      }
    }
    uint32_t v[32];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      v[4 * j] = f[j].x; v[4 * j + 1] = f[j].y; v[4 * j + 2] = f[j].z; v[4 * j + 3] = f[j].w;
      if (s / 4 + j <= last) ql_fix_store(src + (s / 4 + j) * QL_TILE_N, nothing);
    }
    tmem_st32(acc + s, v);
  }
  tmem_wait_st();
  return true;
}

// Leaves a run's sums of a pair for the team that has its end: one group's warps, a lane quarter each.
__device__ __forceinline__ void ql_leave(const QlKernelParams& p, const QlTask& t, uint32_t acc, int q, int lane) {
  uint4* dst = ql_fix_slot(p, t.chunk, blockIdx.x >> 1, q * 32 + lane);
  for (int s = 0; s < p.m_pad; s += 16, dst += 4 * QL_TILE_N) {
    uint32_t e[16];
    tmem_ld16_issue(acc + s, e);
    tmem_wait_ld();
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      asm volatile("" : "+r"(e[j]));   // no use before the wait
      e[j] = e[j] == QL_NOTHING ? 0x7FFFFFFFu : e[j];   // both are NaN
    }
#pragma unroll
    for (int j = 0; j < 16; j += 4) ql_fix_store(dst + j / 4 * QL_TILE_N, make_uint4(e[j], e[j + 1], e[j + 2], e[j + 3]));
  }
}

// The sums of the parts so far, in shared memory: [row / 4][128][4].
__device__ __forceinline__ float4* ql_sums_of(float* sums, int row, int n_in) { return reinterpret_cast<float4*>(sums) + row / 4 * QL_TILE_N + n_in; }
__device__ __forceinline__ void ql_add4(float* v, float4 o) {
  const float2 a = add2(make_float2(o.x, o.y), make_float2(v[0], v[1])), b = add2(make_float2(o.z, o.w), make_float2(v[2], v[3]));
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}

// A group's share of a task's accumulator, with its second chain's where there is one: slices of columns (rows of the step), every
// ng-th from gi. A thread has one weight row (TMEM lane). What is not a pair's last task leaves its sums (in shared memory, or as partials for the next kernel); the last one writes
// y, or the gated activation: in such a weight 16 gate rows and the 16 up rows of the same features take turns, so the two meet in a
// warp. Where the output's rows allow it (p.vec) values leave 8 or 16 bytes a lane, through a buffer of the warp.
//
// Few rows: slices of 8 in a loop of little code. What bounds it is the fetch of its instructions, which a CTA meets for the first
// time at its end: 8B decode steps of 32 rows 6113 -> 5972 us against the form below.
__device__ __forceinline__ void ql_drain(const QlKernelParams& p, const QlTask& t, uint32_t acc, bool two, uint32_t acc1, int gi, int ng, float* sums, uint8_t* stage, int q, int lane) {
  const int tile = 2 * t.pair + (blockIdx.x & 1), n0 = tile * QL_TILE_N + q * 32;
  const bool in_turn = p.way == QL_IN_TURN;
  float* buf = reinterpret_cast<float*>(stage);   // [8][36]
  const int r = lane >> 2, f = (lane & 3) * 8, n = n0 + f;   // the lane's row and features on the way out
#pragma unroll 1
  for (int s = gi * 8; s < p.m_pad; s += ng * 8) {
    const int m = t.chunk * p.m_pad + s + r;
    __syncwarp();                        // lanes left the last turn apart; the loads are the warp's
    float v[8];
    {
      uint32_t e[8], o[8];
      tmem_ld8_issue(acc + s, e);
      if (two) tmem_ld8_issue(acc1 + s, o);
      tmem_wait_ld();
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        asm volatile("" : "+r"(e[j]), "+r"(o[j]));   // no use before the wait
        v[j] = (two ? __uint_as_float(e[j]) + __uint_as_float(o[j]) : __uint_as_float(e[j])) * p.back0 * p.back1;
      }
    }
    if (in_turn && !(t.first && t.last)) {
      float4* before = ql_sums_of(sums, s, q * 32 + lane);
#pragma unroll
      for (int j = 0; j < 8; j += 4) {
        if (!t.first) ql_add4(v + j, before[j / 4 * QL_TILE_N]);
        if (!t.last) before[j / 4 * QL_TILE_N] = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
      }
      if (!t.last) continue;
    }
    __syncwarp();                        // the last turn's reads of the buffer are done
#pragma unroll
    for (int j = 0; j < 8; ++j) buf[j * 36 + lane] = v[j];
    __syncwarp();
    if (!p.vec) {                        // a lane a feature, row by row
      const bool apart = p.way == QL_APART && p.splits > 1;
      const int first = m - r;
#pragma unroll 1
      for (int j = 0; j < 8 && first + j < p.M; ++j) {
        const float x = buf[j * 36 + lane];
        if (n0 + lane >= p.N) continue;
        if (apart) p.partial[((size_t)t.split * p.M + first + j) * p.N + n0 + lane] = x;
        else p.y[(size_t)(p.row0 + first + j) * p.ldy + n0 + lane] = __float2bfloat16_rn(x);
      }
      continue;
    }
    if (m >= p.M) continue;
    if (p.glu) {                         // four features of a row: gate at 32 of a warp's k .., up 16 further
      const int c = (lane & 3) * 4;
      const float4 g = *reinterpret_cast<const float4*>(buf + r * 36 + c), u = *reinterpret_cast<const float4*>(buf + r * 36 + 16 + c);
      const uint2 o = make_uint2(act_pair(pack_bf162(g.x, g.y), pack_bf162(u.x, u.y), p.glu == 2), act_pair(pack_bf162(g.z, g.w), pack_bf162(u.z, u.w), p.glu == 2));
      if (tile * QL_TILE_N < p.N) *reinterpret_cast<uint2*>(p.act + (size_t)(p.row0 + m) * p.ld_act + tile * 64 + q * 16 + c) = o;
      continue;
    }
    const float4 a = *reinterpret_cast<const float4*>(buf + r * 36 + f), b = *reinterpret_cast<const float4*>(buf + r * 36 + f + 4);
    if (p.way == QL_APART && p.splits > 1) {
      float* dst = p.partial + ((size_t)t.split * p.M + m) * p.N + n;
      if (n < p.N) *reinterpret_cast<float4*>(dst) = a;
      if (n + 4 < p.N) *reinterpret_cast<float4*>(dst + 4) = b;
    } else {
      bf16* dst = p.y + (size_t)(p.row0 + m) * p.ldy + n;
      if (n < p.N) *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf162(a.x, a.y), pack_bf162(a.z, a.w), pack_bf162(b.x, b.y), pack_bf162(b.z, b.w));
    }
  }
}

// Many rows: slices of 16, unrolled, lanes taking eight rows of the activation each. The first group's warps get an instruction in about
// ten cycles between those of the dequantisers, so their number counts: 4096 x 14336 at 2048 rows 175 -> 163 us against the form
// above, with stores of 2 bytes a lane 172.
__device__ __forceinline__ void ql_drain_wide(const QlKernelParams& p, const QlTask& t, uint32_t acc, bool two, uint32_t acc1, int gi, int ng, float* sums, uint8_t* stage, int q, int lane) {
  const int tile = 2 * t.pair + (blockIdx.x & 1), n_in = q * 32 + lane, n0 = tile * QL_TILE_N + q * 32, n = n0 + lane;
  const bool live = n < p.N, in_turn = p.way == QL_IN_TURN, apart = p.way == QL_APART && p.splits > 1;
  for (int s = gi; s < p.m_pad >> 4; s += ng) {
    const int m0 = t.chunk * p.m_pad + s * 16, rows = min(16, p.M - m0);
    __syncwarp();                        // as above
    float v[16];
    {
      uint32_t e[16];
      tmem_ld16_issue(acc + s * 16, e);
      tmem_wait_ld();
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        asm volatile("" : "+r"(e[j]));   // no use before the wait
        v[j] = __uint_as_float(e[j]);
      }
      if (two) {
        tmem_ld16_issue(acc1 + s * 16, e);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          asm volatile("" : "+r"(e[j]));
          v[j] += __uint_as_float(e[j]);
        }
      }
    }
    if (p.back0 != 1.f) {
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = v[j] * p.back0 * p.back1;
    }
    float4* before = ql_sums_of(sums, s * 16, n_in);
    if (in_turn && !t.first) {
#pragma unroll
      for (int j = 0; j < 16; j += 4) ql_add4(v + j, before[j / 4 * QL_TILE_N]);
    }
    if (in_turn && !t.last) {
#pragma unroll
      for (int j = 0; j < 16; j += 4) before[j / 4 * QL_TILE_N] = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
    } else if (apart) {
      float* out = p.partial + ((size_t)t.split * p.M + m0) * p.N;
      if (p.vec) {
        float* buf = reinterpret_cast<float*>(stage);   // [8][36]
        const int r = lane >> 3, f = (lane & 7) * 4;
        float* dst = out + (size_t)r * p.N + n0 + f;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 8; ++j) buf[j * 36 + lane] = v[8 * h + j];
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 2; ++k, dst += (size_t)4 * p.N) {
            const float4 x = *reinterpret_cast<const float4*>(buf + (4 * k + r) * 36 + f);
            if (8 * h + 4 * k + r < rows && n0 + f < p.N) *reinterpret_cast<float4*>(dst) = x;
          }
        }
      } else if (live) {
        float* dst = out + n;
#pragma unroll
        for (int j = 0; j < 16; ++j, dst += p.N)
          if (j < rows) *dst = v[j];
      }
    } else if (p.glu) {
      if (tile * QL_TILE_N < p.N) {     // whole tiles only
        uint32_t pair[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) pair[j] = pack_bf162(v[2 * j], v[2 * j + 1]);
        const bool up = lane & 16;      // this lane has up values; it takes rows 8 .. 15, its gate lane 0 .. 7
        uint16_t* buf = reinterpret_cast<uint16_t*>(stage) + (up ? 8 * 24 : 0) + (lane & 15);   // [16][24]
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? pair[j] : pair[4 + j], 16);
          const uint32_t o = act_pair(up ? got : pair[j], up ? pair[4 + j] : got, p.glu == 2);
          buf[2 * j * 24] = (uint16_t)(o & 0xFFFFu);
          buf[(2 * j + 1) * 24] = (uint16_t)(o >> 16);
        }
        __syncwarp();
        const int r = lane >> 1, f = (lane & 1) * 8;
        if (r < rows)
          *reinterpret_cast<uint4*>(p.act + (size_t)(p.row0 + m0 + r) * p.ld_act + tile * 64 + q * 16 + f) =
              *reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(stage) + r * 24 + f);
      }
    } else if (p.vec) {
      bf16* buf = reinterpret_cast<bf16*>(stage);       // [16][40]
      const int r = lane >> 2, f = (lane & 3) * 8;
      bf16* dst = p.y + (size_t)(p.row0 + m0 + r) * p.ldy + n0 + f;
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 16; ++j) buf[j * 40 + lane] = __float2bfloat16_rn(v[j]);
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 2; ++k, dst += (size_t)8 * p.ldy) {
        const uint4 x = *reinterpret_cast<const uint4*>(buf + (8 * k + r) * 40 + f);
        if (8 * k + r < rows && n0 + f < p.N) *reinterpret_cast<uint4*>(dst) = x;
      }
    } else if (live) {
      bf16* dst = p.y + (size_t)(p.row0 + m0) * p.ldy + n;
#pragma unroll
      for (int j = 0; j < 16; ++j, dst += p.ldy)
        if (j < rows) *dst = __float2bfloat16_rn(v[j]);
    }
  }
}

// ---------------------------------------------------------------------------
// The kernel. The dequantised weights reach the tensor core through TENSOR MEMORY (tcgen05.mma with the A operand in TMEM),
// not through shared memory. A dequantiser thread owns one weight row (= one TMEM lane) of a UNIT, one or two 64-feature
// k-blocks of a 128-row tile, expands the 64 weights of a k-block in registers and writes them with one tcgen05.st (column c =
// weights 2c and 2c + 1), so the MMAs read only the activation k-block from shared memory.
//
// TMEM columns: [accs accumulators of round32(m_pad)] [a_slots x unit x 32 columns of bf16 pairs]. With two chains an accumulator is two
// beside each other where CTAs work alone: a unit has a k-block of each. A cluster takes a task's even k-blocks first, then the odd ones, and each
// chain has an accumulator with a barrier of its own: three of 128 rows are as many as tensor memory holds, and the third is what a task starts
// with while the one before it is drained.
// ---------------------------------------------------------------------------

// A wait whose loop holds little. It gives up by the clock, which is looked at once in a thousand tries, however long one takes, and starts when
// the kernel ahead is done: all roles but the first units' dequantisation depend on that one, and it may take long. In one piece, since a loop of
// the compiler's took 28672 x 4096 at 1 and 32 rows from 16.1 and 16.9 us to 16.4 and 17.2, and with the rest in a function that is called to 16.4
// and 17.0 (192 rows 36.7 -> 37.1).
__device__ __forceinline__ bool ql_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;   // nanoseconds: 32 bits of them are 4.3 s
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .u32 tries, start, t;\n\t"
      "mov.u32 tries, 0;\n\tmov.u32 start, 0;\n"
      "AGAIN%=:\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "@p bra OVER%=;\n\t"
      "add.u32 tries, tries, 1;\n\t"
      "and.b32 t, tries, 1023;\n\t"
      "setp.ne.u32 q, t, 0;\n\t"
      "@q bra AGAIN%=;\n\t"
      "griddepcontrol.wait;\n\t"
      "mov.u32 t, %%globaltimer_lo;\n\t"
      "setp.eq.u32 q, tries, 1024;\n\t"
      "selp.u32 start, t, start, q;\n\t"
      "sub.u32 t, t, start;\n\t"
      "setp.le.u32 q, t, %4;\n\t"
      "@q bra AGAIN%=;\n"
      "OVER%=:\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(20000u), "n"((uint32_t)KC_SPIN_LIMIT_NS)
      : "memory");
  return ok != 0;
}
// What was asked for still lands in shared memory; it takes microseconds.
__device__ __noinline__ void ql_gave_up(uint32_t* status, uint32_t wait) {
  if (status) atomicOr(status, KC_DEV_QLINEAR | wait);
  const unsigned long long t0 = globaltimer_ns();
  while (globaltimer_ns() - t0 < 2000000ull) {}
}

template <int CG>
__device__ __forceinline__ void ql_mma(uint32_t d, uint32_t a, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, uint32_t accumulate) {
  if (CG == 1) umma_bf16_ts(d, a, b_lo, b_hi, idesc, accumulate);
  else umma_bf16_ts_pair(d, a, b_lo, b_hi, idesc, accumulate);
}
template <int CG>
__device__ __forceinline__ void ql_commit(uint32_t bar) {
  if (CG == 1) umma_commit(bar);
  else umma_commit_pair(bar);
}

template <int BITS, int GPK, int CG, bool WIDE>
__global__ void __launch_bounds__(QL_THREADS, 1)
qlinear_umma_kernel(const __grid_constant__ CUtensorMap map_rows, const __grid_constant__ QlKernelParams p) {
  constexpr uint32_t PACKED = QL_TILE_N * (QL_KB * BITS / 8);
  constexpr int UNIT = ql_unit(CG), DQ = QL_GROUPS - 1;   // the first group drains
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t kb_bytes = (uint32_t)p.m_pad / CG * 128u, b_bytes = UNIT * kb_bytes;   // this CTA's rows of a k-block, of a unit
  const uint32_t r_bytes = UNIT * p.record_bytes;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int side = blockIdx.x & 1;             // in a cluster: the CTA's rank
  const uint32_t cs = (uint32_t)(p.m_pad + 31) & ~31u, acc_cols = CG == 1 ? p.chains * cs : cs, a_col0 = p.accs * acc_cols;
  const int loops = CG == 1 ? 1 : p.chains, halves = loops - 1;   // a task's k-blocks are taken `loops` at a step, as often

  uint8_t* sB = smem;
  uint8_t* sR = sB + (size_t)p.b_slots * b_bytes;
  uint8_t* stage = sR + (size_t)p.r_slots * r_bytes;
  float* sums = reinterpret_cast<float*>(stage + 4 * QL_GROUPS * QL_STAGE_BYTES);
  const bool has_sums = p.way == QL_IN_TURN && p.splits > 1;
  // Barriers, by shared address: 8 bytes each. The n-th unit has record slot n % r_slots, A slot n % a_slots and activation slot
  // n % b_slots.
  uint64_t* bars = reinterpret_cast<uint64_t*>(sums + (has_sums ? p.m_pad * QL_TILE_N : 0));
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars);
  QlTask* last_task = reinterpret_cast<QlTask*>(bars + 2);   // with its accumulator, for the groups that join at the end
  const uint32_t r_end = 8 * p.r_slots, b_end = 8 * p.b_slots;
  QlCuts* cuts = reinterpret_cast<QlCuts*>(bars + 8);
  const uint32_t raw_full = smem_u32(bars + 8 + (sizeof(QlCuts) + 7) / 8);   // by record slot: the records are in ..
  const uint32_t raw_empty = raw_full + r_end;    // .. and read
  const uint32_t done = raw_empty + r_end;        // by activation slot: the unit's products are; its other slots are free
  const uint32_t ready = done + b_end;            // .. its activations are in, of both CTAs, and its weights dequantised
  const uint32_t acc_full = ready + b_end;        // an accumulator's products are in
  const uint32_t acc_free = acc_full + 32;        // .. it has been read, and holds what the next ones go on from

  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int i = 0; i < p.r_slots; ++i) { mbar_init(raw_full + 8 * i, 1); mbar_init(raw_empty + 8 * i, 4); }
    for (int i = 0; i < p.b_slots; ++i) { mbar_init(ready + 8 * i, 4 * CG + 1); mbar_init(done + 8 * i, 1); }
    for (int i = 0; i < p.accs; ++i) { mbar_init(acc_full + 8 * i, 1); mbar_init(acc_free + 8 * i, 4 * CG); }
    mbar_fence_init();
  }
  if (warp == 2) tmem_alloc<CG>(tmem_slot, p.tmem_cols);
  if (warp == 1 && lane == 0) tma_prefetch_desc(&map_rows);
  if (warp == 3) ql_cut<UNIT>(p, cuts, lane);
  tc_fence_before();
  __syncthreads();
  if (CG == 2) cluster_sync();   // the other CTA's barriers are there
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp < QL_GROUP0) {
    // ---- The roles of one thread each. In a turn of their loops a taken branch costs about 100 cycles, beside the arithmetic of
    // the dequantiser warps on the same scheduler, and the turn has to keep up with a unit's products: so tasks are loops of their
    // own with running addresses, a wait is one loop around one instruction, and one barrier stands for all that a unit waits for. ----
    if (warp == 0 && elect_one()) {
      // the weight records, which depend on no kernel before this one
      const uint32_t r0 = smem_u32(sR);
      const size_t pitch = (size_t)QL_TILE_GROUP * p.record_bytes, step = pitch * (CG == 1 ? UNIT : loops);
      uint32_t dst = r0, slot = 0, phase = 1;
      bool ok = true;
      QlTasks tasks(p, *cuts);
      QlTask t;
      while (ok && tasks.next(t)) {
        const int tile = 2 * t.pair + side;
        const uint8_t* first = p.records + ((size_t)(tile / QL_TILE_GROUP) * p.kblocks + t.kb0) * pitch + (size_t)(tile % QL_TILE_GROUP) * p.record_bytes;
        const uint8_t* src = first;
        auto copy = [&](int kbs) {
          const uint32_t full = raw_full + slot;
          ok = ql_wait(raw_empty + slot, phase);
          if (!ok) return;
          mbar_arrive_expect_tx(full, kbs * p.record_bytes);
          bulk_g2s(dst, src, p.record_bytes, full);
          if (kbs > 1) bulk_g2s(dst + p.record_bytes, src + pitch, p.record_bytes, full);
          src += step; dst += r_bytes; slot += 8;
          if (slot == r_end) { slot = 0; dst = r0; phase ^= 1u; }
        };
        if (UNIT == 2) {
          for (int n = t.nkb / 2; ok && n > 0; --n) copy(2);
          if (ok && (t.nkb & 1)) copy(1);
        } else {
          for (int c = 0; c < loops; ++c) {
            src = first + c * pitch;
            for (int n = (t.nkb + halves - c) >> halves; ok && n > 0; --n) copy(1);
          }
        }
      }
      if (!ok) ql_gave_up(p.status, 1);
    } else if (warp == 1 && elect_one()) {
      // the activations, the first access of this kernel to memory written by earlier kernels
      pdl_wait();
      const uint32_t b0 = smem_u32(sB), lead = CG == 2 ? cluster_addr(ready, 0) : ready;
      uint32_t dst = b0, slot = 0, phase = 1;
      bool ok = true;
      QlTasks tasks(p, *cuts);
      QlTask t;
      while (ok && tasks.next(t)) {
        const int row = p.row0 + t.chunk * p.m_pad + (CG == 2 ? side * (p.m_pad / 2) : 0);
        int x = t.kb0 * QL_KB;
        const int step = QL_KB * (CG == 1 ? UNIT : loops);
        auto copy = [&](int kbs) {
          ok = ql_wait(done + slot, phase);
          if (!ok) return;
          if (CG == 1 || side == 0) mbar_arrive_expect_tx(ready + slot, kbs * kb_bytes * CG);
          tma_load_2d_pair<CG>(dst, &map_rows, x, row, lead + slot);
          if (kbs > 1) tma_load_2d_pair<CG>(dst + kb_bytes, &map_rows, x + QL_KB, row, lead + slot);
          x += step; dst += b_bytes; slot += 8;
          if (slot == b_end) { slot = 0; dst = b0; phase ^= 1u; }
        };
        if (UNIT == 2) {
          for (int n = t.nkb / 2; ok && n > 0; --n) copy(2);
          if (ok && (t.nkb & 1)) copy(1);
        } else {
          for (int c = 0; c < loops; ++c) {
            x = (t.kb0 + c) * QL_KB;
            for (int n = (t.nkb + halves - c) >> halves; ok && n > 0; --n) copy(1);
          }
        }
      }
      if (!ok) ql_gave_up(p.status, 2);
    } else if (warp == 2 && (CG == 1 || side == 0) && elect_one()) {
      // the MMAs. With the loop around the election four of them and two commits took the warp 160 cycles to issue alone, this way 65.
      pdl_wait();
      const uint32_t idesc = umma_idesc_bf16(QL_TILE_N * CG, p.m_pad);
      const uint64_t proto = umma_smem_desc(0, 1024);
      const uint32_t d_hi = (uint32_t)(proto >> 32), b_lo0 = (uint32_t)proto | ((smem_u32(sB) >> 4) & 0x3FFF), b_step = b_bytes >> 4, kb_step = kb_bytes >> 4;
      const uint32_t a_first = tmem_base + a_col0, a_last = a_first + p.a_slots * UNIT * 32;
      uint32_t a_t = a_first, b_lo = b_lo0, slot = 0, phase = 0;
      uint32_t buf = 0, fphase = 0;                   // the accumulator
      const uint32_t apart = CG == 1 && p.chains == 2 ? cs : 0u, one = apart ? 0u : 1u;   // a unit's second k-block: to its own chain, or after the first
      bool ok = true;
      QlTasks tasks(p, *cuts);
      QlTask t;
      while (ok && tasks.next(t)) {
       for (int c = 0; ok && c < loops; ++c) {
        ok = ql_wait(acc_free + 8 * buf, fphase);
        const uint32_t d = tmem_base + buf * acc_cols;
        uint32_t acc = tasks.goes_on(t) ? 1u : 0u;
        auto issue = [&](int kbs) {
          ok = ql_wait(ready + slot, phase);
          if (!ok) return;
          tc_fence_after();   // the A operand was written with tcgen05.st by other threads
#pragma unroll
          for (int ks = 0; ks < QL_KB / 16; ++ks) ql_mma<CG>(d, a_t + 8 * ks, b_lo + 2 * ks, d_hi, idesc, ks == 0 ? acc : 1u);
          if (kbs > 1) {
#pragma unroll
            for (int ks = 0; ks < QL_KB / 16; ++ks) ql_mma<CG>(d + apart, a_t + 32 + 8 * ks, b_lo + kb_step + 2 * ks, d_hi, idesc, ks == 0 ? acc | one : 1u);
          }
          acc = 1;
          ql_commit<CG>(done + slot);
          a_t += UNIT * 32; b_lo += b_step; slot += 8;
          if (a_t == a_last) a_t = a_first;
          if (slot == b_end) { slot = 0; b_lo = b_lo0; phase ^= 1u; }
        };
        if (UNIT == 2) {
          for (int n = t.nkb / 2; ok && n > 0; --n) issue(2);
          if (ok && (t.nkb & 1)) issue(1);
        } else {
          for (int n = (t.nkb + halves - c) >> halves; ok && n > 0; --n) issue(1);
        }
        if (ok) ql_commit<CG>(acc_full + 8 * buf);
        if (++buf == (uint32_t)p.accs) { buf = 0; fphase ^= 1u; }
       }
      }
      if (!ok) ql_gave_up(p.status, 4);
    }
    __syncwarp();
  } else {
    const int group = (warp - QL_GROUP0) >> 2, q = warp & 3;
    const uint32_t lanes = tmem_base + ((uint32_t)(q * 32) << 16);
    stage += (warp - QL_GROUP0) * QL_STAGE_BYTES;
    bool ok = true;
    QlTasks tasks(p, *cuts);
    if (group > 0) {
      // ---- dequantisers: thread = one weight row (TMEM lane 32 q + lane) of every third unit. The first slots are filled under the
      // tail of the previous kernel. A wait names a slot's use by its parity: r_slots is a multiple of three, so that a group meets
      // every use of its record slots, and units are done in order. ----
      const uint32_t d = group - 1;
      const uint32_t row0 = smem_u32(sR) + (q * 32 + lane) * 16, sb0 = smem_u32(sR) + PACKED + (q * 32 + lane) * (GPK * 4);
      const uint32_t lead = CG == 2 ? cluster_addr(ready, 0) : ready;
      const uint32_t a0 = lanes + a_col0, a_end = a0 + p.a_slots * UNIT * 32;
      uint32_t rec = d * r_bytes, raw = 8 * d, a_t = a0 + UNIT * 32 * d, bar = raw, phase = 0;
      uint32_t old = 8 * (p.b_slots - p.a_slots + d), freed = 1;   // barrier of the unit that had the A slot before; none at first
      for (int left = cuts->units - (int)d; left > 0; left -= DQ) {
        ok = __all_sync(0xffffffffu, ql_wait(raw_full + raw, phase));
        if (!ok) break;
#pragma unroll
        for (int k = 0; k < UNIT; ++k) {   // of half a unit at a task's end, the second half is what the slot held before: no MMA reads it
          uint32_t v[32];
          dequant_row<BITS, GPK, WIDE>(row0 + rec + k * p.record_bytes, sb0 + rec + k * p.record_bytes, p.factors, v);
          if (k == 0) {
            ok = __all_sync(0xffffffffu, ql_wait(done + old, freed));
            if (!ok) break;
            tc_fence_after();
          }
          tmem_st32(a_t + 32 * k, v);
        }
        if (!ok) break;
        __syncwarp();
        if (lane == 0) mbar_arrive(raw_empty + raw);   // the records are in registers
        raw += 8 * DQ; rec += DQ * r_bytes;
        if (raw >= r_end) { raw -= r_end; rec -= p.r_slots * r_bytes; phase ^= 1u; }
        a_t += DQ * UNIT * 32;
        if (a_t >= a_end) a_t -= p.a_slots * UNIT * 32;
        old += 8 * DQ;
        if (old >= b_end) { old -= b_end; freed ^= 1u; }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (CG == 1) mbar_arrive(ready + bar);
          else mbar_arrive_cluster(lead + bar);
        }
        bar += 8 * DQ;
        if (bar >= b_end) bar -= b_end;
      }
      if (!ok) ql_gave_up(p.status, 5);
    }
    // ---- the first group prepares accumulators and drains them, a task under the products of the next one; the last task's is
    // everybody's ----
    QlTasks ahead(p, *cuts);
    QlTask t{}, next{}, fresh{};
    bool more = group == 0 && tasks.next(next), some = group == 0 && ahead.next(fresh), last = group > 0, released = false;
    uint32_t acc = 0, facc = 0;                    // index in bits 0 and 1, parity in bit 2
    int prepared = 0, chain = 0;                   // accumulators that are, of tasks not yet drained; of `fresh`, the next one
    auto turn = [&](uint32_t a) { return (a & 3) + 1 == (uint32_t)p.accs ? (a & 4) ^ 4u : a + 1; };
    auto at = [&](uint32_t a) { return lanes + (a & 3) * acc_cols; };
    while (more || last) {
      if (group == 0) {
        while (some && prepared < p.accs) {
          if (ahead.goes_on(fresh)) {
            // Where the task before it is the one that leaves sums for another team, whichever of the two can go first goes first:
            // if all teams waited to go on they would wait for one another in a row.
            if (prepared > 0 && cuts->segments == 2) {
              const uint4* first = ql_fix_slot(p, fresh.chunk, (blockIdx.x >> 1) - 1, q * 32 + lane);
              if (!released) { pdl_wait(); released = true; }
              bool there = false, over = !ok;
              const unsigned long long t0 = globaltimer_ns();
              while (!there && !over) {
                uint4 v;
                there = __all_sync(0xffffffffu, ql_fix_load(first, v));
                over = __all_sync(0xffffffffu, mbar_test_wait(acc_full + 8 * (acc & 3), acc >> 2)) || __any_sync(0xffffffffu, globaltimer_ns() - t0 > KC_SPIN_LIMIT_NS);
              }
              if (!there) break;
            }
            if (!released) { pdl_wait(); released = true; }
            if (ok) ok = ql_go_on(p, fresh, at(facc), q, lane);
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            if (CG == 1) mbar_arrive(acc_free + 8 * (facc & 3));
            else mbar_arrive_cluster(cluster_addr(acc_free + 8 * (facc & 3), 0));
          }
          facc = turn(facc); ++prepared;
          if (++chain == loops) { chain = 0; some = ahead.next(fresh); }
        }
        t = next; t.acc = acc;
        acc = turn(acc);
        if (loops == 2) { t.acc1 = acc; acc = turn(acc); }
        more = tasks.next(next); last = !more;
      }
      if (last) {   // which one, and the sums so far, are there for all who read them
        if (group == 0 && q == 0 && lane == 0) *last_task = t;
        asm volatile("bar.sync 5, %0;" ::"n"(QL_GROUPS * 128) : "memory");
        t = *last_task;
      }
      if (!released) { pdl_wait(); released = true; }   // the stores may overwrite what an earlier kernel still reads
      if (ok) ok = warp_wait(acc_full + 8 * (t.acc & 3), t.acc >> 2, p.status, KC_DEV_QLINEAR | 7);
      if (ok && loops == 2) ok = warp_wait(acc_full + 8 * (t.acc1 & 3), t.acc1 >> 2, p.status, KC_DEV_QLINEAR | 7);
      tc_fence_after();
      const uint32_t acc0 = at(t.acc), acc1 = CG == 1 ? acc0 + cs : at(t.acc1);
      if (p.way == QL_RUNS && !t.last) {   // never the last task: a run starts with it
        if (ok) ql_leave(p, t, acc0, q, lane);
      } else if (ok) {
        if (CG == 1) ql_drain(p, t, acc0, tasks.second(t), acc1, group, last ? QL_GROUPS : 1, sums, stage, q, lane);
        else ql_drain_wide(p, t, acc0, tasks.second(t), acc1, group, last ? QL_GROUPS : 1, sums, stage, q, lane);
      }
      if (last) break;
      prepared -= loops;
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (CG == 2) cluster_sync();   // nothing of the other CTA's is on its way here, or here any more
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc<CG>(tmem_base, p.tmem_cols);
  }
}

// ---------------------------------------------------------------------------
// Plans
// ---------------------------------------------------------------------------

struct UmmaPlan {
  int cg, way, m_pad, chunks, teams;             // teams: of the grid
  int a_slots, b_slots, r_slots, accs;
  uint32_t tmem_cols;
  size_t smem;
};

static int pairs_of(const QWeight& w) { return (w.n_tiles + 1) / 2; }

size_t qlinear_fix_bytes(int sm_count) { return (size_t)QL_FIX_CHUNKS * (sm_count / 2) * 2 * QL_CHUNK_ROWS * QL_TILE_N * sizeof(float); }

// Ring depths, tensor and shared memory. At least three A slots, the step of a dequantiser group; record slots a multiple of it;
// activation slots, by which a unit's barriers go, as many as A slots at least.
static bool plan_rings(UmmaPlan* t, const QWeight& w, bool several_tasks, bool sums) {
  const int cs = (t->m_pad + 31) & ~31, unit = ql_unit(t->cg);
  // of a cluster an accumulator a chain: a task's, and as much of the next one's as leaves three A slots
  t->accs = t->cg == 1 ? several_tasks + 1 : several_tasks ? std::min(2 * w.chains, std::max(w.chains, (512 - 96) / cs)) : w.chains;
  const int acc_cols = t->accs * (t->cg == 1 ? w.chains * cs : cs);
  t->a_slots = std::min(8, (512 - acc_cols) / (unit * 32));
  const size_t extra = 1024 + 1024 + 4 * QL_GROUPS * QL_STAGE_BYTES + (sums ? (size_t)t->m_pad * QL_TILE_N * 4 : 0);
  const size_t all = (size_t)227 * 1024, b_slot = (size_t)unit * t->m_pad / t->cg * 128, r_slot = (size_t)unit * w.record_bytes;
  auto bytes = [&](int b, int r) { return extra + b * b_slot + r * r_slot; };   // 1024: barriers, at most 24 * 2 + 12 * 2 + 8, and the words before them
  while (t->a_slots > 3 && bytes(t->a_slots, 6) > all) --t->a_slots;
  t->r_slots = 6; t->b_slots = t->a_slots;
  if (t->a_slots < 3 || bytes(t->b_slots, t->r_slots) > all) return false;
  for (bool more = true; more;) {   // deeper as far as there is room
    more = false;
    if (t->r_slots < 24 / unit && bytes(t->b_slots, t->r_slots + 3) <= all) { t->r_slots += 3; more = true; }
    if (t->b_slots < 12 && bytes(t->b_slots + 1, t->r_slots) <= all) { ++t->b_slots; more = true; }
  }
  t->tmem_cols = 32;
  while ((int)t->tmem_cols < acc_cols + t->a_slots * unit * 32) t->tmem_cols <<= 1;
  t->smem = bytes(t->b_slots, t->r_slots);
  return true;
}

// Rows of one or two chunks up to which the CTAs of a team read the activations each for itself. Alone and in pairs, us: 65 rows 4096 x 14336 15.7 and
// 18.4, 28672 x 4096 22.1 and 24.7; 96 rows 17.0 and 19.1, 24.6 and 26.9; 128 rows 19.6 and 20.2, 30.1 and 30.8; 200 rows 26.5 and 30.2, 53.6 and 58.1. Records
// of 9216 bytes leave too little shared memory for units of so many activations: 3584 x 18944 of 8 bits 96 rows 21.8 and 22.4, 112 rows 25.3 and 23.0.
static int solo_rows(const QWeight& w) { return w.record_bytes > 5120 ? 96 : 128; }

// What launches of a weight that is split along K take, in nanoseconds, by the rows of a chunk (96, 128, 160, 192): fitted to 17 weights of 8 to
// 72 tiles, 32 to 448 k-blocks, 4 and 8 bits, at 20 row counts from 193 to 3000. A team's k-block takes what its dequantisation does up to 128 rows,
// then its products' two cycles a row; 160 and 192 rows leave no accumulator to start the next split with while one is drained.
constexpr int QL_APART_NS[2][4] = {{200, 205, 250, 285}, {225, 225, 285, 325}};   // a k-block, of records up to 5120 bytes and of larger ones
constexpr int QL_TURN_NS[2][4] = {{167, 168, 227, 274}, {176, 179, 263, 340}};
constexpr int QL_TURN_END_NS[4] = {1600, 2200, 3000, 3400};                         // a split's end, in turn; half more where there are more than eight
constexpr int QL_APART_START_NS = 6000, QL_TURN_START_NS = 3000;                    // a CTA's start and end: of each wave; of a launch

static long long waves_of(long long tasks, const QWeight& w) { const int teams = std::max(1, w.sm_count / 2); return (tasks + teams - 1) / teams; }
static int chunk_rows(int M, int chunks) { return ((M + chunks - 1) / chunks + 31) & ~31; }
static long long apart_ns(const QWeight& w, int M, int per) {
  const int at = std::max(96, per) / 32 - 3;
  return waves_of((long long)pairs_of(w) * w.splits * ((M + per - 1) / per), w) * ((long long)w.kblocks * QL_APART_NS[w.record_bytes > 5120][at] / w.splits + QL_APART_START_NS);
}
static long long turn_ns(const QWeight& w, int M, int per) {
  const int at = per / 32 - 3;
  return waves_of((long long)pairs_of(w) * ((M + per - 1) / per), w) * ((long long)w.kblocks * QL_TURN_NS[w.record_bytes > 5120][at] + (long long)w.splits * QL_TURN_END_NS[at] * (w.splits > 8 ? 3 : 2) / 2) + QL_TURN_START_NS;
}

// Rows of a chunk where splits are apart. All chunks are one launch; smaller ones than 96 rows take no less time and are only more of them. Of
// 153 launches of 193 to 512 rows that chunks of all four sizes were timed for, the choice takes the fastest but for 3 % in one.
static int plan_apart_rows(const QWeight& w, int M) {
  int best = 0;
  for (int chunks = (M + QL_CHUNK_ROWS - 1) / QL_CHUNK_ROWS; best == 0 || chunks * 96 <= M; ++chunks) {
    const int per = chunk_rows(M, chunks);
    if (best == 0 || apart_ns(w, M, per) < apart_ns(w, M, best) * 98 / 100) best = per;
  }
  return best;
}

constexpr int QL_ROWS_MIN = 257;           // below, a chunk or two of rows never fill the SMs
constexpr int QL_ROWS_MAX_KBLOCKS = 300;   // above, apart and in turn, us: 8192 x 28672 1500 rows 680 and 605, 1024 rows 475 and 391, 7000 x 28672 level
// Whether the rows of a weight that is split along K take its splits in turn, and how many a chunk: 0 where they stay apart. In turn has to be the
// faster way by a fifth in these figures, a call of up to QL_MAX_M rows with a reduction of its own by a third: at rows near the line the
// calls keep the way they had. Apart, with the reduction behind it, and in turn, us: 4096 x 14336 320 rows 41.2 and 42.8, 513 82 and 59, 1024 132 and 94,
// 2048 271 and 183; 4096 x 4096 366 rows 27.9 and 20.1 (the reduction is 7 of the first, which a step does not have), 1024 77 and 42, 2048 153
// and 80; 6144 x 4096 512 rows 46.6 and 28.9; 2048 x 8192 513 rows 43.5 and 37.7, 2048 140 and 85. The reduction takes 2 us and 4570 GB/s over the
// partials and the result, of more rows than QL_MAX_M, whose slabs do not stay in L2, 3060. Summed by the kernel that reads the
// result anyway they cost next to nothing. More than eight splits are short ones, whose ends lie less under the next one's start.
// Against the other way and all chunk sizes, in turn's chunk is 0.3 % behind the fastest on the mean of 340 points, 11 % at most.
static int plan_in_turn_rows(const QWeight& w, int M, bool summed) {
  if (w.splits == 1 || M < QL_ROWS_MIN || w.kblocks > QL_ROWS_MAX_KBLOCKS) return 0;
  auto slab = [&](int rows) { return rows ? apart_ns(w, rows, plan_apart_rows(w, rows)) : 0; };
  long long most = M / QL_MAX_M * slab(M >= QL_MAX_M ? QL_MAX_M : 0) + slab(M % QL_MAX_M);
  const long long bytes = (long long)M * w.N * (4 * w.splits + 2);
  if (M > QL_MAX_M) most += bytes * 100 / 306000;
  else if (!summed) most += 2100 + bytes * 100 / 457000;
  most = most * (M > QL_MAX_M || summed ? 80 : 66) / 100;
  int best = 0;
  for (int per = 96; per <= QL_CHUNK_ROWS; per += 32)
    if (turn_ns(w, M, per) < (best ? turn_ns(w, M, best) : most)) best = per;
  return best;
}
bool qlinear_in_turn(const QWeight& w, int M, bool summed) { return plan_in_turn_rows(w, M, summed) > 0; }

// Rows of a chunk for a weight that is not split along K, and whether its teams share the work by runs: the choice whose products take the least
// time. With two chains, turn_ns of one part; runs would hand on two sums of a cut pair, and lose: 26000 x 2048 at 33 rows, whole pairs and runs,
// 14.3 and 21.1 us, 22016 x 4096 at 192 rows 40.8 and 44.0. With one chain 2 cycles a row and k-block and not less than 300, larger chunks where two
// are level. Runs leave no team idle and cost a cut pair's way through global memory, counted as 20 k-blocks a chunk; fix: chunks that
// they may have. Whole pairs and runs, us: 28672 x 4096 (112 pairs, 74 teams) 1 row 19.0 and 17.8, 33 rows 18.9 and 18.5, 192 rows 43.1 and 40.0, 384
// rows 81.6 and 77.3, 512 rows 96.6 and 108.6; the head's 501 pairs 138 and 142 at 192 rows.
static int plan_whole_rows(const QWeight& w, int M, int fix, bool* runs) {
  const int teams = std::max(1, w.sm_count / 2), pairs = pairs_of(w);
  if (pairs < teams) fix = 0;   // a run holds a whole pair's k-blocks at least
  int best = 0;
  double best_cost = 0;
  for (int per = QL_CHUNK_ROWS; per >= 96; per -= 32) {
    if (per - 32 >= M && per > 96) continue;
    const int chunks = (M + per - 1) / per;
    const double whole = (double)waves_of((long long)pairs * chunks, w) * w.kblocks, cut = ((double)pairs * w.kblocks / teams + 20) * chunks;
    const bool r = w.chains == 1 && chunks <= fix && cut < whole;
    const double cost = w.chains == 2 ? (double)turn_ns(w, M, per) : (r ? cut : whole) * (std::max(300, 2 * per) + 20);
    if (best == 0 || cost < best_cost * 0.995) { best = per; best_cost = cost; *runs = r; }
  }
  return best;
}

template <int BITS, int GPK, int CG, bool WIDE>
static cudaError_t launch_umma(const QLinearLaunch& l, const UmmaPlan& t, const QlKernelParams& p, cudaStream_t s) {
  static DeviceOnce configured;   // the attribute belongs to the device's copy of the kernel
  if (configured.first_on_current_device()) {
    cudaError_t e = cudaFuncSetAttribute(qlinear_umma_kernel<BITS, GPK, CG, WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) { configured.forget_current_device(); return e; }
  }
  const CUtensorMap* rows = act_operand_rows_map(l.x, p.m_pad / CG);
  if (!rows) return cudaErrorInvalidValue;
  const dim3 grid = p.way == QL_APART ? dim3(CG == 2 ? 2 * p.n_pairs : l.w->n_tiles, p.splits, p.chunks) : dim3(2 * t.teams);
  return launch_k_cluster(CG, qlinear_umma_kernel<BITS, GPK, CG, WIDE>, grid, dim3(QL_THREADS), t.smem, s, *rows, p);
}
template <int BITS, int GPK>
static cudaError_t launch_umma_cg(const QLinearLaunch& l, const UmmaPlan& t, const QlKernelParams& p, cudaStream_t s) {
  if (l.w->wide) return t.cg == 2 ? launch_umma<BITS, GPK, 2, true>(l, t, p, s) : launch_umma<BITS, GPK, 1, true>(l, t, p, s);
  return t.cg == 2 ? launch_umma<BITS, GPK, 2, false>(l, t, p, s) : launch_umma<BITS, GPK, 1, false>(l, t, p, s);
}

static uint32_t bf16_twice(int exponent) {   // 2^exponent as a pair of bf16, subnormals included
  const uint32_t b = exponent >= -126 ? (uint32_t)(exponent + 127) << 7 : 1u << (exponent + 133);
  return b << 16 | b;
}

cudaError_t qlinear_umma(const QLinearLaunch& l, cudaStream_t s) {
  const QWeight& w = *l.w;
  if (l.M < 1 || l.M > qlinear_slab_rows(w, l.M)) return cudaErrorInvalidValue;
  if (l.row0 % 16 || l.row0 + l.M > l.x->rows) return cudaErrorInvalidValue;   // rows past the operand's end read as zeros
  const bool glu = l.glu && w.splits == 1 && w.N % QL_TILE_N == 0 && l.act && (l.ld_act & 7) == 0 && (reinterpret_cast<uintptr_t>(l.act) & 15) == 0;
  if (l.glu_done) *l.glu_done = glu ? 1 : 0;
  UmmaPlan t{};
  const int pairs = pairs_of(w), all_teams = std::max(1, w.sm_count / 2);
  if (w.splits > 1) {
    const int turn = plan_in_turn_rows(w, l.M, l.summed);
    t.way = turn ? QL_IN_TURN : QL_APART;
    t.m_pad = turn ? turn : plan_apart_rows(w, l.M);
  } else {
    bool runs = false;
    t.m_pad = plan_whole_rows(w, l.M, l.fix ? QL_FIX_CHUNKS : 0, &runs);
    t.way = runs ? QL_RUNS : QL_IN_TURN;
  }
  const bool sums = t.way == QL_IN_TURN && w.splits > 1;
  // with two chains and several tasks a team, tensor memory has room for the accumulators of 64 rows of a CTA alone
  const int rows = t.m_pad, chunks = (l.M + rows - 1) / rows, alone = ((l.M + chunks - 1) / chunks + 15) & ~15;
  for (t.cg = !sums && chunks <= 2 && alone <= solo_rows(w) ? 1 : 2;; t.cg = 2) {
    t.m_pad = t.cg == 1 ? alone : rows;
    t.chunks = (l.M + t.m_pad - 1) / t.m_pad;
    t.teams = t.way == QL_IN_TURN ? (int)std::min<long long>((long long)pairs * t.chunks, all_teams) : all_teams;
    const bool several = t.way == QL_RUNS || (t.way == QL_IN_TURN && (sums || (long long)pairs * t.chunks > t.teams));
    if (plan_rings(&t, w, several, sums)) break;
    if (t.cg == 2) return cudaErrorInvalidValue;
  }
  QlKernelParams p;
  p.records = w.records; p.record_bytes = w.record_bytes;
  p.N = w.N; p.kblocks = w.kblocks; p.n_pairs = pairs; p.splits = w.splits; p.chains = w.chains; p.teams = t.teams;
  p.M = l.M; p.m_pad = t.m_pad; p.chunks = t.chunks; p.row0 = l.row0;
  p.way = t.way;
  p.a_slots = t.a_slots; p.b_slots = t.b_slots; p.r_slots = t.r_slots; p.accs = t.accs; p.tmem_cols = t.tmem_cols;
  const int up = 133 - w.shift, first = std::min(127, up);
  p.factors = QlFactors{bf16_twice(first), bf16_twice(up - first), bf16_twice(-w.shift)};
  p.back0 = ldexpf(1.f, std::min(w.shift, 127)); p.back1 = ldexpf(1.f, w.shift - std::min(w.shift, 127));
  p.glu = glu ? l.glu : 0; p.act = l.act; p.ld_act = l.ld_act;
  p.y = l.y; p.ldy = l.ldy; p.partial = l.partial;
  p.vec = glu ? 1 : t.way == QL_APART && w.splits > 1 ? (w.N & 3) == 0 && (reinterpret_cast<uintptr_t>(l.partial) & 15) == 0
                                            : (w.N & 7) == 0 && (l.ldy & 7) == 0 && (reinterpret_cast<uintptr_t>(l.y) & 15) == 0;
  p.fix = reinterpret_cast<uint4*>(l.fix); p.status = l.status;
  if (w.bits == 4) return w.gpk == 2 ? launch_umma_cg<4, 2>(l, t, p, s) : launch_umma_cg<4, 1>(l, t, p, s);
  return w.gpk == 2 ? launch_umma_cg<8, 2>(l, t, p, s) : launch_umma_cg<8, 1>(l, t, p, s);
}

}  // namespace kc
