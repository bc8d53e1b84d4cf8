// Paged attention of few query rows a unit (at most KEY_ROWS): decode and verify steps. See kc_attn.cu for the path, the
// chunks and the roles; this kernel gives a row the same bits.
//
// A thread of the softmax warps holds a KEY, not a row: S^T = K Q^T and O^T += V^T P, keys and features on the 128 lanes
// of tensor memory, the rows as columns. With a row per thread a unit of 4 to 40 rows kept one or two of the four softmax
// warps busy, 2900 cycles a tile of 128 keys and more under a soft cap, which was the bound of every decode step; here a
// tile's rows x keys lie evenly over the warps. What crosses them is each row's maximum (exact in any order) and its sum
// (over the 32 keys of a warp pairwise, keys 16, 8, 4, 2 and 1 apart, then the warps pairwise: kc_attn.cu adds in the same
// tree). A product has the unit's columns only: the rows are not padded to 128 either.
//
// K and V are separate slots of the ring: scores are taken from half a tile's bytes, and a slot of K is free again one
// product earlier.
//
// What bounds it: over long contexts and up to 32 rows HBM, 5.6 TB/s of the 6.5 that a copy makes (18 sequences of 8191 keys).
// Over 32 sequences of 512 to 2048 keys HBM is at 0.6 of that: 41 to 43 us where the copy's rate would take 26. Of the
// difference 4 us are the start until the first tile is there (3 lie under the kernel ahead in a step), the rest is 256
// units of 4 to 16 tiles that fall on 148 SMs unevenly and begin and end one after the other. At 40 rows and more the softmax
// warps bound it, whose time is instruction fetch and latencies as much as issue: four sets of warps with eight rows each in
// a loop take a third less than one set with all of them unrolled. A call on its own, L2 flushed, attn_kernel -> this: 32
// sequences of 512 to 2048 keys 48.8 -> 41.3 us at 4 rows of a unit, 49.2 -> 43.4 at 24; 64 of 1024 to 4096 and 40 rows 149.6 ->
// 143.7 (102.9 at the copy's rate); 16 of 6144 under a soft cap, head size 256, 212 + 36 for the combine kernel -> 150 (123),
// with a window of 4096 202 + 14 -> 107 (82); one of 1001 13.0 -> 10.9; 48 of 40 18.6 -> 10.5. In a decode step of 32
// sequences a layer's attention adds 48.2 -> 31.1 us. Where it is the slower one: attn_key_rows.
#include "kc_attn_dev.cuh"

#include <algorithm>

namespace kc {

namespace {

constexpr int KEY_SETS = 4;                                 // of four softmax warps
constexpr int KEY_THREADS = (8 + 4 * KEY_SETS) * 32;

// NR: columns of a product, the most rows of a unit.
template <int D, int NR>
struct KeyShape {
  static constexpr int TK = D == 256 ? 64 : 128;      // keys per tile
  static constexpr int SLABS = D / 64;
  static constexpr int GROUP_BYTES = SLABS * 1024;    // 8 keys of K or of V: slabs of [8][128 B]
  static constexpr int SLOT_BYTES = TK / 8 * GROUP_BYTES;
  static constexpr int Q_BYTES = SLABS * NR * 128;
  // Probabilities: a line of 128 bytes a key. Up to 32 rows both parts share it (rows 0 .. 31 of the upper, then of the
  // lower part); more rows have an area for each part.
  static constexpr bool WIDE = NR > 32;
  static constexpr int P_BYTES = TK * 128 * (WIDE ? 2 : 1), P_BUFS = WIDE ? 1 : 2;
  static constexpr int RING = (216 * 1024 - Q_BYTES - P_BUFS * P_BYTES) / SLOT_BYTES;
  static constexpr int HALVES = D == 256 ? 2 : 1;     // products of 128 features
  static constexpr int TMEM_O = 2 * NR, TMEM_ACC = TMEM_O + 2 * HALVES * NR;   // columns: S0, S1, two buffers of O, merged chunks
  static constexpr int TMEM_COLS = TMEM_ACC + HALVES * NR <= 256 ? 256 : 512;
  // maxima and sums [2][KEY_SETS][4][16] each, references [KEY_SETS][4][16], stat [2][NR], barriers
  static constexpr int SMALL_BYTES = 5 * KEY_SETS * 4 * 16 * 4 + 2 * NR * 8 + (2 * RING + 24) * 8;
  // A product of K takes 128 keys from the start of a slot, one of V 128 features: at other tile and head sizes the lanes
  // past them are not read, but what they multiply has to lie inside the allocation.
  static constexpr int USED = RING * SLOT_BYTES + Q_BYTES + P_BUFS * P_BYTES + SMALL_BYTES;
  static constexpr int REACH = (RING - 1) * SLOT_BYTES + 128 / 8 * GROUP_BYTES + 1024;
  static constexpr int SMEM = USED > REACH ? USED : REACH;
  static_assert(RING >= 4 && SMEM <= 227 * 1024, "shared memory of one CTA");
};

// Not a NaN where another lane has a number.
__device__ __forceinline__ float redux_max(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}

// The sums over a warp's lanes of eight values, pairwise over lanes 16, 8, 4, 2 and 1 apart: lane L gets that of value L / 4.
// Both lanes of a pair add the same two numbers.
__device__ __forceinline__ float tree_sum8(const float (&v)[8], int lane) {
  float a[4], b[2];
  const bool u16 = lane & 16, u8 = lane & 8, u4 = lane & 4;
#pragma unroll
  for (int i = 0; i < 4; ++i) a[i] = (u16 ? v[i + 4] : v[i]) + __shfl_xor_sync(0xffffffffu, u16 ? v[i] : v[i + 4], 16);
#pragma unroll
  for (int i = 0; i < 2; ++i) b[i] = (u8 ? a[i + 2] : a[i]) + __shfl_xor_sync(0xffffffffu, u8 ? a[i] : a[i + 2], 8);
  float c = (u4 ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, u4 ? b[0] : b[1], 4);
  c += __shfl_xor_sync(0xffffffffu, c, 2);
  return c + __shfl_xor_sync(0xffffffffu, c, 1);
}

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]),
               "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
// The four softmax warps of a set meet. Also a warp that has given up comes here, tile by tile: the barrier has no time limit.
__device__ __forceinline__ void cross_warps(int set) { asm volatile("bar.sync %0, 128;" ::"r"(1 + set) : "memory"); }

// How scores become the exponents' arguments: with the scale in the multiplier (scale_folds), the same behind a soft cap, or
// scaled and capped where they lie. Instantiations of their own: a branch around the code for another way, in every tile,
// costs a fetch of instructions behind it.
enum { PLAIN, CAPPED, SCALED };

template <int D, int NR, int MODE>
__global__ void __launch_bounds__(KEY_THREADS, 1)
attn_keys_kernel(const __grid_constant__ CUtensorMap kvmap, const __grid_constant__ CUtensorMap qmap,
                 const __grid_constant__ CUtensorMap qmap_small, const AttnParams p) {
  using S = KeyShape<D, NR>;
  constexpr int TK = S::TK, H = S::HALVES;
  extern __shared__ __align__(1024) uint8_t ring[];   // no static shared memory: the dynamic part starts on its boundary
  uint8_t* sQ = ring + S::RING * S::SLOT_BYTES;
  uint8_t* sP = sQ + S::Q_BYTES;
  float* smax = reinterpret_cast<float*>(sP + S::P_BUFS * S::P_BYTES);   // [2][set][4][16] maxima of a tile by warp
  float* ssum = smax + 2 * KEY_SETS * 4 * 16;                    // [2][set][4][16] sums
  float* sref = ssum + 2 * KEY_SETS * 4 * 16;                    // [set][4][16] references of the exponents, negated
  float2* stat = reinterpret_cast<float2*>(sref + KEY_SETS * 4 * 16);   // [2][NR] (m, l) of a finished chunk
  uint64_t* bars = reinterpret_cast<uint64_t*>(stat + 2 * NR);
  uint64_t* kv_full = bars;
  uint64_t* kv_empty = kv_full + S::RING;
  uint64_t* q_full = kv_empty + S::RING;
  uint64_t* q_empty = q_full + 1;
  uint64_t* s_ready = q_empty + 1;      // [2] scores of a tile are in S[tile & 1]
  uint64_t* p_ready = s_ready + 2;      // [2] its probabilities are in P[tile & (P_BUFS - 1)]
  uint64_t* pv_done = p_ready + 2;      // [2] they have been multiplied
  uint64_t* stat_full = pv_done + 2;    // [2] (m, l) of a chunk; with the last PV of the chunk its O is complete
  uint64_t* o_full = stat_full + 2;
  uint64_t* o_empty = o_full + 2;       // [2] O and (m, l) have been read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_empty + 2);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  pdl_launch_dependents();
  // Rows of Q that no load writes are columns that no row reads; as zeros they don't take the soft cap's longer way.
  for (int i = threadIdx.x; i < S::Q_BYTES / 16; i += KEY_THREADS) reinterpret_cast<uint4*>(sQ)[i] = make_uint4(0, 0, 0, 0);
  fence_proxy_async_smem();
  if (threadIdx.x == 0) {
    for (int i = 0; i < S::RING; ++i) { mbar_init(&kv_full[i], 1); mbar_init(&kv_empty[i], 1); }
    mbar_init(q_full, 1); mbar_init(q_empty, 1);
    for (int i = 0; i < 2; ++i) { mbar_init(&s_ready[i], 1); mbar_init(&p_ready[i], 4 * KEY_SETS); mbar_init(&pv_done[i], 1); mbar_init(&stat_full[i], KEY_SETS); mbar_init(&o_full[i], 1); mbar_init(&o_empty[i], 4); }
    mbar_fence_init();
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "n"(S::TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (warp == 0 && lane == 0) { tma_prefetch_desc(&kvmap); tma_prefetch_desc(&qmap); tma_prefetch_desc(&qmap_small); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  // Before pdl_wait only the producer reads memory: units and block tables, and K and V of keys below AttnUnit::old. All of
  // it was written ahead of the step's first kernel, which starts when all that is complete (see pdl_wait), and
  // nothing in the step writes it: old_keys ends a sequence's old keys at the first block that the step writes, but the one
  // in which its new tokens begin, and a tile is loaded early only where all of it lies below. Q is loaded after the wait.
  // The other roles are past it before their first bounded wait: see attn_kernel.

  const int total = p.n_units * p.Hkv;
  if (warp == 0) {
    // ---- TMA producer: a tile's K, its V, the next tile's K, ..; lane i issues the 16 keys of index i ----
    RingPos kv;
    uint32_t qphase = 0;
    bool ok = true, waited = false;
    for (int r = 0, w; ok && r * (int)gridDim.x < total; ++r) {
      if ((w = unit_index(r, blockIdx.x, gridDim.x, total)) < 0) break;
      UnitTiles u;
      const int kvh = w % p.Hkv;
      u.open(p, w / p.Hkv, TK);
      if (!u.live()) continue;
      const int32_t* tbl = p.block_tables + (size_t)u.seq * p.max_blocks;
      const int bs_log2 = 31 - __clz(p.BS);
      auto entries = [&]() {   // of the chunk, one a lane. block_size is a power of two >= 16: chunks start on block edges
        return lane < (u.keys + p.BS - 1) >> bs_log2 ? tbl[u.c * (ATT_CHUNK >> bs_log2) + lane] : 0;
      };
      int my_blk = entries(), loaded_c = u.c;
      bool queries = true;     // still to be loaded: a later unit's behind its first tile, which the last unit's scores don't hold up
      auto load_queries = [&]() {
        queries = false;
        ok = warp_wait(q_empty, qphase ^ 1, p.status, KC_DEV_ATTN | 0x21);
        if (!ok) return;
        qphase ^= 1;
        if (lane == 0) {
          const int tokens = u.small ? ATT_SMALL_TOKENS : p.q_tokens;
          mbar_arrive_expect_tx(q_full, S::SLABS * tokens * p.gqa * 128);
          for (int s = 0; s < S::SLABS; ++s)
            tma_load_5d(sQ + s * NR * 128, u.small ? &qmap_small : &qmap, 0, 0, s, kvh, u.tok0, q_full);
        }
        __syncwarp();
      };
      for (int tiles = 0; u.live() && ok; u.next(TK), ++tiles) {
        // Keys that no kernel of this step writes are there before the step's first kernel starts: the ring is filled with
        // them under the tail of the kernel ahead.
        if (!waited && (tiles == S::RING / 2 || u.key0(TK) + TK > u.old)) { pdl_wait(); waited = true; load_queries(); }
        else if (waited && tiles == 1 && queries) load_queries();
        if (!ok) break;
        if (u.c != loaded_c) { loaded_c = u.c; my_blk = entries(); }
        const int nb = u.blocks(TK);
        const int koff = u.t * TK + lane * 16;
        const int blk = __shfl_sync(0xffffffffu, my_blk, (koff >> bs_log2) & 31);
        const int row = (blk * p.Hkv + kvh) * p.BS + (koff & (p.BS - 1));   // of a plane
#pragma unroll 1
        for (int pl = 0; pl < 2; ++pl) {
          ok = ok && warp_wait(&kv_empty[kv.stage], kv.phase ^ 1, p.status, KC_DEV_ATTN | 0x22);
          if (!ok) break;
          if (lane == 0) mbar_arrive_expect_tx(&kv_full[kv.stage], nb * 2 * S::GROUP_BYTES);
          __syncwarp();   // the byte count is announced
          if (lane < nb) {
            uint8_t* to = ring + (size_t)kv.stage * S::SLOT_BYTES + lane * 2 * S::GROUP_BYTES;
            if (p.kv5d) {
              tma_load_5d(to, &kvmap, 0, 0, 0, p.layer * 2 + pl, row >> 3, &kv_full[kv.stage]);
            } else {
              for (int g = 0; g < 2; ++g)
                for (int s = 0; s < S::SLABS; ++s)
                  tma_load_2d(to + g * S::GROUP_BYTES + s * 1024, &kvmap, s * 64,
                              (int)((long long)(p.layer * 2 + pl) * p.NB * p.Hkv * p.BS) + row + g * 8, &kv_full[kv.stage]);
            }
          }
          __syncwarp();
          kv.advance(S::RING);
        }
      }
      if (!waited) { pdl_wait(); waited = true; }
      if (ok && queries) load_queries();
    }
  } else if (warp == 1) {
    // ---- MMA issuer: converged, one elected lane around the MMAs ----
    pdl_wait();
    const uint64_t kd = umma_smem_desc(smem_u32(ring), S::GROUP_BYTES);           // K-major
    const uint64_t vd = umma_smem_desc(smem_u32(ring), S::GROUP_BYTES, 1024);     // MN-major
    const uint64_t qd = umma_smem_desc(smem_u32(sQ), 1024);                       // K-major
    const uint64_t pd = umma_smem_desc(smem_u32(sP), 1024);                       // MN-major, one slab
    const uint32_t k_hi = (uint32_t)(kd >> 32), v_hi = (uint32_t)(vd >> 32), q_hi = (uint32_t)(qd >> 32), p_hi = (uint32_t)(pd >> 32);
    const uint32_t idesc_qk = umma_idesc_bf16(128, NR), idesc_pv = umma_idesc_bf16(128, NR, true, true);
    constexpr uint32_t SLOT = S::SLOT_BYTES >> 4, P_LOW = (S::WIDE ? TK * 128 : 64) >> 4;
    RingPos kv;                   // the slot of the next tile's K
    int tile = 0;                 // tiles issued by this CTA so far (S buffer = tile & 1)
    int chunks = 0;               // chunks begun (O buffer = chunk & 1)
    uint32_t qphase = 0;
    bool ok = true;
    // the tile whose PV is still to be issued
    bool pend = false, pend_first = false, pend_last = false;
    int pend_nb = 0, pend_tile = 0, pend_chunk = 0;
    RingPos pend_v;
    auto issue_pv = [&]() {
      const int ob = pend_chunk & 1;
      if (pend_first) ok = ok && warp_wait(&o_empty[ob], ((pend_chunk >> 1) & 1) ^ 1, p.status, KC_DEV_ATTN | 0x23);
      ok = ok && warp_wait(&kv_full[pend_v.stage], pend_v.phase, p.status, KC_DEV_ATTN | 0x24) &&
           warp_wait(&p_ready[pend_tile & 1], (pend_tile >> 1) & 1, p.status, KC_DEV_ATTN | 0x25);
      if (!ok) return;
      tc_fence_after();
      const uint32_t v_lo = (uint32_t)vd + pend_v.stage * SLOT, p_lo = (uint32_t)pd + (pend_tile & (S::P_BUFS - 1)) * (S::P_BYTES >> 4);
      const uint32_t o = tmem + S::TMEM_O + ob * H * NR;
      if (elect_one()) {
        for (int b = 0; b < pend_nb; ++b) {
          const uint32_t vb = v_lo + b * (2 * S::GROUP_BYTES >> 4), pb = p_lo + b * (16 * 128 >> 4);
          const uint32_t acc = pend_first && b == 0 ? 0u : 1u;
#pragma unroll
          for (int h = 0; h < H; ++h) {
            umma_bf16_ss(o + h * NR, vb + h * (2 * 1024 >> 4), v_hi, pb, p_hi, idesc_pv, acc);
            umma_bf16_ss(o + h * NR, vb + h * (2 * 1024 >> 4), v_hi, pb + P_LOW, p_hi, idesc_pv, 1u);
          }
        }
        umma_commit(&pv_done[pend_tile & 1]);
        umma_commit(&kv_empty[pend_v.stage]);
        if (pend_last) umma_commit(&o_full[ob]);
      }
      __syncwarp();
      pend = false;
    };
    for (int r = 0, w; ok && r * (int)gridDim.x < total; ++r) {
      if ((w = unit_index(r, blockIdx.x, gridDim.x, total)) < 0) break;
      UnitTiles u;
      u.open(p, w / p.Hkv, TK);
      if (!u.live()) continue;
      bool first_of_unit = true;
      for (; u.live() && ok;) {
        // Whichever product has its operands first: see attn_kernel. The looks are limited, what is missing after them is
        // waited for in the bounded waits below.
        if (pend) {
          for (int looks = 0; looks < 256; ++looks) {
            const bool scores = mbar_test_wait(&kv_full[kv.stage], kv.phase) && (!first_of_unit || mbar_test_wait(q_full, qphase));
            if (__all_sync(0xffffffffu, scores)) break;
            if (looks == 255 || __all_sync(0xffffffffu, mbar_test_wait(&p_ready[pend_tile & 1], (pend_tile >> 1) & 1) && mbar_test_wait(&kv_full[pend_v.stage], pend_v.phase))) { issue_pv(); break; }
          }
          if (!ok) break;
        }
        if (first_of_unit) {
          ok = warp_wait(q_full, qphase, p.status, KC_DEV_ATTN | 0x26);
          if (!ok) break;
          qphase ^= 1;
        }
        ok = warp_wait(&kv_full[kv.stage], kv.phase, p.status, KC_DEV_ATTN | 0x27);
        if (!ok) break;
        first_of_unit = false;
        tc_fence_after();
        const int nb = u.blocks(TK), sb = tile & 1, stage = kv.stage, chunk = chunks;
        const bool first = u.t == u.first_tile(TK), last = u.last();
        if (last) ++chunks;
        u.next(TK);
        const bool unit_done = !u.live();
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks)
            umma_bf16_ss(tmem + sb * NR, (uint32_t)kd + stage * SLOT + (ks >> 2) * (1024 >> 4) + (ks & 3) * 2, k_hi,
                         (uint32_t)qd + (ks >> 2) * (NR * 128 >> 4) + (ks & 3) * 2, q_hi, idesc_qk, ks == 0 ? 0u : 1u);
          umma_commit(&s_ready[sb]);
          umma_commit(&kv_empty[stage]);
          if (unit_done) umma_commit(q_empty);
        }
        __syncwarp();
        kv.advance(S::RING);
        if (pend) issue_pv();
        pend = true; pend_first = first; pend_last = last; pend_nb = nb; pend_tile = tile; pend_chunk = chunk; pend_v = kv;
        kv.advance(S::RING);
        ++tile;
      }
    }
    if (ok && pend) issue_pv();
  } else if (warp >= 4 && (warp < 8 || warp >= 12)) {
    // ---- softmax: sets of four warps, set i with the groups of eight rows i, i + KEY_SETS. Thread = key 32 * (warp & 3) + lane
    // of the tile against those rows, or one of the rows (the first sixteen lanes) where maxima and sums meet ----
    pdl_wait();
    const int quarter = warp & 3, set = warp < 8 ? 0 : (warp >> 2) - 2;
    const bool has_keys = quarter * 32 < TK, has_features = quarter * 32 < D;   // of tensor memory's lanes, S and O
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const float mul = (MODE == CAPPED ? p.softcap : MODE == PLAIN ? p.scale : 1.f) * 1.4426950408889634f;
    const float cap_arg = MODE == CAPPED ? p.scale / p.softcap : 0.f;
    uint8_t* p_line = sP + (quarter * 32 + lane) * 128;
    float* my_ref = sref + (set * 4 + quarter) * 16;
    float *max0 = smax + set * 4 * 16, *sum0 = ssum + set * 4 * 16;   // of an even tile
    constexpr int ODD = KEY_SETS * 4 * 16;
    const int row = (set + KEY_SETS * (lane >> 3)) * 8 + (lane & 7), slot = lane & 15;
    int tile = 0, chunks = 0;
    bool ok = true;   // once false: no more waits, but the crossings
    for (int r0 = 0, w; r0 * (int)gridDim.x < total; ++r0) {
      if ((w = unit_index(r0, blockIdx.x, gridDim.x, total)) < 0) break;
      UnitTiles u;
      u.open(p, w / p.Hkv, TK);
      if (!u.live()) continue;
      const int groups = (u.rows + 7) >> 3;
      const bool row_live = row < u.rows && lane < 16;
      const int pos = u.pos0 + min(row / p.gqa, u.ntok - 1);
      float m = -INFINITY, l = 0.f, alpha = 1.f;
      // the sums of a tile, once every warp's are there
      auto add_sums = [&](int t) {
        const float* s = sum0 + (t & 1) * ODD + slot;
        const float lo = s[0] + s[16];
        l = __fmaf_rn(l, alpha, TK == 64 ? lo : lo + (s[32] + s[48]));
      };
      for (; u.live(); u.next(TK), ++tile) {
        const int sb = tile & 1, nb = u.blocks(TK), key0 = u.key0(TK), key = key0 + quarter * 32 + lane;
        const bool first = u.t == u.first_tile(TK), last = u.last();
        // every key of the tile is visible to every row of the unit: the same arithmetic without the predicates
        const bool edge = !(nb * 16 == TK && key0 + TK - 1 <= u.pos0 && (p.window == 0 || key0 > u.pos_max - p.window));
        // rows that see this thread's key: r_lo <= r < r_hi
        const int r_lo = max(key - u.pos0, 0) * p.gqa;
        const int r_hi = p.window > 0 ? (int)max(min((long long)key - u.pos0 + p.window, 1ll << 16), 0ll) * p.gqa : 1 << 30;
        const uint32_t s_addr = tmem + lane_addr + sb * NR;
        ok = ok && warp_wait(&s_ready[sb], (tile >> 1) & 1, p.status, KC_DEV_ATTN | 0x29);
        uint32_t x[8];   // scores of a group on their way
        auto scores = [&](float (&v)[8]) {   // .. are here
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            asm volatile("" : "+r"(x[j]));   // no use before the wait
            v[j] = __uint_as_float(x[j]);
            if (MODE == SCALED) {
              v[j] *= p.scale;
              if (p.softcap > 0.f) v[j] = p.softcap * tanhf(v[j] / p.softcap);
            }
          }
        };
        auto mask = [&](float (&v)[8], int g) {
          if (edge) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (g * 8 + j < r_lo || g * 8 + j >= r_hi) v[j] = -INFINITY;
          }
        };
        // ---- maxima: a row's, over the warp's keys ----
        const bool works = ok && has_keys && set < groups;
        if (works) {
          tc_fence_after();
          tmem_ld8_issue(s_addr + set * 8, x);
          float4* to = reinterpret_cast<float4*>(max0 + (tile & 1) * ODD + quarter * 16);
#pragma unroll 1
          for (int g = set; g < groups; g += KEY_SETS, to += 2) {
            float v[8];
            scores(v);
            tmem_ld8_issue(s_addr + (g + KEY_SETS < groups ? g + KEY_SETS : set) * 8, x);   // the next ones, or the first again
            mask(v, g);
            const float4 a = make_float4(redux_max(v[0]), redux_max(v[1]), redux_max(v[2]), redux_max(v[3]));
            const float4 b = make_float4(redux_max(v[4]), redux_max(v[5]), redux_max(v[6]), redux_max(v[7]));
            if (lane == 0) { to[0] = a; to[1] = b; }
          }
        }
        cross_warps(set);
        if (first) { m = -INFINITY; l = 0.f; }
        else add_sums(tile - 1);
        // ---- a row's maximum over the tile, its reference and what that rescales: every warp for itself ----
        const float* s = max0 + (tile & 1) * ODD + slot;
        float tmax = fmaxf(s[0], s[16]);
        if (TK > 64) tmax = fmaxf(tmax, fmaxf(s[32], s[48]));
        tmax = fmaxf(tmax, -INFINITY);
        if (MODE == CAPPED) {
          const int hi = pos - key0, lo = p.window > 0 ? pos - p.window - key0 + 1 : -key0;
          const bool seen = !edge || (hi >= 0 && lo < TK && lo <= hi);   // any key: a score of -inf is a key of weight e^-cap
          if (seen) { tmax *= cap_arg; tmax = tanh_any(tmax, tanh_near(make_float2(tmax, tmax)).x); }   // grows with the score
        }
        tmax *= mul;
        alpha = 1.f;
        if (tmax > m + 8.f) { alpha = ex2(m - tmax); m = tmax; }   // the reference lags: see attn_kernel
        if (lane < 16) my_ref[lane] = m == -INFINITY ? -0.f : -m;
        const bool rescale = __any_sync(0xffffffffu, row_live && alpha != 1.f) && !first;
        __syncwarp();   // the references are there
        // ---- the products are in: of the tile whose probabilities are replaced, and of the last one where O is rescaled ----
        if (S::P_BUFS == 1 && tile > 0) ok = ok && warp_wait(&pv_done[sb ^ 1], ((tile - 1) >> 1) & 1, p.status, KC_DEV_ATTN | 0x2a);
        if (S::P_BUFS == 2 && tile > 1) ok = ok && warp_wait(&pv_done[sb], ((tile >> 1) & 1) ^ 1, p.status, KC_DEV_ATTN | 0x2a);
        if (ok && rescale && has_features) {
          ok = warp_wait(&pv_done[sb ^ 1], ((tile - 1) >> 1) & 1, p.status, KC_DEV_ATTN | 0x2c);
          tc_fence_after();
          if (works) tmem_wait_ld();   // keeps x apart from what follows
          const uint32_t o_addr = tmem + lane_addr + S::TMEM_O + (chunks & 1) * H * NR;
#pragma unroll 1
          for (int g = set; ok && g < groups; g += KEY_SETS) {
#pragma unroll
            for (int h = 0; h < H; ++h) {
              uint32_t o[8];
              tmem_ld8_issue(o_addr + h * NR + g * 8, o);
              tmem_wait_ld();
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                asm volatile("" : "+r"(o[j]));   // no use before the wait
                o[j] = __float_as_uint(__uint_as_float(o[j]) * __shfl_sync(0xffffffffu, alpha, g / KEY_SETS * 8 + j));
              }
              tmem_st8(o_addr + h * NR + g * 8, o);
            }
          }
          tmem_wait_st();
        }
        // ---- probabilities and their sums over the warp's keys ----
        if (works && ok) {
          uint8_t* line = p_line + (tile & (S::P_BUFS - 1)) * S::P_BYTES;
          const float4* refs = reinterpret_cast<const float4*>(my_ref);
          float* sums = sum0 + (tile & 1) * ODD + quarter * 16 + (lane >> 2);
#pragma unroll 1
          for (int g = set; g < groups; g += KEY_SETS, refs += 2, sums += 8) {
            float v[8];
            scores(v);
            if (g + KEY_SETS < groups) tmem_ld8_issue(s_addr + (g + KEY_SETS) * 8, x);
            if (MODE == CAPPED) {
              float b0 = 0.f, b1 = 0.f;
#pragma unroll
              for (int j = 0; j < 8; j += 2) { b0 = fmaxf(b0, fabsf(v[j])); b1 = fmaxf(b1, fabsf(v[j + 1])); }
              // no score past 0.75 caps: the polynomial alone (an element's value is the same on both sides). Keys past the
              // sequence have no say.
              const bool all_near = __all_sync(0xffffffffu, fmaxf(b0, b1) * cap_arg < TANH_NEAR || key > u.pos_max);
              const float2 arg = make_float2(cap_arg, cap_arg);
              if (all_near) {
#pragma unroll
                for (int j = 0; j < 8; j += 2) {
                  const float2 t = tanh_near(mul2(make_float2(v[j], v[j + 1]), arg));
                  v[j] = t.x; v[j + 1] = t.y;
                }
              } else {
#pragma unroll
                for (int j = 0; j < 8; j += 2) {
                  const float2 y = mul2(make_float2(v[j], v[j + 1]), arg), t = tanh_near(y);
                  v[j] = tanh_any(y.x, t.x); v[j + 1] = tanh_any(y.y, t.y);
                }
              }
            }
            mask(v, g);
            const float4 ra = refs[0], rb = refs[1];
            const float ref[8] = {ra.x, ra.y, ra.z, ra.w, rb.x, rb.y, rb.z, rb.w};
            uint32_t ph[4], pl[4];
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
              const float2 e = fma2(make_float2(v[j], v[j + 1]), make_float2(mul, mul), make_float2(ref[j], ref[j + 1]));
              v[j] = ex2(e.x); v[j + 1] = ex2(e.y);
            }
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
              const uint32_t a = __float_as_uint(v[j]) & 0xffff0000u, b = __float_as_uint(v[j + 1]) & 0xffff0000u;
              ph[j / 2] = __byte_perm(a, b, 0x7632);
              const float2 rest = fma2(make_float2(__uint_as_float(a), __uint_as_float(b)), make_float2(-1.f, -1.f), make_float2(v[j], v[j + 1]));
              pl[j / 2] = pack_bf162(rest.x, rest.y);
            }
            // 16-byte pieces of a line are exchanged by the line's index, as the 128-byte swizzle wants them
            *reinterpret_cast<uint4*>(line + ((g ^ (lane & 7)) << 4)) = make_uint4(ph[0], ph[1], ph[2], ph[3]);
            *reinterpret_cast<uint4*>(line + (S::WIDE ? TK * 128 + ((g ^ (lane & 7)) << 4) : ((g + 4) ^ (lane & 7)) << 4)) = make_uint4(pl[0], pl[1], pl[2], pl[3]);
            const float sum = tree_sum8(v, lane);
            if ((lane & 3) == 0) *sums = sum;
          }
          fence_proxy_async_smem();
        }
        tc_fence_before();
        __syncwarp();
        if (ok && lane == 0) mbar_arrive(&p_ready[sb]);
        if (last) {
          cross_warps(set);
          add_sums(tile);
          if (quarter == 0) {
            const int cb = chunks & 1;
            ok = ok && warp_wait(&o_empty[cb], ((chunks >> 1) & 1) ^ 1, p.status, KC_DEV_ATTN | 0x2b);   // (m, l) of the chunk two before has been read
            if (ok) {
              if (row_live) stat[cb * NR + row] = make_float2(m, l);
              __syncwarp();
              if (lane == 0) mbar_arrive(&stat_full[cb]);
            }
          }
          ++chunks;
        }
      }
    }
  } else if (warp >= 8) {
    // ---- a finished chunk: thread = feature 32 * (warp & 3) + lane, and that 128 further on. What a unit of whole rows has
    // merged so far stays in tensor memory, so that groups of eight rows are turns of a loop: with the rows in registers, and
    // the code of each of 64, the end of a unit took 7 us, most of them fetching it. ----
    pdl_wait();   // the stores below may overwrite what an earlier kernel still reads
    const int quarter = warp & 3, feature = quarter * 32 + lane;
    const bool has_features = quarter * 32 < D;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16, acc_addr = tmem + lane_addr + S::TMEM_ACC;
    constexpr int RL = NR / 32;   // rows of a lane where a lane stands for rows
    int chunks = 0;
    bool ok = true;
    for (int r0 = 0, w; ok && r0 * (int)gridDim.x < total; ++r0) {
      if ((w = unit_index(r0, blockIdx.x, gridDim.x, total)) < 0) break;
      UnitTiles u;
      const int kvh = w % p.Hkv;
      u.open(p, w / p.Hkv, TK);
      if (!u.live()) continue;
      // rows are (token, head of the group); row + 1 is the next row of the output but at the end of a group
      const size_t row0 = (size_t)u.tok0 * p.Hq + kvh * p.gqa;
      const int groups = (u.rows + 7) >> 3;
      // Rows of a finished unit (DONE: values of the rows divided by their sums l) or of a chunk's partial sums, one after the other.
      auto store = [&](uint32_t from, bool done, const float* l, int chunk) {
        float rs[RL], rest[RL];
#pragma unroll
        for (int i = 0; i < RL; ++i) { const RowSum s = row_sum(l[i]); rs[i] = s.r.x; rest[i] = s.rest.x; }
        size_t row = row0;
        int head = 0;
#pragma unroll 1
        for (int g = 0; g < groups; ++g) {
          uint32_t o[H][8];
#pragma unroll
          for (int h = 0; h < H; ++h) tmem_ld8_issue(from + h * NR + g * 8, o[h]);
          const float rg = RL == 2 && g >= 4 ? rs[RL - 1] : rs[0], eg = RL == 2 && g >= 4 ? rest[RL - 1] : rest[0];
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float r = __shfl_sync(0xffffffffu, rg, (g * 8 + j) & 31), e = __shfl_sync(0xffffffffu, eg, (g * 8 + j) & 31);
            if (g * 8 + j < u.rows) {
#pragma unroll
              for (int h = 0; h < H; ++h) {
                asm volatile("" : "+r"(o[h][j]));   // no use before the wait
                const float v = __uint_as_float(o[h][j]);
                if (done) p.out[row * D + h * 128 + feature] = __float2bfloat16_rn(__fmaf_rn(v, r, __fmaf_rn(v, e, 0.f)));
                else p.part_o[(row * p.max_chunks + chunk) * D + h * 128 + feature] = v;
              }
              ++row;
              if (++head == p.gqa) { head = 0; row += p.Hq - p.gqa; }
            }
          }
        }
      };
      float macc[RL], lacc[RL];
#pragma unroll
      for (int i = 0; i < RL; ++i) { macc[i] = -INFINITY; lacc[i] = 0.f; }
      bool first = true;
      for (; u.c < u.c1 && ok; ++u.c, ++chunks, first = false) {
        const int cb = chunks & 1;
        ok = warp_wait(&stat_full[cb], (chunks >> 1) & 1, p.status, KC_DEV_ATTN | 0x2d) &&
             warp_wait(&o_full[cb], (chunks >> 1) & 1, p.status, KC_DEV_ATTN | 0x2e);
        if (!ok) break;
        float2 ml[RL];
#pragma unroll
        for (int i = 0; i < RL; ++i) ml[i] = stat[cb * NR + lane + 32 * i];
        tc_fence_after();
        const uint32_t o_addr = tmem + lane_addr + S::TMEM_O + cb * H * NR;
        if (p.whole) {
          MergeW mw[RL];
#pragma unroll
          for (int i = 0; i < RL; ++i) {
            mw[i] = merge_weights(macc[i], ml[i].x);
            macc[i] = mw[i].m;
            lacc[i] = merge_value(lacc[i], ml[i].y, mw[i]);
          }
          if (has_features) {
#pragma unroll 1
            for (int i = 0; i < H * groups; ++i) {
              const int h = H == 2 && i >= groups ? 1 : 0, g = i - h * groups;
              uint32_t o[8], acc[8];
              tmem_ld8_issue(o_addr + h * NR + g * 8, o);
              tmem_ld8_issue(acc_addr + h * NR + g * 8, acc);
              const MergeW wg = RL == 2 && g >= 4 ? mw[RL - 1] : mw[0];
              tmem_wait_ld();
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                asm volatile("" : "+r"(o[j]), "+r"(acc[j]));   // no use before the wait
                MergeW t;
                t.a = __shfl_sync(0xffffffffu, wg.a, (g * 8 + j) & 31);
                t.b = __shfl_sync(0xffffffffu, wg.b, (g * 8 + j) & 31);
                acc[j] = __float_as_uint(merge_value(first ? 0.f : __uint_as_float(acc[j]), __uint_as_float(o[j]), t));
              }
              tmem_st8(acc_addr + h * NR + g * 8, acc);
            }
            tmem_wait_st();
          }
        } else {
          if (quarter == 0 && !p.single) {
#pragma unroll
            for (int i = 0; i < RL; ++i) {
              const int row = lane + 32 * i, t = row / p.gqa;
              if (row < u.rows) p.part_ml[(row0 + (size_t)t * p.Hq + (row - t * p.gqa)) * p.max_chunks + u.c] = ml[i];
            }
          }
          float l[RL];
#pragma unroll
          for (int i = 0; i < RL; ++i) l[i] = ml[i].y;
          // a row's only chunk is finished here: see attn_kernel
          if (has_features) store(o_addr, p.single, l, u.c);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&o_empty[cb]);
      }
      if (p.whole && ok && has_features) store(acc_addr, true, lacc, 0);
      __syncwarp();
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(S::TMEM_COLS) : "memory");
  }
}

template <int D, int NR, int MODE>
cudaError_t launch_keys_as(const CUtensorMap& kv, const CUtensorMap& q, const CUtensorMap& q_small, const AttnParams& p, bool in_order,
                           int sm_count, cudaStream_t s) {
  using S = KeyShape<D, NR>;
  static DeviceOnce configured;   // the attribute belongs to the device's copy of the kernel
  if (configured.first_on_current_device()) {
    cudaError_t e = cudaFuncSetAttribute(attn_keys_kernel<D, NR, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM);
    if (e != cudaSuccess) { configured.forget_current_device(); return e; }
  }
  const int grid = std::min(p.n_units * p.Hkv, sm_count);
  return launch_k_opt(!in_order, attn_keys_kernel<D, NR, MODE>, dim3(grid), dim3(KEY_THREADS), S::SMEM, s, kv, q, q_small, p);
}
template <int D, int NR>
cudaError_t launch_keys(const CUtensorMap& kv, const CUtensorMap& q, const CUtensorMap& q_small, const AttnParams& p, bool in_order, bool folded,
                        int sm_count, cudaStream_t s) {
  if (!folded) return launch_keys_as<D, NR, SCALED>(kv, q, q_small, p, in_order, sm_count, s);
  return p.softcap > 0.f ? launch_keys_as<D, NR, CAPPED>(kv, q, q_small, p, in_order, sm_count, s)
                         : launch_keys_as<D, NR, PLAIN>(kv, q, q_small, p, in_order, sm_count, s);
}
template <int D>
cudaError_t launch_keys_d(const CUtensorMap& kv, const CUtensorMap& q, const CUtensorMap& q_small, const AttnParams& p, bool in_order, bool folded,
                          int sm_count, cudaStream_t s) {
  return p.gqa * p.q_tokens <= 32 ? launch_keys<D, 32>(kv, q, q_small, p, in_order, folded, sm_count, s)
                                  : launch_keys<D, 64>(kv, q, q_small, p, in_order, folded, sm_count, s);
}

}  // namespace

cudaError_t attn_keys(const CUtensorMap& kv, const CUtensorMap& q, const CUtensorMap& q_small, const AttnParams& p, bool in_order, bool folded,
                      int head_dim, int sm_count, cudaStream_t s) {
  if (p.gqa * p.q_tokens > KEY_ROWS) return cudaErrorInvalidValue;
  switch (head_dim) {
    case 64: return launch_keys_d<64>(kv, q, q_small, p, in_order, folded, sm_count, s);
    case 128: return launch_keys_d<128>(kv, q, q_small, p, in_order, folded, sm_count, s);
    case 256: return launch_keys_d<256>(kv, q, q_small, p, in_order, folded, sm_count, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace kc
