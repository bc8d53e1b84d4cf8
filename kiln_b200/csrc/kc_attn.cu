// Paged multi-query attention over block tables (sm_100a).
//
// Replaces, for every query length, the reference's gather + fused SDPA
// (crates/kiln-engine/src/paged.rs:191-225; crates/kiln-models/src/nn.rs:800-817)
// and its decode-only Metal kernels (crates/kiln-engine/src/paged_attn.rs:59-303):
// token i of kv-head h is read at pool[tbl[i / BS], h, i % BS, :] (paged_attn.rs:95-99),
// never copied. Scores use the reference's algebra — fp32 scores, fp32 online softmax
// (paged_attn.rs:106-153); the causal predicate is bottom-right aligned: query at absolute
// position p sees keys 0..p. Gemma-2's softcap (nn.rs:527-534) and a sliding window are
// optional.
//
// Both contractions run on tcgen05: S = Q K^T with Q and K in shared memory, O += P V with P in tensor
// memory (written over S) and V in shared memory. One warp-wide lane = one query row (token x head of
// the kv head's group), up to 128 rows of one sequence per unit, so K/V bytes cross HBM once per
// (sequence, kv head, 128 rows).
//
// What a row sees is a function of its own position only, so its bits do not depend on how many other rows share the
// launch: keys are cut into chunks of ATT_CHUNK at absolute positions and a chunk into tiles; a chunk's sums start from
// nothing, and the chunks of a row are merged one after the other in index order (merge_values) — by the kernel itself
// where a unit holds all chunks of its rows, by the combine kernel where the chunks of an item are units of their own.
//
// A probability goes to the tensor core as two bf16 numbers, its upper 16 bits and what they leave: with one, rounded, the
// result was 0.3 to 5 % further from fp64 than with the kernel before this one, whose smaller tiles had more of their
// largest weights at exactly 1; with two the error is that of rounding the output (1.65e-3 of its norm; one: up to 2.2e-3).
// Whether a row is computed alone or among others, its probabilities, their order and so its bits are the same.
//
// Roles (12 warps, one CTA per SM, units taken grid-stride so that K/V tiles of the next unit arrive under the last one):
//   warp 0      TMA: queries of a unit, K/V tiles through a ring
//   warp 1      issues the MMAs: QK of tile i + 1 before PV of tile i
//   warps 4-7   softmax, one row per thread: S -> P, rescaling O when a row's maximum moved
//   warps 8-11  a finished chunk's O: store the partial, or merge it into the row and store the row
//
// Units of few rows go to kc_attn_keys.cu (attn_key_rows): this kernel takes prompts and steps that hold a piece of one.
//
// What bounds it: per 128-key tile of head size 128, HBM takes 2800 cycles of an SM's share, a softmax warp about 2900
// (scores and maximum 590, exponentials and both parts of the probabilities 2000, of which 1024 the special-function
// unit's, next tile 200) and 800 to 1300 in which it waits for scores, the MMAs 1500. 1024 rows after 2048 keys 83 us (397 by
// one mma.sync warp per 16 query rows with a combine launch).
#include "kc_attn.cuh"

#include "kc_attn_dev.cuh"

#include <algorithm>
#include <vector>

namespace kc {

namespace {

constexpr int ATT_THREADS = 12 * 32;
template <int D>
struct AttnShape {
  static constexpr int TK = D == 256 ? 64 : 128;      // keys per tile
  static constexpr int SLABS = D / 64;
  static constexpr int GROUP_BYTES = 2 * SLABS * 1024; // 8 keys: K slabs, then V slabs, [8][128 B] each
  static constexpr int TILE_BYTES = TK / 8 * GROUP_BYTES;
  static constexpr int RING = D == 64 ? 6 : D == 128 ? 3 : 2;
  static constexpr int Q_BYTES = SLABS * ATT_ROWS * 128;
  static constexpr int O_BUFS = D == 256 ? 1 : 2;
  static constexpr int TMEM_O = 256;                   // columns: S0 at 0, S1 at TK, O from 256
  static constexpr int TMEM_COLS = 512;
  static constexpr int SMEM = RING * TILE_BYTES + Q_BYTES + 2 * ATT_ROWS * 8 + 32 * 8;
  static_assert(SMEM <= 227 * 1024, "shared memory of one CTA");
};

// Whether the scale can go into the multiplier of the exponent, behind mask and maximum (FOLDED): right for a positive one
// only (a masked -inf times 0 is NaN, times a negative scale +inf) whose factors stay in the range of fp32. With any other
// scale the scores are scaled and capped where they lie first. That is an instantiation of its own: the code for it in the
// tile loop cost every call 2 to 5 %.
bool scale_folds(float scale, float softcap) {
  if (!(scale > 0.f && scale * 1.4426950408889634f < INFINITY)) return false;
  return !(softcap > 0.f) || (scale / softcap > 0.f && scale / softcap < INFINITY && softcap * 1.4426950408889634f < INFINITY);
}

template <int D, bool WHOLE, bool FOLDED>
__global__ void __launch_bounds__(ATT_THREADS, 1)
attn_kernel(const __grid_constant__ CUtensorMap kvmap, const __grid_constant__ CUtensorMap qmap,
            const __grid_constant__ CUtensorMap qmap_small, const AttnParams p) {
  using S = AttnShape<D>;
  constexpr int TK = S::TK;
  extern __shared__ __align__(1024) uint8_t ring[];   // no static shared memory: the dynamic part starts on its boundary
  uint8_t* sQ = ring + S::RING * S::TILE_BYTES;
  float2* stat = reinterpret_cast<float2*>(sQ + S::Q_BYTES);          // [2][ATT_ROWS] (m, l) of a finished chunk
  uint64_t* bars = reinterpret_cast<uint64_t*>(stat + 2 * ATT_ROWS);
  uint64_t* kv_full = bars;
  uint64_t* kv_empty = kv_full + S::RING;
  uint64_t* q_full = kv_empty + S::RING;
  uint64_t* q_empty = q_full + 1;
  uint64_t* s_ready = q_empty + 1;      // [2] scores of a tile are in S[tile & 1]
  uint64_t* p_ready = s_ready + 2;      // [2] its probabilities are
  uint64_t* pv_done = p_ready + 2;      // [2] they have been multiplied
  uint64_t* stat_full = pv_done + 2;    // [2] (m, l) of a chunk; with the last PV of the chunk its O is complete
  uint64_t* o_full = stat_full + 2;
  uint64_t* o_empty = o_full + 2;       // [2] O and (m, l) have been read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_empty + 2);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int i = 0; i < S::RING; ++i) { mbar_init(&kv_full[i], 1); mbar_init(&kv_empty[i], 1); }
    mbar_init(q_full, 1); mbar_init(q_empty, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_ready[i], 1); mbar_init(&p_ready[i], 4); mbar_init(&pv_done[i], 1);
      mbar_init(&stat_full[i], 4); mbar_init(&o_full[i], 1); mbar_init(&o_empty[i], 4);
    }
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
  // Units and block tables reach the device before a step's first kernel and no kernel writes them, so in a step the
  // producer reads them under the tail of the kernel before this one; where this kernel is the first one behind their copy
  // it is launched in plain stream order (paged_attention). This kernel loads q, K and V after pdl_wait, and every role is past it
  // before its first bounded wait: the time that the kernel before this one takes does not count against the limit.

  const int total = p.n_units * p.Hkv;
  if (warp == 0) {
    // ---- TMA producer. A chunk's block-table entries (at most ATT_CHUNK / 16 = 32) are fetched once, one per lane ----
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
      auto entries = [&]() {   // of the chunk. block_size is a power of two >= 16: chunks start on block edges
        return lane < (u.keys + p.BS - 1) >> bs_log2 ? tbl[u.c * (ATT_CHUNK >> bs_log2) + lane] : 0;
      };
      int my_blk = entries(), loaded_c = u.c;
      if (!waited) { pdl_wait(); waited = true; }
      ok = warp_wait(q_empty, qphase ^ 1, p.status, KC_DEV_ATTN | 1);
      if (!ok) break;
      qphase ^= 1;
      if (lane == 0) {
        const int tokens = u.small ? ATT_SMALL_TOKENS : p.q_tokens;
        mbar_arrive_expect_tx(q_full, S::SLABS * tokens * p.gqa * 128);
        for (int s = 0; s < S::SLABS; ++s)
          tma_load_5d(sQ + s * ATT_ROWS * 128, u.small ? &qmap_small : &qmap, 0, 0, s, kvh, u.tok0, q_full);
      }
      for (; u.live() && ok; u.next(TK)) {
        if (u.c != loaded_c) { loaded_c = u.c; my_blk = entries(); }
        const int nb = u.blocks(TK);
        ok = warp_wait(&kv_empty[kv.stage], kv.phase ^ 1, p.status, KC_DEV_ATTN | 2);
        if (!ok) break;
        if (lane == 0) mbar_arrive_expect_tx(&kv_full[kv.stage], nb * 2 * S::GROUP_BYTES);
        uint8_t* dst = ring + (size_t)kv.stage * S::TILE_BYTES;
        __syncwarp();   // the byte count is announced
        // A lane issues the 16-key block of its index. One lane issuing them in turn, with a division by the block size
        // each, took 340 cycles a block, 2800 of a tile's 3600: the bound of every step, whatever its rows.
        const int koff = u.t * TK + lane * 16;
        const int blk = __shfl_sync(0xffffffffu, my_blk, (koff >> bs_log2) & 31);
        const int row = (blk * p.Hkv + kvh) * p.BS + (koff & (p.BS - 1));   // of a plane
        if (lane < nb) {
          uint8_t* to = dst + lane * 2 * S::GROUP_BYTES;
          if (p.kv5d) {
            tma_load_5d(to, &kvmap, 0, 0, 0, p.layer * 2, row >> 3, &kv_full[kv.stage]);
          } else {
            for (int g = 0; g < 2; ++g)
              for (int pl = 0; pl < 2; ++pl)
                for (int s = 0; s < S::SLABS; ++s)
                  tma_load_2d(to + g * S::GROUP_BYTES + (pl * S::SLABS + s) * 1024, &kvmap, s * 64,
                              (int)((long long)(p.layer * 2 + pl) * p.NB * p.Hkv * p.BS) + row + g * 8, &kv_full[kv.stage]);
          }
        }
        __syncwarp();
        kv.advance(S::RING);
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer: converged, one elected lane around the MMAs ----
    pdl_wait();
    const uint64_t qd = umma_smem_desc(smem_u32(sQ), 1024);
    const uint64_t kd = umma_smem_desc(smem_u32(ring), S::GROUP_BYTES);
    const uint64_t vd = umma_smem_desc(smem_u32(ring) + S::SLABS * 1024, S::GROUP_BYTES, 1024);
    const uint32_t q_hi = (uint32_t)(qd >> 32), k_hi = (uint32_t)(kd >> 32), v_hi = (uint32_t)(vd >> 32);
    const uint32_t idesc_pv = umma_idesc_bf16(ATT_ROWS, D, true);
    RingPos kv;
    int tile = 0;                 // tiles issued by this CTA so far (S buffer = tile & 1)
    int chunks = 0;               // chunks begun (O buffer)
    uint32_t qphase = 0;
    bool ok = true;
    // the tile whose PV is still to be issued
    bool pend = false, pend_first = false, pend_last = false;
    int pend_nb = 0, pend_stage = 0, pend_tile = 0, pend_chunk = 0;
    auto issue_pv = [&]() {
      const int sb = pend_tile & 1, ob = S::O_BUFS == 2 ? pend_chunk & 1 : 0;
      if (pend_first) {
        // the O buffer's previous chunk has been read
        const int use = S::O_BUFS == 2 ? pend_chunk >> 1 : pend_chunk;
        ok = ok && warp_wait(&o_empty[ob], (use & 1) ^ 1, p.status, KC_DEV_ATTN | 3);
      }
      ok = ok && warp_wait(&p_ready[sb], (pend_tile >> 1) & 1, p.status, KC_DEV_ATTN | 4);
      if (!ok) return;
      tc_fence_after();
      const uint32_t v_lo = (uint32_t)vd + pend_stage * (S::TILE_BYTES >> 4);
      const uint32_t o = tmem + S::TMEM_O + ob * D, a = tmem + sb * TK;
      if (elect_one()) {
        for (int b = 0; b < pend_nb; ++b) {
          const uint32_t vb = v_lo + b * (2 * S::GROUP_BYTES >> 4);
          umma_bf16_ts(o, a + b * 16, vb, v_hi, idesc_pv, pend_first && b == 0 ? 0u : 1u);
          umma_bf16_ts(o, a + b * 16 + 8, vb, v_hi, idesc_pv, 1u);
        }
        umma_commit(&pv_done[sb]);
        umma_commit(&kv_empty[pend_stage]);
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
        // QK of this tile goes ahead of the pending PV when its operands are there before the probabilities are; a PV that
        // is waited for first leaves the softmax warps without scores for the time of both products. The looks are limited:
        // whatever is missing after them is waited for in the bounded waits below.
        if (pend) {
          for (int looks = 0; looks < 256; ++looks) {
            const bool scores = mbar_test_wait(&kv_full[kv.stage], kv.phase) && (!first_of_unit || mbar_test_wait(q_full, qphase));
            if (__all_sync(0xffffffffu, scores)) break;
            if (looks == 255 || __all_sync(0xffffffffu, mbar_test_wait(&p_ready[pend_tile & 1], (pend_tile >> 1) & 1))) { issue_pv(); break; }
          }
          if (!ok) break;
        }
        if (first_of_unit) {
          ok = warp_wait(q_full, qphase, p.status, KC_DEV_ATTN | 5);
          if (!ok) break;
          qphase ^= 1;
        }
        ok = warp_wait(&kv_full[kv.stage], kv.phase, p.status, KC_DEV_ATTN | 6);
        if (!ok) break;
        first_of_unit = false;
        tc_fence_after();
        const int nb = u.blocks(TK), sb = tile & 1;
        const bool first = u.t == u.first_tile(TK), last = u.last();
        const uint32_t k_lo = (uint32_t)kd + kv.stage * (S::TILE_BYTES >> 4);
        const uint32_t idesc = umma_idesc_bf16(ATT_ROWS, nb * 16);
        const int stage = kv.stage;
        const int chunk = chunks;
        if (last) ++chunks;
        u.next(TK);
        const bool unit_done = !u.live();
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks)
            umma_bf16_ss(tmem + sb * TK, (uint32_t)qd + (ks >> 2) * (ATT_ROWS * 128 >> 4) + (ks & 3) * 2, q_hi,
                         k_lo + (ks >> 2) * (1024 >> 4) + (ks & 3) * 2, k_hi, idesc, ks == 0 ? 0u : 1u);
          umma_commit(&s_ready[sb]);
          if (unit_done) umma_commit(q_empty);
        }
        __syncwarp();
        if (pend) issue_pv();
        pend = true; pend_first = first; pend_last = last; pend_nb = nb; pend_stage = stage; pend_tile = tile; pend_chunk = chunk;
        ++tile;
        kv.advance(S::RING);
      }
    }
    if (ok && pend) issue_pv();
  } else if (warp >= 4 && warp < 8) {
    // ---- softmax: thread = query row 32 * (warp & 3) + lane ----
    pdl_wait();
    const int quarter = warp & 3, row = quarter * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const float scale_log2 = FOLDED ? p.scale * 1.4426950408889634f : 1.4426950408889634f;
    const float cap_arg = FOLDED && p.softcap > 0.f ? p.scale / p.softcap : 0.f;
    const float cap_log2 = p.softcap * 1.4426950408889634f;
    int tile = 0, chunks = 0;
    bool ok = true;
    for (int r = 0, w; ok && r * (int)gridDim.x < total; ++r) {
      if ((w = unit_index(r, blockIdx.x, gridDim.x, total)) < 0) break;
      UnitTiles u;
      u.open(p, w / p.Hkv, TK);
      if (!u.live()) continue;
      const bool warp_live = quarter * 32 < u.rows;
      const int pos = u.pos0 + min(row / p.gqa, u.ntok - 1);      // dead rows of a live warp compute the last token's row
      const int w_excl = p.window > 0 ? pos - p.window : -1;       // keys <= this are outside the window
      float m = -INFINITY, l = 0.f;
      for (; u.live() && ok; u.next(TK), ++tile) {
        const int sb = tile & 1;
        const bool first = u.t == u.first_tile(TK), last = u.last();
        ok = warp_wait(&s_ready[sb], (tile >> 1) & 1, p.status, KC_DEV_ATTN | 7);
        if (!ok) break;
        if (first) { m = -INFINITY; l = 0.f; }
        if (warp_live) {
          tc_fence_after();
          const uint32_t s_addr = tmem + lane_addr + sb * TK;
          const int nb = u.blocks(TK), key0 = u.key0(TK);
          // columns of the tile that this row does not see: j > hi or j < lo. Columns past 16 nb hold an older tile's scores.
          const int hi = pos - key0, lo = w_excl - key0 + 1;
          // every key of the tile is visible to every row of the unit: the same arithmetic without the predicates
          const bool edge = !(nb * 16 == TK && key0 + TK - 1 <= u.pos0 && (p.window == 0 || key0 > u.pos_max - p.window));
          if (!FOLDED) {
#pragma unroll 1
            for (int c = 0; c < TK / 32; ++c) {
              uint32_t x[32];
              tmem_ld32(s_addr + c * 32, x);
#pragma unroll
              for (int j = 0; j < 32; ++j) {
                float f = __uint_as_float(x[j]) * p.scale;
                if (p.softcap > 0.f) f = p.softcap * tanhf(f / p.softcap);
                x[j] = __float_as_uint(f);
              }
              tmem_st32(s_addr + c * 32, x);
            }
            tmem_wait_st();
          }
          // Two passes over the tile's scores, 64 columns a turn: unrolled over the tile they were 25 KB of instructions, which
          // a launch fetches anew, most of the time of a short context.
          uint32_t va[32], vb[32];
          auto mask = [&](uint32_t (&v)[32], int c) {
            if (edge) {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (c + j > hi || c + j < lo) v[j] = 0xff800000u;   // -inf
            }
          };
          // three operands an instruction
          float t0 = -INFINITY, t1 = -INFINITY, t2 = -INFINITY, t3 = -INFINITY;
#pragma unroll 1
          for (int c = 0; c < TK; c += 64) {
            tmem_ld32_issue(s_addr + c, va);
            tmem_ld32_issue(s_addr + c + 32, vb);
            tmem_wait_ld();
            tmem_pin32(va);
            tmem_pin32(vb);
            mask(va, c);
            mask(vb, c + 32);
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
              t0 = fmaxf(t0, fmaxf(__uint_as_float(va[j]), __uint_as_float(va[j + 1])));
              t1 = fmaxf(t1, fmaxf(__uint_as_float(va[j + 2]), __uint_as_float(va[j + 3])));
              t2 = fmaxf(t2, fmaxf(__uint_as_float(vb[j]), __uint_as_float(vb[j + 1])));
              t3 = fmaxf(t3, fmaxf(__uint_as_float(vb[j + 2]), __uint_as_float(vb[j + 3])));
            }
          }
          tmem_ld32_issue(s_addr, va);   // arrives under what follows
          float tmax = fmaxf(fmaxf(t0, t1), fmaxf(t2, t3)), mul = scale_log2;
          const bool capped = FOLDED && p.softcap > 0.f;
          if (capped) {
            mul = cap_log2;
            const bool seen = !edge || (hi >= 0 && lo < TK && lo <= hi);   // any key: a score of -inf is a key of weight e^-cap
            if (seen) { tmax *= cap_arg; tmax = tanh_any(tmax, tanh_near(make_float2(tmax, tmax)).x); }   // grows with the score
          }
          tmax *= mul;
          float alpha = 1.f;
          // The reference lags behind the running maximum by up to 8 powers of two, which spares most rescales and costs no
          // precision: l, O and the two parts of a probability are floating-point numbers.
          if (tmax > m + 8.f) { alpha = ex2(m - tmax); m = tmax; }   // from -inf: alpha = 0
          const float ref = m == -INFINITY ? 0.f : m;
          const float2 muls = make_float2(mul, mul), refs = make_float2(-ref, -ref), minus1 = make_float2(-1.f, -1.f);
          // Sums: 32 keys pairwise, keys 16, 8, 4, 2 and 1 apart, then the tile's (kc_attn_keys.cu adds across lanes in this order).
          float part = 0.f, tile_sum = 0.f;
          // 32 scores of the row -> 32 columns of probabilities, as two bf16 numbers each: the columns of a 16-key block get
          // its eight pairs' upper parts, then what those leave over
          auto group = [&](uint32_t (&v)[32], int c) {
            if (capped) {
              // A group with no score past 0.75 caps takes the polynomial alone, two elements at a time; an element's value
              // is the same on both sides.
              float b0 = 0.f, b1 = 0.f;
#pragma unroll
              for (int j = 0; j < 32; j += 2) { b0 = fmaxf(b0, fabsf(__uint_as_float(v[j]))); b1 = fmaxf(b1, fabsf(__uint_as_float(v[j + 1]))); }
              // columns that hold an older tile's scores and rows past the unit's have no say but in the time it takes
              const bool all_near = __all_sync(0xffffffffu, fmaxf(b0, b1) * cap_arg < TANH_NEAR || row >= u.rows);
              const float2 arg = make_float2(cap_arg, cap_arg);
              if (all_near) {
#pragma unroll
                for (int j = 0; j < 32; j += 2) {
                  const float2 r = tanh_near(mul2(make_float2(__uint_as_float(v[j]), __uint_as_float(v[j + 1])), arg));
                  v[j] = __float_as_uint(r.x); v[j + 1] = __float_as_uint(r.y);
                }
              } else {
#pragma unroll
                for (int j = 0; j < 32; j += 2) {
                  const float2 y = mul2(make_float2(__uint_as_float(v[j]), __uint_as_float(v[j + 1])), arg);
                  const float2 r = tanh_near(y);
                  v[j] = __float_as_uint(tanh_any(y.x, r.x)); v[j + 1] = __float_as_uint(tanh_any(y.y, r.y));
                }
              }
            }
            mask(v, c);
            uint32_t w[32];
            float2 sums[8];
#pragma unroll
            for (int j = 0; j < 16; j += 2) {
              float2 e = fma2(make_float2(__uint_as_float(v[j]), __uint_as_float(v[j + 1])), muls, refs);
              float2 f = fma2(make_float2(__uint_as_float(v[j + 16]), __uint_as_float(v[j + 17])), muls, refs);
              e.x = ex2(e.x); e.y = ex2(e.y); f.x = ex2(f.x); f.y = ex2(f.y);
              sums[j / 2] = add2(e, f);
              const uint32_t eh[2] = {__float_as_uint(e.x) & 0xffff0000u, __float_as_uint(e.y) & 0xffff0000u};
              const uint32_t fh[2] = {__float_as_uint(f.x) & 0xffff0000u, __float_as_uint(f.y) & 0xffff0000u};
              w[j / 2] = __byte_perm(eh[0], eh[1], 0x7632);
              w[j / 2 + 16] = __byte_perm(fh[0], fh[1], 0x7632);
              const float2 el = fma2(make_float2(__uint_as_float(eh[0]), __uint_as_float(eh[1])), minus1, e);
              const float2 fl = fma2(make_float2(__uint_as_float(fh[0]), __uint_as_float(fh[1])), minus1, f);
              w[j / 2 + 8] = pack_bf162(el.x, el.y);
              w[j / 2 + 24] = pack_bf162(fl.x, fl.y);
            }
            tmem_st32(s_addr + c, w);
#pragma unroll
            for (int d = 4; d > 0; d /= 2)
#pragma unroll
              for (int j = 0; j < d; ++j) sums[j] = add2(sums[j], sums[j + d]);
            return sums[0].x + sums[0].y;
          };
          tmem_wait_ld();
          tmem_pin32(va);
#pragma unroll 1
          for (int c = 0; c < TK; c += 64) {
            tmem_ld32_issue(s_addr + c + 32, vb);
            part = group(va, c);
            tmem_wait_ld();
            tmem_pin32(vb);
            if (c + 64 < TK) tmem_ld32_issue(s_addr + c + 64, va);
            part += group(vb, c + 32);
            tile_sum = c == 0 ? part : tile_sum + part;
            tmem_wait_ld();
            tmem_pin32(va);
          }
          l = __fmaf_rn(l, alpha, tile_sum);
          if (!first && !__all_sync(0xffffffffu, alpha == 1.f || row >= u.rows)) {
            // a row's maximum moved: what O holds of it is rescaled once the previous tile's product is in
            const int pt = tile - 1;
            ok = warp_wait(&pv_done[pt & 1], (pt >> 1) & 1, p.status, KC_DEV_ATTN | 8);
            if (!ok) break;
            tc_fence_after();
            const uint32_t o_addr = tmem + lane_addr + S::TMEM_O + (S::O_BUFS == 2 ? (chunks & 1) * D : 0);
#pragma unroll 1
            for (int c = 0; c < D / 64; ++c) {
              uint32_t o[64];
              tmem_ld32_issue(o_addr + c * 64, o);
              tmem_ld32_issue(o_addr + c * 64 + 32, o + 32);
              tmem_wait_ld();
#pragma unroll
              for (int j = 0; j < 64; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
              tmem_st32(o_addr + c * 64, o);
              tmem_st32(o_addr + c * 64 + 32, o + 32);
            }
          }
          tmem_wait_st();
          tc_fence_before();
        }
        if (last) {
          const int cb = chunks & 1;
          // (m, l) of the chunk two before this one has been read (with one O buffer the wait is implied by that buffer's)
          ok = warp_wait(&o_empty[S::O_BUFS == 2 ? cb : 0], S::O_BUFS == 2 ? ((chunks >> 1) & 1) ^ 1 : (chunks & 1) ^ 1, p.status, KC_DEV_ATTN | 9);
          if (!ok) break;
          stat[cb * ATT_ROWS + row] = make_float2(m, l);
          __syncwarp();
          if (lane == 0) mbar_arrive(&stat_full[cb]);
          ++chunks;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_ready[sb]);
      }
    }
  } else if (warp >= 8) {
    // ---- a finished chunk: thread = query row ----
    pdl_wait();   // the stores below may overwrite what an earlier kernel still reads
    const int quarter = warp & 3, row = quarter * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    int chunks = 0;
    bool ok = true;
    constexpr int ACC = WHOLE ? D : 1;
    float acc[ACC];
    for (int r = 0, w; ok && r * (int)gridDim.x < total; ++r) {
      if ((w = unit_index(r, blockIdx.x, gridDim.x, total)) < 0) break;
      UnitTiles u;
      const int kvh = w % p.Hkv;
      u.open(p, w / p.Hkv, TK);
      if (!u.live()) continue;
      const bool warp_live = quarter * 32 < u.rows, row_live = row < u.rows;
      const int t = row / p.gqa;
      const size_t orow = (size_t)(u.tok0 + t) * p.Hq + kvh * p.gqa + (row - t * p.gqa);
      float macc = -INFINITY, lacc = 0.f;
      if (WHOLE) {
#pragma unroll
        for (int j = 0; j < ACC; ++j) acc[j] = 0.f;
      }
      for (; u.c < u.c1 && ok; ++u.c, ++chunks) {
        const int cb = chunks & 1, ob = S::O_BUFS == 2 ? cb : 0;
        const uint32_t oph = S::O_BUFS == 2 ? (chunks >> 1) & 1 : chunks & 1;
        ok = warp_wait(&stat_full[cb], (chunks >> 1) & 1, p.status, KC_DEV_ATTN | 10) && warp_wait(&o_full[ob], oph, p.status, KC_DEV_ATTN | 11);
        if (!ok) break;
        if (warp_live) {
          tc_fence_after();
          const float2 ml = stat[cb * ATT_ROWS + row];
          const uint32_t o_addr = tmem + lane_addr + S::TMEM_O + ob * D;
          if (WHOLE) {
            const MergeW mw = merge_weights(macc, ml.x);
            macc = mw.m;
            lacc = merge_value(lacc, ml.y, mw);
#pragma unroll
            for (int c = 0; c < D / 32; ++c) {
              uint32_t o[32];
              tmem_ld32(o_addr + c * 32, o);
#pragma unroll
              for (int j = 0; j < 32; j += 2) {
                const float2 v = merge_values(make_float2(acc[(c * 32 + j) % ACC], acc[(c * 32 + j + 1) % ACC]),
                                              make_float2(__uint_as_float(o[j]), __uint_as_float(o[j + 1])), mw);
                acc[(c * 32 + j) % ACC] = v.x; acc[(c * 32 + j + 1) % ACC] = v.y;
              }
            }
          } else {
            const size_t prow = orow * p.max_chunks + u.c;
            float* po = p.part_o + prow * D;
            if (row_live && !p.single) p.part_ml[prow] = ml;
            const RowSum l = row_sum(ml.y);
#pragma unroll 1
            for (int c = 0; c < D / 32; ++c) {
              uint32_t o[32];
              tmem_ld32(o_addr + c * 32, o);
              if (row_live && p.single) {
                // the row's only chunk: merging it into nothing changes no bit but the sign of a -0, so the row is finished
                // here, with the 0 added that merging adds
                bf16* out = p.out + orow * D + c * 32;
#pragma unroll
                for (int j = 0; j < 32; j += 8) {
                  uint32_t q[4];
#pragma unroll
                  for (int k = 0; k < 4; ++k)
                    q[k] = finish2(__uint_as_float(o[j + 2 * k]), __uint_as_float(o[j + 2 * k + 1]), l);
                  *reinterpret_cast<uint4*>(out + j) = make_uint4(q[0], q[1], q[2], q[3]);
                }
              } else if (row_live) {
#pragma unroll
                for (int j = 0; j < 32; j += 4)
                  *reinterpret_cast<uint4*>(po + c * 32 + j) = make_uint4(o[j], o[j + 1], o[j + 2], o[j + 3]);
              }
            }
          }
          tc_fence_before();
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&o_empty[ob]);
      }
      if (WHOLE && ok && row_live) {
        const RowSum l = row_sum(lacc);
        bf16* out = p.out + orow * D;
#pragma unroll
        for (int j = 0; j < ACC; j += 8) {
          uint32_t q[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) q[k] = finish2(acc[(j + 2 * k) % ACC], acc[(j + 2 * k + 1) % ACC], l);
          *reinterpret_cast<uint4*>(out + j) = make_uint4(q[0], q[1], q[2], q[3]);
        }
      }
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

// The chunks of a row merged in index order: the arithmetic of a whole-row unit (merge_weights, merge_value) over the
// stored partials. Chunks are taken eight at a time with all of a batch's loads issued before the first use.
template <int D>
__global__ void attn_combine_kernel(const AttnParams p, int n_rows) {
  pdl_launch_dependents();
  pdl_wait();
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= n_rows) return;
  const int tok = row / p.Hq;
  const int pos = p.token_pos[tok];
  const int c_hi = pos / ATT_CHUNK;
  const int c_lo = p.window > 0 ? max(0, pos - p.window + 1) / ATT_CHUNK : 0;
  const float2* ml = p.part_ml + (size_t)row * p.max_chunks;
  constexpr int CB = 8;
  constexpr int PER = D / 32;
  float acc[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) acc[i] = 0.f;
  float macc = -INFINITY, lacc = 0.f;
  for (int c0 = c_lo; c0 <= c_hi; c0 += CB) {
    float2 v[CB];
    float po[CB][PER];
#pragma unroll
    for (int j = 0; j < CB; ++j) {
      const bool on = c0 + j <= c_hi;
      v[j] = on ? ml[c0 + j] : make_float2(-INFINITY, 0.f);
      const float* src = p.part_o + ((size_t)row * p.max_chunks + (on ? c0 + j : c_lo)) * D + lane * PER;
      if (PER % 4 == 0) {
#pragma unroll
        for (int i = 0; i < PER; i += 4) {
          const float4 q = on ? *reinterpret_cast<const float4*>(src + i) : make_float4(0.f, 0.f, 0.f, 0.f);
          po[j][i] = q.x; po[j][i + 1] = q.y; po[j][i + 2] = q.z; po[j][i + 3] = q.w;
        }
      } else {
        const float2 q = on ? *reinterpret_cast<const float2*>(src) : make_float2(0.f, 0.f);
        po[j][0] = q.x; po[j][PER - 1] = q.y;
      }
    }
#pragma unroll
    for (int j = 0; j < CB; ++j) {
      if (c0 + j <= c_hi) {
        const MergeW mw = merge_weights(macc, v[j].x);
        macc = mw.m;
        lacc = merge_value(lacc, v[j].y, mw);
#pragma unroll
        for (int i = 0; i < PER; ++i) acc[i] = merge_value(acc[i], po[j][i], mw);
      }
    }
  }
  const RowSum l = row_sum(lacc);
  bf16* out = p.out + (size_t)row * D + lane * PER;
  uint32_t q[PER / 2];
#pragma unroll
  for (int i = 0; i < PER / 2; ++i) q[i] = finish2(acc[2 * i], acc[2 * i + 1], l);
  if constexpr (PER == 8) *reinterpret_cast<uint4*>(out) = make_uint4(q[0], q[1], q[2], q[3]);
  else if constexpr (PER == 4) *reinterpret_cast<uint2*>(out) = make_uint2(q[0], q[1]);
  else *reinterpret_cast<uint32_t*>(out) = q[0];
}

template <int D, bool WHOLE, bool FOLDED>
cudaError_t launch_attn_as(const CUtensorMap& map, const CUtensorMap& q, const CUtensorMap& q_small, const AttnParams& p, bool in_order, int sm_count,
                        cudaStream_t s) {
  using S = AttnShape<D>;
  static DeviceOnce configured;   // the attribute belongs to the device's copy of the kernel
  if (configured.first_on_current_device()) {
    cudaError_t e = cudaFuncSetAttribute(attn_kernel<D, WHOLE, FOLDED>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM);
    if (e != cudaSuccess) { configured.forget_current_device(); return e; }
  }
  const int grid = std::min(p.n_units * p.Hkv, sm_count);
  return launch_k_opt(!in_order, attn_kernel<D, WHOLE, FOLDED>, dim3(grid), dim3(ATT_THREADS), S::SMEM, s, map, q, q_small, p);
}
template <int D, bool WHOLE>
cudaError_t launch_attn(const CUtensorMap& map, const CUtensorMap& q, const CUtensorMap& q_small, const AttnParams& p, bool in_order, int sm_count,
                        cudaStream_t s) {
  return scale_folds(p.scale, p.softcap) ? launch_attn_as<D, WHOLE, true>(map, q, q_small, p, in_order, sm_count, s)
                                         : launch_attn_as<D, WHOLE, false>(map, q, q_small, p, in_order, sm_count, s);
}

template <int D>
cudaError_t launch_d(const CUtensorMap& map, const CUtensorMap& kmap, const CUtensorMap& q, const CUtensorMap& q_small, const AttnParams& p,
                     bool in_order, int n_tokens, int sm_count, cudaStream_t s) {
  cudaError_t e;
  if (p.keys) {
    e = attn_keys(kmap, q, q_small, p, in_order, scale_folds(p.scale, p.softcap), D, sm_count, s);
    if (p.whole) return e;
  } else {
    if (p.whole) {
      if constexpr (D <= 128) return launch_attn<D, true>(map, q, q_small, p, in_order, sm_count, s);
      else return cudaErrorInvalidValue;
    }
    e = launch_attn<D, false>(map, q, q_small, p, in_order, sm_count, s);
  }
  if (e != cudaSuccess || p.single) return e;
  const int n_rows = n_tokens * p.Hq;
  return launch_k(attn_combine_kernel<D>, dim3((n_rows + 7) / 8), dim3(256), 0, s, p, n_rows);
}

}  // namespace

int attn_tokens_per_item(int gqa, int max_len) {
  return std::min(std::max(1, ATT_ROWS / gqa), std::max(1, max_len));
}

// In a step attn_keys_kernel has its first tiles from under the tail of the kernel ahead, 3 us or more that a call on its own
// doesn't save. attn_kernel -> attn_keys_kernel, us a layer that a step gains: head sizes 128 and 256 at 64 rows 0 to 24
// (one sequence of 100 keys and head size 256 loses 1.5), at 36 rows 1 to 34; head size 64 at 28 rows 0 to 14, at 32 rows 0
// to 7, at 36 rows -6 to 4, at 64 -20 to 0: its tile is half the bytes and costs the softmax warps the same. Where no row has
// a second chunk there is little but the start: one sequence of 100 keys 2.1 at 36 rows, 0.4 at 64; 32 of 100 1.8 at 48, -1.1
// at 64.
// On its own the line falls with fewer tiles an SM, where a unit's start and end weigh, and rises under a cap, which costs
// a row per thread more: one sequence of 1001 keys, head size 64, 19 -> 20.5 us at 8 rows, 18 -> 25 at 64; 48 of 6000 159 ->
// 139 at 24, 203 -> 248 at 64; 128 and 64 rows, 32 of 1400 60 -> 64, under a cap 118 -> 110; 256, 48 of 40 21 -> 24 at 32
// rows, 23 -> 33 at 64; 64 of 2500, units of whole rows, which attn_kernel does not have at that size, 84 us less at 64.
// Over 7500 such calls the choice is 0.13 % behind the better kernel on average, 12 % at most.
int attn_key_rows(int head_dim, bool alone, bool capped, AttnForm form, long long tiles, int sm_count) {
  if (!alone) return head_dim > 64 ? KEY_ROWS : form != AttnForm::one_chunk ? 32 : tiles < sm_count ? KEY_ROWS : 48;
  // by tiles an SM: under 1, 2, 4, 8, and more
  static constexpr uint8_t apart[3][2][5] = {{{0, 0, 16, 24, 32}, {24, 32, 32, 40, 56}}, {{16, 24, 32, 32, 48}, {32, 40, 48, 56, 64}}, {{32, 32, 56, 64, 64}, {32, 32, 56, 64, 64}}};
  static constexpr uint8_t rest[3][2][5] = {{{32, 32, 32, 32, 32}, {40, 48, 56, 56, 64}}, {{32, 40, 40, 40, 40}, {40, 56, 64, 64, 64}}, {{24, 24, 28, 40, 40}, {24, 24, 28, 40, 40}}};
  if (head_dim == 256 && form == AttnForm::whole) return KEY_ROWS;
  int load = 0;
  while (load < 4 && tiles >= (long long)sm_count << load) ++load;
  return (form == AttnForm::apart ? apart : rest)[head_dim / 128][capped ? 1 : 0][load];
}

bool attn_whole(const int* item_tiles, int n_items, int kv_heads, int sm_count) {
  const int total = n_items * kv_heads, ctas = std::min(total, sm_count);
  long long sum = 0, most = 0;
  for (int i = 0; i < n_items; ++i) sum += (long long)item_tiles[i] * kv_heads;
  std::vector<int> load(ctas, 0);
  for (int r = 0; r * ctas < total; ++r)
    for (int c = 0; c < ctas; ++c) {
      const int w = unit_index(r, c, ctas, total);
      if (w >= 0) load[c] += item_tiles[w / kv_heads];
    }
  for (int c = 0; c < ctas; ++c) most = std::max<long long>(most, load[c]);
  // Four tiles are one chunk: nothing to split. Whole rows save the partials' round trip through memory and the combine
  // launch (about a tenth of a step of 32 long sequences); units of one chunk are for steps whose items leave SMs idle
  // for longer than that.
  return most <= 4 || most * sm_count * 4 <= sum * 5;
}

// Queries [n_tokens][Hkv][gqa][D] as {64 features, gqa, slabs, Hkv, tokens}: one operation brings a slab of up to 128
// rows in (token, head) order. Tokens past the end read as zeros.
bool make_tmap_q(CUtensorMap* map, const bf16* q, int n_tokens, int Hq, int gqa, int head_dim, int box_tokens, const char** err) {
  const uint64_t D = head_dim, dims[5] = {64, (uint64_t)gqa, D / 64, (uint64_t)(Hq / gqa), (uint64_t)n_tokens};
  const uint64_t strides[4] = {D * 2, 128, (uint64_t)gqa * D * 2, (uint64_t)Hq * D * 2};
  const uint32_t box[5] = {64, (uint32_t)gqa, 1, 1, (uint32_t)box_tokens};
  return encode_tmap_bf16(map, 5, q, dims, strides, box, err);
}

// K/V pools as a 5-D tensor {64 features, 8 rows, head_dim / 64 slabs, planes, plane_rows / 8} with box {64, 8, slabs, 1 or 2, 2}:
// ONE operation brings 16 keys of K or V, or of both, of a layer (plane 2 * layer and the next) as two groups of 8 keys, each
// with its K slabs and then its V slabs of [8][128 B], 128-byte swizzle. Groups of 8 rows at one constant stride are what a
// tensor-core operand of many 16-key blocks needs, wherever the block table scatters them. The slab stride (128 B) is
// smaller than the row stride, which the encoder may refuse: the caller then keeps the 2-D map (8 rows x 64 features).
bool make_tmap_kv_5d(CUtensorMap* map, const void* pool, uint32_t head_dim, uint64_t plane_rows, uint64_t planes, uint32_t box_planes, const char** err) {
  const uint64_t D = head_dim, dims[5] = {64, 8, D / 64, planes, plane_rows / 8};
  const uint64_t strides[4] = {D * 2, 128, plane_rows * D * 2, 8 * D * 2};
  const uint32_t box[5] = {64, 8, head_dim / 64, box_planes, 2};
  return encode_tmap_bf16(map, 5, pool, dims, strides, box, err);
}
bool make_tmap_kv_2d(CUtensorMap* map, const void* pool, uint32_t head_dim, uint64_t rows, const char** err) {
  const uint64_t dims[2] = {head_dim, rows}, strides[1] = {(uint64_t)head_dim * 2};
  const uint32_t box[2] = {64, 8};
  return encode_tmap_bf16(map, 2, pool, dims, strides, box, err);
}

cudaError_t paged_attention(const CUtensorMap& kvmap, const CUtensorMap& kmap, const CUtensorMap& qmap, const CUtensorMap& qmap_small,
                            const AttnParams& p, bool in_order, int head_dim, int n_tokens, int sm_count, cudaStream_t s) {
  if (p.gqa < 1 || p.gqa * p.q_tokens > ATT_ROWS || p.n_units < 1) return cudaErrorInvalidValue;
  switch (head_dim) {
    case 64: return launch_d<64>(kvmap, kmap, qmap, qmap_small, p, in_order, n_tokens, sm_count, s);
    case 128: return launch_d<128>(kvmap, kmap, qmap, qmap_small, p, in_order, n_tokens, sm_count, s);
    case 256: return launch_d<256>(kvmap, kmap, qmap, qmap_small, p, in_order, n_tokens, sm_count, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace kc
