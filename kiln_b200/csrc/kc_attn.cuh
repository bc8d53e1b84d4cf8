// Paged multi-query attention: launch parameters. See kc_attn.cu.
#pragma once

#include "kc_common.cuh"

namespace kc {

// Keys per chunk. Chunks are cut at absolute key positions, so the partition a
// query row sees depends only on its own position.
constexpr int ATT_CHUNK = 512;
constexpr int ATT_ROWS = 128;   // query rows (token x head of the group) of one work item: the lanes of tensor memory

// One unit of work for every kv head: consecutive tokens of one sequence against the chunks [chunk0, chunk1).
struct AttnUnit {
  int seq, tok0, ntok, pos0;    // sequence, first token row in the step, tokens, absolute position of the first
  int chunk0, chunk1;
  int small;                    // 1: at most ATT_SMALL_TOKENS tokens (the query map with the small box)
  int old;                      // keys from the sequence's start that nothing in this step writes
};
constexpr int ATT_SMALL_TOKENS = 8;
constexpr int KEY_ROWS = 64;    // the most rows of a unit of the kernel with a key per thread (kc_attn_keys.cu)

struct AttnParams {
  bf16* out;                   // [n_tokens, Hq * D], 16-byte aligned
  float* part_o;               // [n_tokens * Hq][max_chunks][D]  un-normalised partial outputs
  float2* part_ml;             // [n_tokens * Hq][max_chunks]     (running max in log2 units, sum)
  const int32_t* block_tables; // [n_seqs][max_blocks]
  const AttnUnit* units;       // [n_units]
  int n_units;
  const int32_t* token_pos;    // [n_tokens] absolute position of each token row
  uint32_t* status;
  int max_blocks;
  int Hq, Hkv, gqa;
  int layer, NB, BS;
  int max_chunks;
  int whole;                   // 1: every unit holds all chunks of its rows: the kernel writes `out`, no combine kernel follows
  int single;                  // 1: no row of the step has a second chunk (max_chunks == 1): no combine kernel either
  float scale;                 // softmax scale (applied to fp32 scores)
  float softcap;               // 0 = off
  int window;                  // 0 = global
  int keys;                    // 1: the kernel with a key per thread (attn_key_rows), 0: with a row per thread
  int q_tokens;                // tokens in the box of the large query map
  int kv5d;                    // the maps of the pools are 5-D (one operation per 16 keys) instead of 2-D
};

// Tokens of one sequence that share a CTA (their rows x gqa must fit ATT_ROWS).
int attn_tokens_per_item(int gqa, int max_len);
// Whether units of whole rows (all chunks of an item in one unit) keep the SMs about as busy as units of single chunks:
// item_tiles = tiles of 128 keys of each item, in the order of the units.
bool attn_whole(const int* item_tiles, int n_items, int kv_heads, int sm_count);
// The most rows of a unit with which the kernel with a key per thread is the faster one. alone: a call on its own, in plain
// stream order; else a step's. tiles: of 128 keys, over all items and kv heads.
enum class AttnForm { one_chunk, apart, whole };   // no row has a second chunk; units of single chunks, merged afterwards; units of whole rows
int attn_key_rows(int head_dim, bool alone, bool capped, AttnForm form, long long tiles, int sm_count);

// Query maps over [n_tokens, Hq, D] (5-D: 64 features, heads of a group, slabs, groups, tokens).
bool make_tmap_q(CUtensorMap* map, const bf16* q, int n_tokens, int Hq, int gqa, int head_dim, int box_tokens, const char** err);
// K/V pools [planes = layers * 2][plane_rows = NB * Hkv * BS][head_dim]: see kc_attn.cu.
// box_planes: 2 for K and V in one operation, 1 for either.
bool make_tmap_kv_5d(CUtensorMap* map, const void* pool, uint32_t head_dim, uint64_t plane_rows, uint64_t planes, uint32_t box_planes, const char** err);
bool make_tmap_kv_2d(CUtensorMap* map, const void* pool, uint32_t head_dim, uint64_t rows, const char** err);

// in_order: the work before this call in the stream is not one of a step's kernels (the copy of units and block tables, a
// caller's own work): the first kernel is then launched behind it in plain stream order. kvmap: K and V of 16 keys; kmap: either.
cudaError_t paged_attention(const CUtensorMap& kvmap, const CUtensorMap& kmap, const CUtensorMap& qmap, const CUtensorMap& qmap_small,
                            const AttnParams& p, bool in_order, int head_dim, int n_tokens, int sm_count, cudaStream_t s);
// Its kernel for units of at most KEY_ROWS rows (kc_attn_keys.cu).
cudaError_t attn_keys(const CUtensorMap& kmap, const CUtensorMap& qmap, const CUtensorMap& qmap_small, const AttnParams& p, bool in_order, bool folded,
                      int head_dim, int sm_count, cudaStream_t s);

}  // namespace kc
