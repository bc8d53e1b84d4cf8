// Device code that both attention kernels share (kc_attn.cu: a row per thread; kc_attn_keys.cu: a key per thread): the same
// functions in the same order, so that a row has the same bits in either.
#pragma once

#include "kc_attn.cuh"
#include "kc_umma.cuh"

namespace kc {

// Adds a chunk (o scaled by 2^-m, sum l) to what a row has accumulated: the weights of one merge.
struct MergeW { float a, b, m; };
__device__ __forceinline__ MergeW merge_weights(float m_acc, float m_chunk) {
  MergeW w;
  w.m = fmaxf(m_acc, m_chunk);
  w.a = m_acc == -INFINITY ? 0.f : ex2(m_acc - w.m);
  w.b = m_chunk == -INFINITY ? 0.f : ex2(m_chunk - w.m);
  return w;
}
__device__ __forceinline__ float merge_value(float acc, float v, const MergeW& w) { return __fmaf_rn(v, w.b, __fmul_rn(acc, w.a)); }
__device__ __forceinline__ float2 merge_values(float2 acc, float2 v, const MergeW& w) { return fma2(v, make_float2(w.b, w.b), mul2(acc, make_float2(w.a, w.a))); }
// Two values of a finished row divided by its sum (a row without one keeps its zeros): times the reciprocal in two parts,
// one rounded down and what it leaves, so that the fp32 result is the rounded quotient but for quotients within 2^-48 of a
// rounding boundary. (The division operator took 5 us a unit of 128 values a thread more.) The second part is positive: an
// infinite value stays what it is. A -0 becomes +0.
struct RowSum { float2 r, rest; };
__device__ __forceinline__ RowSum row_sum(float l) {
  if (l == 0.f) l = 1.f;
  const float r = __frcp_rd(l), rest = fmaxf(__fmaf_rn(-l, r, 1.f) * r, 1e-35f);
  return {make_float2(r, r), make_float2(rest, rest)};
}
__device__ __forceinline__ uint32_t finish2(float a, float b, const RowSum& s) {
  const float2 x = make_float2(a, b), v = fma2(x, s.r, fma2(x, s.rest, make_float2(0.f, 0.f)));
  return pack_bf162(v.x, v.y);
}

// The tiles of one unit in order, as every role walks them.
struct UnitTiles {
  int seq, tok0, ntok, pos0, small, old, rows, pos_max, wlo;
  int c, c1, t, t1, keys;       // chunk, end of chunks, tile, end of tiles of the chunk, keys of the chunk
  __device__ __forceinline__ void open(const AttnParams& p, int unit, int tk) {
    const int4 a = *reinterpret_cast<const int4*>(&p.units[unit]);
    const int4 b = *(reinterpret_cast<const int4*>(&p.units[unit]) + 1);
    seq = a.x; tok0 = a.y; ntok = a.z; pos0 = a.w;
    c = b.x; c1 = b.y; small = b.z; old = b.w;
    rows = ntok * p.gqa;
    pos_max = pos0 + ntok - 1;
    wlo = p.window > 0 ? max(0, pos0 - p.window + 1) : 0;    // first key that any row of the unit sees
    c = max(c, wlo / ATT_CHUNK);
    chunk(tk);
  }
  __device__ __forceinline__ void chunk(int tk) {
    keys = min(ATT_CHUNK, pos_max + 1 - c * ATT_CHUNK);
    t = max(0, wlo - c * ATT_CHUNK) / tk;
    t1 = (keys + tk - 1) / tk;
  }
  __device__ __forceinline__ bool live() const { return c < c1; }
  __device__ __forceinline__ bool last() const { return t == t1 - 1; }
  __device__ __forceinline__ int first_tile(int tk) const { return max(0, wlo - c * ATT_CHUNK) / tk; }
  __device__ __forceinline__ int key0(int tk) const { return c * ATT_CHUNK + t * tk; }
  // 16-key blocks of the tile that hold a key of the sequence
  __device__ __forceinline__ int blocks(int tk) const { return (min(tk, keys - t * tk) + 15) >> 4; }
  __device__ __forceinline__ void next(int tk) {
    if (++t == t1) { if (++c < c1) chunk(tk); }
  }
};

// The r-th unit of a CTA: forth and back over the CTAs, so that with units in falling order of length every CTA gets about
// the same number of tiles (attn_whole counts them the same way). -1: no more.
__host__ __device__ __forceinline__ int unit_index(int r, int cta, int ctas, int total) {
  const int i = r * ctas + ((r & 1) ? ctas - 1 - cta : cta);
  return i < total ? i : -1;
}

}  // namespace kc
