// Arguments shared by the float32 decode kernels (decode_generic.cu, decode_pages.cu).
#pragma once

#include "common.cuh"

struct DecodeArgs {
  tq_geom g;
  const uint8_t* pages;
  const void* hot_k;
  const void* hot_v;
  const uint32_t* pool_dec;
  const PageMeta* page_meta;
  const int32_t* seq_len;
  const Tables* tables;
  const void* q;
  float* partials;  // [units][max_splits][G][2 + D]
  float* out;       // [n_seqs][n_q_heads][D] or null
  float* mlo;       // [n_seqs][n_q_heads][2 + D] or null
  int layer, q_dtype;
  int ns_cold, ns_hot;
  int block_begin, block_end, with_hot;
  float scale;
};

// Query groups of five and more on 256-token blocks (per-channel keys) take the page kernel; its times
// beside the general kernel's, and its distance from 64 bits, stand in decode_pages.cu.
TQ_HD bool tq_decode_pages_form(const tq_geom& g) {
  return g.block_tokens == 256 && g.key_mode != TQ_KEYS_POLAR && g.group > 4;
}
// The page kernel's scores, and the maxima of its partials, are in units of log 2, so that neither a score
// nor the exponent of a probability is rounded once more at its full size: of pages the query is multiplied
// by 1 / (sqrt(128) ln 2) before its weights are formed, of the window the sum is.  (A factor as two
// floats: a rounded one would move all scores by the same part in 2^25.)
// by = hi + lo, both positive: infinities stay what they are.
constexpr double TQ_LN2 = 0.69314718055994530942, TQ_SCORE_LOG2 = 1.0 / (11.313708498984760390 * TQ_LN2);
struct TqFactor {
  double by;
  float hi = (double)(float)by <= by ? (float)by : (float)(by - by * 0x1p-24), lo = (float)(by - (double)hi);
};
template <bool SCORE>
TQ_DEV float tq_scaled(float x) {  // times TQ_SCORE_LOG2, else times TQ_LN2
  constexpr TqFactor f{SCORE ? TQ_SCORE_LOG2 : TQ_LN2};
  static_assert(f.hi > 0.0f && f.lo > 0.0f, "");
  constexpr float hi = f.hi, lo = f.lo;
  return fmaf(x, hi, x * lo);
}
TQ_DEV float tq_exp2(float x) {
  float y;
  asm("ex2.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
constexpr int TQ_PAGES_SEQS = 2048;  // sequences a launch of the page kernel covers
int tq_launch_decode_pages(const DecodeArgs& a, int sm_count, cudaStream_t st);
