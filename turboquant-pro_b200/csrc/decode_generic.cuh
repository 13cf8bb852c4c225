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
// beside the general kernel's stand at its launch.  Distance from 64 bits over 30 to 12 000 tokens: 8.9e-7
// at five heads, 7.3e-7 at seven, 8.9e-7 at twelve; with plain float32 multiply-adds in place of the split
// products 1.11e-6, 9.2e-7 and 9.0e-7, the general kernel about 1.12e-6.
TQ_HD bool tq_decode_pages_form(const tq_geom& g) {
  return g.block_tokens == 256 && g.key_mode != TQ_KEYS_POLAR && g.group > 4;
}
constexpr int TQ_PAGES_SEQS = 2048;  // sequences a launch of the page kernel covers
int tq_launch_decode_pages(const DecodeArgs& a, int sm_count, cudaStream_t st);
