// Shared by the encoder kernels of the append path: their arguments, where a token's row is
// found, packed 16-bit helpers.
#pragma once

#include "common.cuh"

struct EncodeArgs {
  tq_geom g;
  uint8_t* pages;
  void* hot_k;
  void* hot_v;
  uint32_t* pool_dec;
  uint16_t* pool_val;
  PageMeta* page_meta;
  int32_t* seq_len;      // [L][B]
  uint32_t* pool_cursor; // [L][B][H]
  int32_t* status;
  const Tables* tables;
  const float* bias_means;  // given key zero-points [max_blocks][H][D], or null
  const void* k;
  const void* v;
  int layer, seq_begin, seq_count, n_tokens, max_new_blocks;
  int64_t seq_stride, tok_stride, head_stride;
  // PolarQuant keys (TQ_KEYS_POLAR): the value encoder also runs over the keys, writing their
  // codes where the per-channel codes would go and their norms over the scale / mean arrays
  int polar_keys_pass;
  // bounded waits of the encoders: probes (0: their defaults); test hook: the row of the first new
  // block whose copy the key encoder never starts, or 2^20 + the tile whose products the first CTA of the
  // value encoder never starts (-1: none)
  int wait_limit, withhold_row;
};

// Where token `pos` of (seq, head) currently lives: positions below n0 are already in the
// hot ring, the rest are in the caller's tensor.
template <int DT>
struct TokenSource {
  const void* ring;
  const void* in;
  int n0, cap;
  int64_t tok_stride;
  // one load from a selected address (no branch: loads of several positions can then be
  // in flight together)
  TQ_DEV float ld(int pos, int d) const {
    const bool old = pos < n0;
    const void* base = old ? ring : in;
    const size_t idx =
        old ? (size_t)(pos % cap) * TQ_D + d : (size_t)(pos - n0) * tok_stride + d;
    return Elem<DT>::ld(base, idx);
  }
};

template <int DT>
TQ_DEV TokenSource<DT> make_source(const EncodeArgs& a, const void* ring_base, const void* in_base,
                                   int seq, int head, int n0) {
  TokenSource<DT> s;
  s.ring = (const uint8_t*)ring_base +
           hot_offset_elems(a.g, a.layer, seq, head) * sizeof(typename Elem<DT>::type);
  s.in = (const uint8_t*)in_base +
         ((size_t)(seq - a.seq_begin) * a.seq_stride + (size_t)head * a.head_stride) *
             sizeof(typename Elem<DT>::type);
  s.n0 = n0;
  s.cap = a.g.hot_cap;
  s.tok_stride = a.tok_stride;
  return s;
}

// Packed minimum / maximum of two 16-bit floats (fp16 or bf16 by BF): the statistics of two
// tokens of a channel in one instruction.  The values are the tokens themselves, so nothing
// is rounded.
template <bool BF>
TQ_DEV uint32_t max2_16(uint32_t a, uint32_t b) {
  uint32_t r;
  if (BF) asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  else asm("max.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
template <bool BF>
TQ_DEV uint32_t min2_16(uint32_t a, uint32_t b) {
  uint32_t r;
  if (BF) asm("min.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  else asm("min.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
template <bool BF>
TQ_DEV float f16bits_to_float(uint32_t h) {
  return BF ? __uint_as_float(h << 16) : __half2float(__ushort_as_half((unsigned short)h));
}

// Key encoder for 256-token blocks with up to eight outliers per channel (encode_keys.cu), and
// whether a geometry is of that form.
bool tq_keys_block_form(const tq_geom& g);
int tq_launch_encode_keys_block(const EncodeArgs& a, int device, cudaStream_t st);

// Value encoder for blocks of 128 or 256 tokens (encode_values.cu).
constexpr float VALUE_SPAN = 1023.0f / 1024.0f;  // z = 1 still has a mantissa below 2^23
// `after_keys`: the kernel before it in the stream is the key encoder of the same call.
int tq_launch_encode_values_tiles(const EncodeArgs& a, const ValueTable& vt, bool after_keys,
                                  int sm_count, int device, cudaStream_t st);

TQ_DEV uint32_t enc_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// Shared-memory operand of tcgen05.mma, K-major without swizzling: 8 x 8 core matrices of 16-bit
// values (8 rows of 16 bytes), start address, "leading" offset to the next eight K and "stride"
// to the next eight rows in 16-byte units; descriptor version 1.
TQ_DEV uint64_t umma_desc_k_major(uint32_t saddr, uint32_t leading_bytes, uint32_t stride_bytes) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((leading_bytes >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((stride_bytes >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
TQ_DEV void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}
TQ_DEV void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
TQ_DEV void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
TQ_DEV bool mbar_try_wait(uint32_t bar, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(done)
      : "r"(bar), "r"(parity), "r"(2000u)  // (at most so many nanoseconds a probe)
      : "memory");
  return done != 0;
}
