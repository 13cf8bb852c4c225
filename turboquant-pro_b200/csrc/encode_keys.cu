// Key encoder for the usual block (256 tokens, up to eight outliers per channel).
//
// What the general key encoder (encode.cu) computes, bit for bit.  That kernel was bound by
// instruction issue (150 instructions per element); this one spends 37 (16-bit tokens) or 43:
//   - a thread owns two neighbouring channels and a segment of the tokens, so 16-bit statistics
//     are packed two channels to an instruction and a code byte (two channels) is one store;
//   - the nearest level comes from one table look-up: the range of a channel is cut into 32 bins,
//     narrower than the distance of two code borders, and the channel's table gives for each bin
//     the border that can lie in it, with the code below the border in its low mantissa bits.
//     An element so close to the border that the rounding of the reference's distances could
//     decide (a few in a hundred thousand) is computed again the reference's way;
//   - the arithmetic up to the look-up runs on the FMA pipe (four warps a clock), integers
//     included: an address is formed as a denormal number, whose bits are its integer value;
//     the logic unit (two warps a clock) would be the limit otherwise;
//   - outliers: where a block is cut into 32 groups of eight tokens, the k largest magnitudes of a
//     channel lie in the k groups with the largest maxima (in a few more where maxima are equal),
//     so only those groups are searched for the k-th magnitude and for the tokens that reach it.
// Measured (B200): 8 x 16 384 fp16 tokens x 8 heads about 780 us with the general encoder, 234 us
// here; 4001 float32 tokens x 32 heads about 300 us and 60 us; the 32 blocks of one flush, alone on the
// GPU, 16 us.  What bounds it: latency.  Cycles of a CTA with another beside it on the SM (fp16): first rows
// 5.1 k, pass 1 4.5 k, table 3.5 k, pass 2 5.3 k, redos 1.5 k, outliers' search 5.4 k, their lists 6.7 k.
// (With the table behind a barrier of its own, all rows waited for at once and the outliers' slots stored
// one by one from the registers 246 us; with 512 threads a CTA 258 us.)
// The passes read the block from shared memory, eight tokens an iteration: all loads of an
// iteration first and its stores last, so that the eight chains of dependent steps overlap.
#include "encode.cuh"

namespace {

constexpr int EK_S = 256;       // tokens per block
constexpr int EK_K = 8;         // most outliers per channel and block
constexpr int EK_BINS = 32;
constexpr int EK_GROUPS = 32;   // groups of eight tokens per block
constexpr int EK_WAIT = 1 << 16;  // probes for the block's copies before the CTA gives up
constexpr float EK_MAGIC = 12582912.0f;  // 1.5 * 2^23: adding it rounds to an integer

template <int DT>
struct EkWord {  // two neighbouring channels of a token
  using type = uint32_t;
};
template <>
struct EkWord<TQ_F32> {
  using type = float2;
};

// Split of a block over the threads: 16-bit tokens 4 segments of 64 tokens x 64 channel pairs (two
// CTAs per SM), float32 8 segments of 32 tokens (its 128 KB of tokens leave room for one).
template <int DT>
struct Ek {
  using W = typename EkWord<DT>::type;
  static constexpr int NT = DT == TQ_F32 ? 32 : 64;
  static constexpr int SEG = EK_S / NT;
  static constexpr int THREADS = 64 * SEG;
  // shared memory
  static constexpr int ROWS = EK_S * TQ_D * (DT == TQ_F32 ? 4 : 2);
  static constexpr int TAB = EK_BINS * TQ_D * 4;       // the table, then the outlier list
  static constexpr int IMG = EK_S * TQ_D / 2;          // group maxima, then the page's code rows
  static constexpr int MM = 2 * SEG * TQ_D * 4;        // extremes of the segments, list of redos, the page's tail
  static constexpr int MASK = EK_S * 16;               // outlier channels of every token
  static constexpr int SMEM = ROWS + TAB + IMG + MM + MASK;
};
constexpr int EK_REDOS = EK_S / 8 * (TQ_D / 2);  // eight tokens of a channel pair each
static_assert(EK_GROUPS * TQ_D * 4 <= Ek<TQ_F32>::IMG && EK_REDOS * 2 <= Ek<TQ_F16>::MM &&
                  TQ_TAIL_BYTES <= Ek<TQ_F16>::MM,
              "shared areas");

// column of channel ch in the table: a warp's 32 even (odd) channels on 32 different banks
TQ_DEV int ek_col(int ch) { return (ch >> 1) + 64 * (ch & 1); }

TQ_DEV unsigned long long ek_pack(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
TQ_DEV void ek_unpack(unsigned long long v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
TQ_DEV unsigned long long ek_fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
TQ_DEV unsigned long long ek_add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
TQ_DEV float ek_fma_sat(float a, float b, float c) {
  float r;
  asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// smallest of m, |a| and |b|
TQ_DEV float ek_min_abs(float m, float a, float b) {
  float r;
  asm("min.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(m), "f"(a), "f"(b));
  return r;
}
// bit sets of the two halves: `bit` where a >= b (magnitudes of two channels)
template <bool BF>
TQ_DEV void ek_reach2(uint32_t a, uint32_t b, uint32_t bit, uint32_t& lo, uint32_t& hi) {
  if (BF)
    asm("{\n\t.reg .pred p, q;\n\tsetp.ge.bf16x2 p|q, %2, %3;\n\t@p or.b32 %0, %0, %4;\n\t"
        "@q or.b32 %1, %1, %4;\n\t}"
        : "+r"(lo), "+r"(hi)
        : "r"(a), "r"(b), "r"(bit));
  else
    asm("{\n\t.reg .pred p, q;\n\tsetp.ge.f16x2 p|q, %2, %3;\n\t@p or.b32 %0, %0, %4;\n\t"
        "@q or.b32 %1, %1, %4;\n\t}"
        : "+r"(lo), "+r"(hi)
        : "r"(a), "r"(b), "r"(bit));
}

template <int DT>
__global__ void __launch_bounds__(Ek<DT>::THREADS, DT == TQ_F32 ? 1 : 2)
    encode_keys_block_kernel(EncodeArgs a, int aligned) {
  using C = Ek<DT>;
  using W = typename C::W;
  using T = typename Elem<DT>::type;
  constexpr int NT = C::NT, SEG = C::SEG, THREADS = C::THREADS;
  constexpr int GPT = EK_GROUPS / SEG;  // groups per thread; token i of a segment is in group i % GPT
  constexpr bool BF = DT == TQ_BF16, F32 = DT == TQ_F32;
  const tq_geom& g = a.g;
  const int seq = a.seq_begin + blockIdx.z, head = blockIdx.y;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int p = tid & 63, seg = tid >> 6;  // channels 2p, 2p + 1; tokens seg * NT ...
  // (the value encoder behind this kernel in the stream touches nothing that it writes)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int n0 = a.seq_len[a.layer * g.n_seqs + seq];
  const int nb0 = n_cold_blocks(n0, g.hot_window, EK_S);
  const int nb1 = n_cold_blocks(n0 + a.n_tokens, g.hot_window, EK_S);
  const int blk = nb0 + blockIdx.x;
  if (blk >= nb1) return;
  const int pos0 = blk * EK_S;
  const int mode = g.key_mode, kk = g.outlier_k;
  uint8_t* page = a.pages + page_offset(g, a.layer, seq, head, blk);

  extern __shared__ __align__(128) uint8_t ek_smem[];
  const T* rows = (const T*)ek_smem;  // [256][128]
  uint32_t* tab = (uint32_t*)(ek_smem + C::ROWS);
  uint8_t* img = ek_smem + C::ROWS + C::TAB;
  float* s_mn = (float*)(img + C::IMG);  // [SEG][128]
  float* s_mx = s_mn + SEG * TQ_D;
  uint32_t* mask = (uint32_t*)(s_mx + SEG * TQ_D);  // [256][4]
  unsigned short* redos = (unsigned short*)s_mn;    // channel pair | group of eight tokens << 6
  __shared__ float s_sum[TQ_D], s_mu[TQ_D], s_scale[TQ_D], s_inv[TQ_D], s_off[TQ_D], s_tol[TQ_D];
  __shared__ float s_grid[16];
  __shared__ float4 s_bin[EK_BINS];  // levels beside the bin's border, code below it (as bits)
  __shared__ uint32_t s_groups[TQ_D];  // groups a channel's outliers lie in
  __shared__ int s_n_redo;
  __shared__ int s_alloc;
  __shared__ uint32_t s_off_pool, s_scan[EK_S / 32];
  __shared__ unsigned short s_row[EK_S], s_orow[EK_S];  // a token's first outlier, first overflow entry
  __shared__ int s_wide[TQ_WIDE];
  __shared__ __align__(8) unsigned long long s_bar[SEG];

  // Row of token t: below n0 the ring's (a block never wraps in it: its capacity is a multiple
  // of the block), else the caller's.
  const TokenSource<DT> src = make_source<DT>(a, a.hot_k, a.k, seq, head, n0);
  const T* ring_row0 = (const T*)src.ring + (size_t)(pos0 % src.cap) * TQ_D;
  const T* in_row0 = (const T*)src.in + ((int64_t)pos0 - n0) * src.tok_stride;
  const int n_old = n0 - pos0;  // tokens t < n_old are in the ring
  auto row_of = [&](int t) -> const T* {
    return t < n_old ? ring_row0 + (size_t)t * TQ_D : in_row0 + (int64_t)t * src.tok_stride;
  };
  // the block into shared memory: a bulk copy per row where rows are on the 16-byte grid (a barrier per
  // segment, so that the first pass starts before the last rows are there), else element by element
  constexpr int ROW_BYTES = TQ_D * (int)sizeof(T);
  if (aligned) {
    const uint32_t bar = (uint32_t)__cvta_generic_to_shared(s_bar);
    if (tid == 0) {
#pragma unroll
      for (int s = 0; s < SEG; ++s)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar + 8 * s) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
#pragma unroll
      for (int s = 0; s < SEG; ++s)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar + 8 * s), "r"(C::ROWS / SEG)
                     : "memory");
    }
    __syncthreads();
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(ek_smem);
    const bool held = tid == a.withhold_row && blockIdx.x + blockIdx.y + blockIdx.z == 0;  // test hook
    if (tid < EK_S && !held)
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
              dst + tid * ROW_BYTES),
          "l"(row_of(tid)), "r"(ROW_BYTES), "r"(bar + 8 * (tid / NT))
          : "memory");
  } else {
    for (int i = tid; i < EK_S * TQ_D; i += THREADS) ((T*)ek_smem)[i] = row_of(i >> 7)[i & 127];
  }
  // two channels of token t
  auto ldw = [&](int t) -> W { return ((const W*)rows)[t * 64 + p]; };
  auto lo_of = [&](const W& w) -> float {
    if constexpr (F32) return w.x;
    else return BF ? __uint_as_float(w << 16) : __low2float(*(const __half2*)&w);
  };
  auto hi_of = [&](const W& w) -> float {
    if constexpr (F32) return w.y;
    else return BF ? __uint_as_float(w & 0xFFFF0000u) : __high2float(*(const __half2*)&w);
  };
  if (tid < 16) s_grid[tid] = a.tables->grid[tid];
  if (tid == 0) s_n_redo = 0;
  for (int i = tid; i < EK_S * 4; i += THREADS) mask[i] = 0u;
  auto landed = [&](int s) -> bool {  // bounded
    const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&s_bar[s]);
    const int limit = a.wait_limit > 0 ? a.wait_limit : EK_WAIT;
    unsigned done = 0;
    for (int i = 0; i < limit && !done; ++i)
      asm volatile(
          "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t}\n"
          : "=r"(done)
          : "r"(bar)
          : "memory");
    return done != 0;
  };
  // (last warp) for each bin the number of borders below its left edge; borders and bins in units
  // where a channel spans [0, 1]
  if (warp == THREADS / 32 - 1) {
    const float level = a.tables->grid[lane & 15];
    const float edge = ((float)lane - 0.5f) * (1.0f / (EK_BINS - 1)) - 5.0e-4f;
    int cell = 0;
    for (int l = 0; l < 15; ++l) {
      const float here = __shfl_sync(0xffffffffu, level, l), next = __shfl_sync(0xffffffffu, level, l + 1);
      const float b = mode == TQ_KEYS_UNIFORM ? ((float)l + 0.5f) * (1.0f / 15.0f) : 0.25f * (here + next) + 0.5f;
      cell += b < edge ? 1 : 0;
    }
    // (above the last border: a huge one)
    const float here = __shfl_sync(0xffffffffu, level, cell), next = __shfl_sync(0xffffffffu, level, min(cell + 1, 15));
    s_bin[lane] = make_float4(here, next, __uint_as_float((uint32_t)cell), 0.0f);
  }
  bool lost = false;
  if (aligned)
    lost = !landed(seg);
  else
    __syncthreads();

  // ---- pass 1: sum in token order, extremes, group maxima -------------------------------------
  // The sum is a chain over all tokens: a segment's threads take it over from the segment before
  // (a named barrier for each hand-over), the first one adds up before anything else.
  const int t0 = seg * NT;
  auto sum_segment = [&]() {
    unsigned long long sum;
    W w[8], nx[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) nx[k] = ldw(t0 + k);
    if (seg == 0) {
      sum = ek_pack(-0.0f, -0.0f);  // (-0 + x is x, a first token of -0 included)
    } else {
      asm volatile("bar.sync %0, 128;" ::"r"(seg) : "memory");
      const float2 s = *(const float2*)&s_sum[2 * p];
      sum = ek_pack(s.x, s.y);
    }
#pragma unroll 2
    for (int i = 0; i < NT; i += 8) {
#pragma unroll
      for (int k = 0; k < 8; ++k) w[k] = nx[k];
#pragma unroll
      for (int k = 0; k < 8; ++k) nx[k] = ldw(t0 + (i + 8 + k) % NT);
#pragma unroll
      for (int k = 0; k < 8; ++k) sum = ek_add2(sum, ek_pack(lo_of(w[k]), hi_of(w[k])));
    }
    float a0, a1;
    ek_unpack(sum, a0, a1);
    *(float2*)&s_sum[2 * p] = make_float2(a0, a1);
    if (seg + 1 < SEG) asm volatile("bar.arrive %0, 128;" ::"r"(seg + 1) : "memory");
  };
  if (seg == 0 && mode == TQ_KEYS_NF4_ASYM) sum_segment();
  {
    W* gmax = (W*)img;  // [32 groups][64 pairs]
    if constexpr (F32) {
      float2 mn = make_float2(INFINITY, INFINITY), mx = make_float2(-INFINITY, -INFINITY), gm[GPT];
#pragma unroll
      for (int j = 0; j < GPT; ++j) gm[j] = make_float2(0.0f, 0.0f);
#pragma unroll 1
      for (int i = 0; i < NT; i += 8)
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float2 w = ldw(t0 + i + k);
          mn = make_float2(fminf(mn.x, w.x), fminf(mn.y, w.y));
          mx = make_float2(fmaxf(mx.x, w.x), fmaxf(mx.y, w.y));
          gm[k % GPT] = make_float2(fmaxf(gm[k % GPT].x, fabsf(w.x)), fmaxf(gm[k % GPT].y, fabsf(w.y)));
        }
#pragma unroll
      for (int j = 0; j < GPT; ++j) gmax[(seg * GPT + j) * 64 + p] = gm[j];
      *(float2*)&s_mn[seg * TQ_D + 2 * p] = mn;
      *(float2*)&s_mx[seg * TQ_D + 2 * p] = mx;
    } else {
      constexpr uint32_t PINF = BF ? 0x7F807F80u : 0x7C007C00u;
      uint32_t mn = PINF, mx = PINF | 0x80008000u, gm[GPT];  // (not a first token: it may be NaN)
#pragma unroll
      for (int j = 0; j < GPT; ++j) gm[j] = 0u;
#pragma unroll 1
      for (int i = 0; i < NT; i += 8)
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint32_t w = ldw(t0 + i + k);
          mn = min2_16<BF>(mn, w);
          mx = max2_16<BF>(mx, w);
          gm[k % GPT] = max2_16<BF>(gm[k % GPT], w & 0x7FFF7FFFu);
        }
#pragma unroll
      for (int j = 0; j < GPT; ++j) gmax[(seg * GPT + j) * 64 + p] = gm[j];
      *(float2*)&s_mn[seg * TQ_D + 2 * p] = make_float2(lo_of(mn), hi_of(mn));
      *(float2*)&s_mx[seg * TQ_D + 2 * p] = make_float2(lo_of(mx), hi_of(mx));
    }
  }
  if (seg > 0 && mode == TQ_KEYS_NF4_ASYM) sum_segment();
  if (__syncthreads_or(lost)) {
    // A copy did not arrive: nothing is encoded from rows that are not there.  The status word says
    // so, the page becomes an empty one (scales, zero-points and corrections of zero), and the
    // copies still on their way get another bounded wait before the CTA gives up its shared memory.
    if (tid == 0) {
      atomicOr(a.status, TQ_STATUS_WAIT_TIMEOUT);
      a.page_meta[unit_index(g, a.layer, seq, head) * g.max_blocks + blk] = {0u, 0u};
      for (int s = 0; s < SEG; ++s) landed(s);
    }
    auto zero = [&](int from, int to) {  // (multiples of 16, as all parts of a page are)
      for (int i = from + 16 * tid; i < to; i += 16 * THREADS) *(uint4*)(page + i) = make_uint4(0, 0, 0, 0);
    };
    zero(0, g.k_bytes);
    zero(g.scale_off, g.page_bytes);
    __syncthreads();
    return;
  }

  // ---- per channel: zero-point, scale, bin mapping, table; the groups with the k largest maxima ------
  // (a thread computes the zero-points and scales of the channels whose bins it fills: no barrier between)
  auto channel = [&](int d, float& mu, float& amax) {
    float xmin = s_mn[d], xmax = s_mx[d];
#pragma unroll
    for (int s = 1; s < SEG; ++s) {
      xmin = fminf(xmin, s_mn[s * TQ_D + d]);
      xmax = fmaxf(xmax, s_mx[s * TQ_D + d]);
    }
    mu = mode == TQ_KEYS_NF4_ASYM
             ? (a.bias_means != nullptr ? a.bias_means[((size_t)blk * g.n_kv_heads + head) * TQ_D + d]
                : a.tables->mean_mask[d] ? __fdiv_rn(s_sum[d], (float)EK_S)
                                         : 0.0f)
         : mode == TQ_KEYS_NF4 ? 0.0f
                               : xmin;
    // (rounding is monotone: the largest |fl(x - mu)| is reached at an extreme)
    amax = mode == TQ_KEYS_NF4_ASYM ? fmaxf(fabsf(__fsub_rn(xmax, mu)), fabsf(__fsub_rn(xmin, mu)))
                                    : fmaxf(fabsf(xmax), fabsf(xmin));
    amax = fmaxf(amax, 1e-8f);
    if (mode == TQ_KEYS_UNIFORM) amax = __fdiv_rn(fmaxf(__fsub_rn(xmax, xmin), 1e-8f), 15.0f);
  };
  auto fill = [&](int d, float mu, float sc, int from, int to) {
    uint32_t* col = tab + ek_col(d);
#pragma unroll 4
    for (int bin = from; bin < to; ++bin) {
      const float4 b4 = s_bin[bin];
      const uint32_t cell = __float_as_uint(b4.z);
      const float l2 = 0.5f * (__fmul_rn(sc, b4.x) + __fmul_rn(sc, b4.y));
      const float b = mode == TQ_KEYS_NF4 ? l2 : mu + l2;
      // (the nearest number whose low bits are the code)
      const int near16 = max((int)(__float_as_uint(b) & 0x7FFFFFFFu) + 8 - (int)cell, 0) & ~15;
      col[bin * TQ_D] = cell < 15u ? (__float_as_uint(b) & 0x80000000u) | (uint32_t)near16 | cell
                                   : 0x7F700000u | 15u;
    }
  };
  constexpr int FILL0 = F32 ? 10 : 22;  // bins of the threads that also store the channel's numbers
  if (tid < TQ_D) {
    const int d = tid;
    float mu, amax;
    channel(d, mu, amax);
    s_mu[d] = mu;
    s_scale[d] = amax;
    ((float*)(page + g.scale_off))[d] = amax;
    ((float*)(page + g.mean_off))[d] = mu;
    // s = (x - mu) / (2 amax) + 1/2, or (x - mu) / (15 amax) on the uniform grid, in [0, 1]
    const float inv = mode == TQ_KEYS_UNIFORM ? 1.0f / (15.0f * amax) : 0.5f / amax;
    s_inv[d] = inv;
    s_off[d] = (mode == TQ_KEYS_UNIFORM ? 0.0f : 0.5f) - mu * inv;
    // An element closer than this to a border is computed again.  The table holds the border with
    // its four low mantissa bits replaced (at most 8 ulp, 2^-20 of |border| <= |mu| + range) and
    // the reference's levels and distances round by an ulp each: 2^-19 of the sum covers both.
    // Where the range is tiny against the zero-point the levels themselves round together, and near
    // the top of float32's range (or beyond it: infinities, a NaN mean) borders and steps overflow:
    // everything again.
    const float range = mode == TQ_KEYS_UNIFORM ? 15.0f * amax : amax;
    const bool plain = range >= fabsf(mu) * (1.0f / 512.0f) && fabsf(mu) + range < 0x1p126f;
    s_tol[d] = plain ? (fabsf(mu) + range) * 0x1p-19f : INFINITY;
    fill(d, mu, amax, 0, FILL0);
  } else if (!F32 && tid < TQ_D + 64) {  // packed: a thread per channel pair
    const uint32_t* gm = (const uint32_t*)img + (tid - TQ_D);
    uint32_t top[EK_K];
#pragma unroll
    for (int j = 0; j < EK_K; ++j) top[j] = 0u;
#pragma unroll 8
    for (int i = 0; i < EK_GROUPS; ++i) {
      const uint32_t v = gm[i * 64];
      if (kk > 5) {
#pragma unroll
        for (int j = 0; j < 3; ++j) top[j] = min2_16<BF>(max2_16<BF>(v, top[j]), top[j + 1]);
      }
#pragma unroll
      for (int j = 3; j < EK_K - 1; ++j) top[j] = min2_16<BF>(max2_16<BF>(v, top[j]), top[j + 1]);
      top[EK_K - 1] = max2_16<BF>(v, top[EK_K - 1]);
    }
    uint32_t low = 0u;
#pragma unroll
    for (int j = 0; j < EK_K; ++j) low = j == EK_K - kk ? top[j] : low;
    uint32_t lo = 0u, hi = 0u;
#pragma unroll
    for (int i = 0; i < EK_GROUPS; ++i) ek_reach2<BF>(gm[i * 64], low, 1u << i, lo, hi);
    s_groups[2 * (tid - TQ_D)] = lo;
    s_groups[2 * (tid - TQ_D) + 1] = hi;
  } else if (F32 && tid < 2 * TQ_D) {
    const int d = tid - TQ_D;
    const float* gm = (const float*)img + d;  // [32][128]
    float top[EK_K];
#pragma unroll
    for (int j = 0; j < EK_K; ++j) top[j] = 0.0f;
#pragma unroll 4
    for (int i = 0; i < EK_GROUPS; ++i) {
      const float v = gm[i * TQ_D];
#pragma unroll
      for (int j = 0; j < EK_K - 1; ++j) top[j] = fminf(fmaxf(v, top[j]), top[j + 1]);
      top[EK_K - 1] = fmaxf(v, top[EK_K - 1]);
    }
    float low = 0.0f;
#pragma unroll
    for (int j = 0; j < EK_K; ++j) low = j == EK_K - kk ? top[j] : low;
    uint32_t sel = 0u;
#pragma unroll
    for (int i = 0; i < EK_GROUPS; ++i) sel |= gm[i * TQ_D] >= low ? 1u << i : 0u;
    s_groups[d] = sel;
  } else if (F32) {  // two threads a channel
    const int d = tid & (TQ_D - 1), half = (tid >> 7) & 1;
    float mu, amax;
    channel(d, mu, amax);
    fill(d, mu, amax, FILL0 + 11 * half, FILL0 + 11 * (half + 1));
  } else {  // a thread per two channels
#pragma unroll 1
    for (int d = tid - 192; d < TQ_D; d += 64) {
      float mu, amax;
      channel(d, mu, amax);
      fill(d, mu, amax, FILL0, EK_BINS);
    }
  }
  __syncthreads();

  // ---- pass 2: codes ----------------------------------------------------------------------------
  {
    const float inv0 = s_inv[2 * p], inv1 = s_inv[2 * p + 1], off0 = s_off[2 * p], off1 = s_off[2 * p + 1];
    const float tol0 = s_tol[2 * p], tol1 = s_tol[2 * p + 1];
    // the table's address for bin 0 of each channel as a denormal number, and 512 (a bin's
    // distance in bytes) likewise
    const uint32_t tab_addr = (uint32_t)__cvta_generic_to_shared(tab);
    const unsigned long long base2 = ek_pack(__uint_as_float(tab_addr + 4 * p), __uint_as_float(tab_addr + 256 + 4 * p));
    const unsigned long long step2 = ek_pack(__uint_as_float(TQ_D * 4), __uint_as_float(TQ_D * 4));
    const unsigned long long bins2 = ek_pack((float)(EK_BINS - 1), (float)(EK_BINS - 1));
    const unsigned long long magic2 = ek_pack(EK_MAGIC, EK_MAGIC), unmagic2 = ek_pack(-EK_MAGIC, -EK_MAGIC);
    uint8_t* out = img + t0 * (TQ_D / 2) + p;
#pragma unroll 1
    for (int c = 0; c < NT / 8; ++c) {
      float m0 = INFINITY, m1 = INFINITY;
      uint32_t code[8];
      W w[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) w[k] = ldw(t0 + 8 * c + k);
#pragma unroll
      for (int k = 0; k < 8; k += 2) {
        float x0[2], x1[2], d0[2], d1[2];
        uint32_t e0[2], e1[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          x0[j] = lo_of(w[k + j]);
          x1[j] = hi_of(w[k + j]);
          const float s0 = ek_fma_sat(x0[j], inv0, off0), s1 = ek_fma_sat(x1[j], inv1, off1);
          const unsigned long long n2 = ek_add2(ek_fma2(ek_pack(s0, s1), bins2, magic2), unmagic2);
          float a0, a1;
          ek_unpack(ek_fma2(n2, step2, base2), a0, a1);
          asm volatile("ld.shared.u32 %0, [%1];" : "=r"(e0[j]) : "r"(__float_as_uint(a0)));
          asm volatile("ld.shared.u32 %0, [%1];" : "=r"(e1[j]) : "r"(__float_as_uint(a1)));
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          d0[j] = x0[j] - __uint_as_float(e0[j]);
          d1[j] = x1[j] - __uint_as_float(e1[j]);
          // 1 above the border, 0 below it; both steps as bits 0 and 4 of an integer
          const float up0 = ek_fma_sat(d0[j], 0x1p120f, 0.0f), up1 = ek_fma_sat(d1[j], 0x1p120f, 0.0f);
          const uint32_t up = __float_as_uint(fmaf(up1, 16.0f, up0 + EK_MAGIC));
          const uint32_t e1s = e1[j] << 4;
          code[k + j] = ((e0[j] & 15u) | (e1s & ~15u)) + up;  // (the low byte)
        }
        m0 = ek_min_abs(m0, d0[0], d0[1]);
        m1 = ek_min_abs(m1, d1[0], d1[1]);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) out[(8 * c + k) * (TQ_D / 2)] = (uint8_t)code[k];
      // (not closer than the tolerance: a channel that is computed again as a whole has an infinite
      // one, and its minima may be infinite too)
      if (!(m0 > tol0) || !(m1 > tol1))
        redos[atomicAdd(&s_n_redo, 1)] = (unsigned short)(p | ((t0 / 8 + c) << 6));
    }
  }
  __syncthreads();

  // ---- elements close to a border; outliers -----------------------------------------------------
  // (meanwhile the last warp ranks the four widest channels)
  if (warp == THREADS / 32 - 1) {  // largest scale first, ties to the lower channel
    uint32_t key[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) key[i] = __float_as_uint(s_scale[4 * lane + i]);
    for (int r = 0; r < TQ_WIDE; ++r) {
      const uint32_t best = max(max(key[0], key[1]), max(key[2], key[3]));
      const uint32_t top = __reduce_max_sync(0xffffffffu, best);
      const int at = __ffs((int)__ballot_sync(0xffffffffu, best == top)) - 1;
      if (lane == at) {
        bool taken = false;
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (!taken && key[i] == top) {
            taken = true;
            key[i] = 0u;
            s_wide[r] = 4 * lane + i;
          }
      }
      __syncwarp();
    }
  }
  {
    // The reference's nearest level: the first minimum of the rounded distances.  An element
    // close to a border has one of the two levels beside it (the code found, or a neighbour);
    // where the levels themselves round together all sixteen are tried.  Channels near or beyond
    // the top of float32's range get the general encoder's two candidates of a bin, so that both
    // give them the same codes.
    auto exact_code = [&](float v, float mu, float sc, float tol, int c) -> int {
      if (mode == TQ_KEYS_UNIFORM) {
        const float qv = rintf(__fdiv_rn(__fsub_rn(v, mu), sc));  // ties to even, like np.round
        return (int)fminf(fmaxf(qv, 0.0f), 15.0f);
      }
      auto dist = [&](int l) -> float {
        const float sl = __fmul_rn(sc, s_grid[l]);
        return fabsf(__fsub_rn(v, mode == TQ_KEYS_NF4 ? sl : __fadd_rn(mu, sl)));
      };
      int l_lo = max(c - 1, 0), l_hi = min(c + 1, 15);
      if (isinf(tol)) {
        l_lo = 0;
        l_hi = 15;
        if (sc >= fabsf(mu) * (1.0f / 512.0f)) {
          const int bin = min(max(__float2int_rd(fmaf(v - mu, 32.0f / sc, 32.0f)), 0), 63);
          const float left = -1.0f + (float)bin * (1.0f / 32.0f) - 1.0e-4f;
          for (int l = 0; l < 15; ++l) l_lo += (0.5f * (s_grid[l] + s_grid[l + 1]) < left) ? 1 : 0;
          l_hi = min(l_lo + 1, 15);
        }
      }
      int best = l_lo;
      float bd = dist(l_lo);  // (a NaN stays: nothing is less)
      for (int l = l_lo + 1; l <= l_hi; ++l) {
        const float dv = dist(l);
        if (dv < bd) {
          bd = dv;
          best = l;
        }
      }
      return best;
    };
    // (a thread per token of a listed group: its two channels share a byte of the image)
    const int n_redo = s_n_redo * 8;
    for (int i = tid; i < n_redo; i += THREADS) {
      const int r = redos[i >> 3], rp = r & 63, t = (r >> 6) * 8 + (i & 7);
      const W w = ((const W*)rows)[t * 64 + rp];
      const int b = img[t * (TQ_D / 2) + rp];
      const int c0 = exact_code(lo_of(w), s_mu[2 * rp], s_scale[2 * rp], s_tol[2 * rp], b & 15);
      const int c1 = exact_code(hi_of(w), s_mu[2 * rp + 1], s_scale[2 * rp + 1], s_tol[2 * rp + 1], b >> 4);
      img[t * (TQ_D / 2) + rp] = (uint8_t)(c0 | (c1 << 4));
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // (the image is read by a bulk copy)
  if (kk > 0) {
    // NSUB threads a channel share the eight tokens of each of its groups; magnitudes as integers
    // (their bit patterns order like the numbers; a NaN is below all of them and never an outlier)
    constexpr int NSUB = THREADS / TQ_D, PER = 8 / NSUB;
    const int d = tid / NSUB, sub = tid % NSUB;
    constexpr int INF_BITS = F32 ? 0x7F800000 : BF ? 0x7F80 : 0x7C00;
    auto mag = [&](int t) -> int {
      int m;
      if constexpr (F32) m = (int)(((const uint32_t*)rows)[t * TQ_D + d] & 0x7FFFFFFFu);
      else m = ((const unsigned short*)rows)[t * TQ_D + d] & 0x7FFF;
      return m > INF_BITS ? -1 : m;
    };
    auto token = [&](int gi, int k) -> int { return gi / GPT * NT + gi % GPT + GPT * (sub + NSUB * k); };
    int top[EK_K];
#pragma unroll
    for (int j = 0; j < EK_K; ++j) top[j] = 0;
    auto insert = [&](int v) {
      if (kk > 5) {
#pragma unroll
        for (int j = 0; j < 3; ++j) top[j] = min(max(v, top[j]), top[j + 1]);
      }
#pragma unroll
      for (int j = 3; j < EK_K - 1; ++j) top[j] = min(max(v, top[j]), top[j + 1]);
      top[EK_K - 1] = max(v, top[EK_K - 1]);
    };
    const uint32_t sel = s_groups[d];
    for (uint32_t left = sel; left != 0u; left &= left - 1u) {
      const int gi = __ffs((int)left) - 1;
      int v[PER];
#pragma unroll
      for (int k = 0; k < PER; ++k) v[k] = mag(token(gi, k));
#pragma unroll
      for (int k = 0; k < PER; ++k) insert(v[k]);
    }
#pragma unroll
    for (int o = 1; o < NSUB; o <<= 1) {  // the threads of a channel merge their lists
      int other[EK_K];
#pragma unroll
      for (int j = 0; j < EK_K; ++j) other[j] = __shfl_xor_sync(0xffffffffu, top[j], o);
#pragma unroll
      for (int j = 0; j < EK_K; ++j)
        if (kk > 5 || j >= 3) insert(other[j]);
    }
    int kth = 0;
#pragma unroll
    for (int j = 0; j < EK_K; ++j) kth = j == EK_K - kk ? top[j] : kth;
    // every token's outlier channels as a bit mask
    for (uint32_t left = sel; left != 0u; left &= left - 1u) {
      const int gi = __ffs((int)left) - 1;
#pragma unroll
      for (int k = 0; k < PER; ++k) {
        const int t = token(gi, k);
        if (mag(t) >= kth) atomicOr(&mask[t * 4 + (d >> 5)], 1u << (d & 31));
      }
    }
  }
  __syncthreads();
  if (tid == THREADS - 1) {  // the code rows to the page
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(page),
                 "r"((uint32_t)__cvta_generic_to_shared(img)), "r"(C::IMG)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  }

  // The page's tail is put together in shared memory and stored as one piece: slots, counts and codes of
  // single tokens would be some forty scattered stores a warp.
  uint8_t* tail = (uint8_t*)s_mn;
  PageHeader* hdr = (PageHeader*)tail;
  if (tid < TQ_SIDE_OFF / 4) ((uint32_t*)tail)[tid] = 0u;
  else if (tid >= 64 && tid < 64 + TQ_OVF_CAP) ((uint32_t*)(tail + TQ_OVF_OFF))[tid - 64] = 0u;
  auto store_tail = [&]() {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(page + g.hdr_off),
                 "r"((uint32_t)__cvta_generic_to_shared(tail)), "r"(TQ_TAIL_BYTES)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  };
  // Exclusive prefix sums over the tokens of their outlier counts and of the counts beyond the
  // fixed slots (both in one word: each total stays below 65536); thread t owns token t.
  uint32_t mine = 0u, incl = 0u, m4[4] = {0u, 0u, 0u, 0u};
  int cnt = 0;
  if (tid < EK_S) {
    const uint4 m = *(const uint4*)&mask[tid * 4];
    m4[0] = m.x; m4[1] = m.y; m4[2] = m.z; m4[3] = m.w;
    cnt = __popc(m.x) + __popc(m.y) + __popc(m.z) + __popc(m.w);
    mine = (uint32_t)cnt | ((uint32_t)max(cnt - TQ_ELL_SLOTS, 0) << 16);
    incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t nv = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += nv;
    }
    if (lane == 31) s_scan[warp] = incl;
  }
  __syncthreads();
  int n_out = 0;
  {
    uint32_t sum = 0u;
#pragma unroll
    for (int w = 0; w < EK_S / 32; ++w) sum += s_scan[w];
    n_out = (int)(sum & 0xffffu);
  }
  // This page's slice of the (layer, seq, head) outlier slab.  (Its place is not waited for until the
  // page's own lists are written.)
  uint32_t pool_at = 0u;
  if (tid == THREADS - 32 && n_out > 0)
    pool_at = atomicAdd(&a.pool_cursor[unit_index(g, a.layer, seq, head)], (uint32_t)((n_out + 3) & ~3));
  auto take_slice = [&]() {
    uint32_t sum = 0u;
    for (int w = 0; w < EK_S / 32; ++w) sum += s_scan[w];
    const int n = n_out, n_ovf = (int)(sum >> 16);
    uint32_t off = pool_at;
    int alloc = 0;
    if (n > 0) {
      const int n4 = (n + 3) & ~3;
      if (off >= (uint32_t)g.pool_entries) off = 0;
      else alloc = min(n4, g.pool_entries - (int)off);
      if (alloc < n4) atomicOr(a.status, TQ_STATUS_POOL_OVERFLOW);
    }
    PageMeta pm;
    pm.off = off;
    pm.cnt = (uint32_t)min(n, alloc);
    a.page_meta[unit_index(g, a.layer, seq, head) * g.max_blocks + blk] = pm;
    hdr->off = pm.off;  // the page carries its own copy for the decode kernel
    hdr->cnt = pm.cnt;
    hdr->ovf_start[4] = (uint16_t)min(n_ovf, TQ_OVF_CAP);
    hdr->ovf_n = (uint16_t)min(n_ovf, TQ_OVF_CAP);
    // the in-page copy is complete unless the overflow list is too long or the pool slab could
    // not take every entry (then the pool's shorter list is the cache's content)
    hdr->flags = (n_ovf > TQ_OVF_CAP || alloc < n) ? TQ_PAGE_SPILLED : 0;
    s_off_pool = off;
    s_alloc = alloc;
  };
  uint16_t* ell_delta = (uint16_t*)(tail + TQ_ELL_OFF);  // [slot][token]
  uint8_t* ell_col = tail + TQ_ELL_COL_OFF;               // [slot][token]
  uint32_t* ovf = (uint32_t*)(tail + TQ_OVF_OFF);
  int row = 0;  // where this token's outliers start
  if (tid < EK_S) {
    uint32_t excl = incl - mine;
    for (int w = 0; w < warp; ++w) excl += s_scan[w];
    row = (int)(excl & 0xffffu);
    const int orow = (int)(excl >> 16);
    s_row[tid] = (unsigned short)row;
    s_orow[tid] = (unsigned short)orow;
    if ((tid & 63) == 0) hdr->ovf_start[tid >> 6] = (uint16_t)min(orow, TQ_OVF_CAP);
    // slots the token does not use hold a zero delta on channel 0
    for (int j = cnt; j < TQ_ELL_SLOTS; ++j) {
      ell_delta[j * 256 + tid] = 0;
      ell_col[j * 256 + tid] = 0;
    }
    // the codes of the widest channels a second time
    uint32_t side = 0u;
#pragma unroll
    for (int r = 0; r < TQ_WIDE; ++r) {
      const int d = s_wide[r];
      side |= (uint32_t)((img[tid * (TQ_D / 2) + (d >> 1)] >> (4 * (d & 1))) & 15) << (4 * r);
    }
    ((uint16_t*)(tail + TQ_SIDE_OFF))[tid] = (uint16_t)side;
  }
  if (tid < TQ_WIDE) hdr->wide[tid] = (uint8_t)s_wide[tid];
  // The outliers by token, then channel (the order of the reference's flat indices), listed in
  // shared memory and stored one per thread; in several rounds where there are more than fit.
  unsigned short* list = (unsigned short*)tab;  // token | channel << 8
  constexpr int LIST = C::TAB / 2;
  constexpr int PRE = 4;  // entries of a thread that are ready before the slice is known
  for (int base = 0; base < n_out; base += LIST) {
    if (base > 0) __syncthreads();
    if (cnt > 0) {
      int i = row - base;
#pragma unroll
      for (int w = 0; w < 4; ++w)
        for (uint32_t left = m4[w]; left != 0u; left &= left - 1u, ++i)
          if (i >= 0 && i < LIST) list[i] = (unsigned short)(tid | ((32 * w + __ffs((int)left) - 1) << 8));
    }
    __syncthreads();
    const int n = min(n_out - base, LIST);
    auto entry = [&](int i) -> uint2 {  // (the pool's two words); and to the page
      const int t = list[i] & 255, d = list[i] >> 8, slot = base + i, below = slot - (int)s_row[t];
      const float v = Elem<DT>::ld(rows, t * TQ_D + d);
      const int code = (img[t * (TQ_D / 2) + (d >> 1)] >> (4 * (d & 1))) & 15;
      const __half hv = __float2half_rn(v);
      const float sl = __fmul_rn(s_scale[d], s_grid[code]);  // the decoder's value of this position
      const float dense = mode == TQ_KEYS_NF4 ? sl : __fadd_rn(s_mu[d], sl);
      const __half delta = __float2half_rn(__fsub_rn(__half2float(hv), dense));
      const uint32_t ent = (uint32_t)__half_as_ushort(delta) | ((uint32_t)d << 16) | ((uint32_t)t << 24);
      if (below < TQ_ELL_SLOTS) {
        ell_delta[below * 256 + t] = __half_as_ushort(delta);
        ell_col[below * 256 + t] = (uint8_t)q_row(d);
      } else {
        const int oi = (int)s_orow[t] + below - TQ_ELL_SLOTS;
        if (oi < TQ_OVF_CAP) ovf[oi] = ent;
      }
      return make_uint2(ent, __half_as_ushort(hv));
    };
    uint2 pre[PRE];
#pragma unroll
    for (int j = 0; j < PRE; ++j)
      if (tid + j * THREADS < n) pre[j] = entry(tid + j * THREADS);
    if (base == 0) {
      if (tid == THREADS - 32) take_slice();
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncthreads();
      if (n_out <= PRE * THREADS && tid == THREADS - 1) store_tail();
    }
    const int alloc = s_alloc;
    const size_t slab = unit_index(g, a.layer, seq, head) * (size_t)g.pool_entries + s_off_pool + base;
    auto store = [&](int i, uint2 e) {
      if (base + i < alloc) {
        a.pool_dec[slab + i] = e.x;
        a.pool_val[slab + i] = (uint16_t)e.y;
      }
    };
#pragma unroll
    for (int j = 0; j < PRE; ++j)
      if (tid + j * THREADS < n) store(tid + j * THREADS, pre[j]);
    for (int i = tid + PRE * THREADS; i < n; i += THREADS) store(i, entry(i));
  }
  if (n_out == 0 || n_out > PRE * THREADS) {
    if (n_out == 0 && tid == THREADS - 32) take_slice();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (tid == THREADS - 1) store_tail();
  }
  if (tid == THREADS - 1)  // the image has been read before the CTA gives its shared memory back
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

template <int DT>
int launch_t(const EncodeArgs& a, int device, cudaStream_t st) {
  const tq_geom& g = a.g;
  static bool attr_set[16] = {};  // per device: the attribute belongs to the device's context
  if (!attr_set[device & 15]) {
    TQ_CUDA(cudaFuncSetAttribute(encode_keys_block_kernel<DT>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, Ek<DT>::SMEM));
    attr_set[device & 15] = true;
  }
  // whether every row of the caller's tensor starts on a 16-byte boundary (the ring's do)
  const int epc = 16 / elem_size(DT);
  const int aligned = ((uintptr_t)a.k & 15) == 0 && a.seq_stride % epc == 0 &&
                      a.tok_stride % epc == 0 && a.head_stride % epc == 0;
  const dim3 grid(a.max_new_blocks, g.n_kv_heads, a.seq_count);
  encode_keys_block_kernel<DT><<<grid, Ek<DT>::THREADS, Ek<DT>::SMEM, st>>>(a, aligned);
  return TQ_OK;
}

}  // namespace

bool tq_keys_block_form(const tq_geom& g) {
  return g.key_mode != TQ_KEYS_POLAR && g.block_tokens == EK_S && g.outlier_k <= EK_K &&
         g.hot_cap % EK_S == 0;
}

int tq_launch_encode_keys_block(const EncodeArgs& a, int device, cudaStream_t st) {
  switch (a.g.kv_dtype) {
    case TQ_F32: return launch_t<TQ_F32>(a, device, st);
    case TQ_F16: return launch_t<TQ_F16>(a, device, st);
    default: return launch_t<TQ_BF16>(a, device, st);
  }
}
