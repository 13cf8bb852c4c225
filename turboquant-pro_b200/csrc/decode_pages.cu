// Decode-on-codes attention to float32 accuracy for 256-token blocks and query groups the tensor-core
// kernel has no tile for (5, 6, 7 and 9 to 16 query heads per KV head), and for larger groups wherever
// the general-shape kernel is asked for.  The partials have the layout of decode_generic.cu and go
// through its combine kernel.
//
// The products run on mma.sync tiles (m16n8k16, eight query heads across) with every float32 operand
// split into two fp16 parts, x = hi + lo, good to 2^-23 of x.  Powers of two keep lo in fp16's range: a head's
// weights are scaled by their largest, a head's probabilities times norms by the strip's largest such
// product.  (By its largest norm alone, as this once was, lo and then hi drop out where a token with
// a small value dominates the softmax: 1.7e-2 of the output with 24 nats between the two.)  An operand
// that is itself a product is split before it is rounded.  hi * hi + hi * lo + lo * hi leaves out 2^-22 of a
// term at most.  The tensor cores cut sums off where float32 rounds them, so of the scores only hi * hi
// of 16 channels is summed there; these are added up in float32, and the small products have a sum of
// their own.  Scores are in units of log 2 (decode_generic.cuh).
// Distance from 64 bits, plain float32 multiply-adds / this, 24 caches of 700 and 3 000 tokens at seven heads:
// 4.8e-7 / 4.5e-7 and 6.2e-7 / 5.6e-7; queries three times as large 6.2e-7 / 5.7e-7 and 7.6e-7 / 7.4e-7; a
// token without a value 24 nats above the rest 1.65e-6 / 1.50e-6.
//
// Persistent CTAs of three groups of four warps, one CTA an SM.  The pages of all sequences, heads and
// head tiles form one list that is cut into equal shares, one per group, so ragged batches balance;
// where a share leaves a (sequence, head) the group writes a partial.  A warp takes a strip of 64 tokens
// of each page of the share and works on it alone, without barriers: it copies what it needs of the
// page (codes, scales, outlier slots; value codes, norms) into its own piece of shared memory with
// cp.async, the key half of the next page while it works on the values of this one and the other way
// round (loading them where they are used left the warps waiting most of the time).
//   weights  w = q * scale as B fragments of its own (a lane forms the 32 weights it holds), the
//            zero-points' share of the score beside them;
//   scores   a byte of codes (two channels) becomes the hi and lo pairs by one 8-byte look-up in a
//            table with a copy per lane of a half warp: no bank conflicts, no arithmetic;
//   softmax  once per strip, in registers: a lane has two heads of two tokens a tile;
//   values   probability times norm, split, goes from the score tile's layout to the value tile's by
//            8x8 transposes; two tokens' codes of a channel are one look-up, as above.
// Outliers come from the page's own list by token (four fixed slots, then the overflow entries).
//
// The uncompressed window follows, in splits of its own: rounds of 64 tokens, their rows copied into
// shared memory (stride padded by 16 bytes: a thread per token reads them without conflicts), two
// threads a token for the scores, a thread per channel for the values, in packed float32 multiply-adds.
#include "decode_generic.cuh"

namespace {

constexpr int DP_GROUPS = 3;
constexpr int DP_GTH = 128;          // threads of a group
constexpr int DP_THREADS = DP_GROUPS * DP_GTH;
constexpr int DP_GT = 8;             // query heads of a tile
constexpr int DP_S = 256;
constexpr int DP_STRIP = 64;         // tokens of a page a warp takes
constexpr int DP_HOT = 64;           // hot tokens per round
constexpr int DP_SROW = DP_HOT + 4;  // scores of a head
constexpr int DP_PROW = DP_GT + 4;   // floats per token of the probabilities
constexpr int DP_SEQS = TQ_PAGES_SEQS;

// A warp's strip of a page.
template <int VB>
struct alignas(16) DpStrip {
  uint8_t keys[DP_STRIP * TQ_D / 2];
  uint16_t delta[TQ_ELL_SLOTS][DP_STRIP];
  uint8_t col[TQ_ELL_SLOTS][DP_STRIP];
  float scale[4][36], mean[4][36];  // 32 channels a row (the pad spreads a lane's rows over the banks)
  PageHeader hdr;
  uint32_t ovf[TQ_OVF_CAP];
  uint8_t values[DP_STRIP * TQ_D * VB / 8];
  float norms[DP_STRIP];
};
struct DpHot {
  float s[DP_GT][DP_SROW];
  float p[DP_HOT][DP_PROW];
  alignas(16) uint8_t rows[DP_HOT * (TQ_D * 4 + 16)];
};

template <int VB>
struct DpShared {
  static constexpr int NV = VB == 4 ? 256 : 64;
  uint2 lutk[256][16], lutv[NV][16];  // (hi pair, lo pair) of two codes, a copy per lane mod 16
  union {
    DpStrip<VB> strip[4];
    DpHot hot;
  } group[DP_GROUPS];
  float corr[DP_GROUPS][4][32][DP_GT];  // per warp: outlier corrections of 32 tokens; the merge area
  float q[DP_GROUPS][TQ_D][DP_GT];      // row q_row(d): channel d
  float m[DP_GROUPS][4][DP_GT], l[DP_GROUPS][4][DP_GT], f[DP_GROUPS][DP_GT];
  float grid[16], cent[16];
  int cum[DP_SEQS + 1];                 // pages of the sequences before each one (a head tile's worth)
  int scan[DP_THREADS / 32], most[DP_THREADS / 32];
};

TQ_DEV unsigned long long dp_pack(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
TQ_DEV float2 dp_unpack(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
TQ_DEV unsigned long long dp_fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
TQ_DEV unsigned long long dp_mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

TQ_DEV unsigned long long dp_add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

TQ_DEV float dp_ld(const void* p, size_t i, int dt) {
  if (dt == TQ_F32) return ((const float*)p)[i];
  if (dt == TQ_F16) return __half2float(((const __half*)p)[i]);
  return __bfloat162float(((const __nv_bfloat16*)p)[i]);
}

TQ_DEV uint32_t dp_h2(float lo, float hi) {
  const __half2 h = __floats2half2_rn(lo, hi);
  return *(const uint32_t*)&h;
}
// a pair of floats as fp16 pairs, hi + lo
TQ_DEV void dp_split(float a, float b, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(a, b);
  const float2 f = __half22float2(h);
  hi = *(const uint32_t*)&h;
  lo = dp_h2(a - f.x, b - f.y);
}
// the same of a * x and b * y: lo takes what the products' rounding would drop, too
TQ_DEV void dp_split_products(float a, float x, float b, float y, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(a * x, b * y);
  const float2 f = __half22float2(h);
  hi = *(const uint32_t*)&h;
  lo = dp_h2(fmaf(a, x, -f.x), fmaf(b, y, -f.y));
}
TQ_DEV uint2 dp_lut(uint32_t addr) {  // (the tables never change: not volatile)
  uint2 v;
  asm("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
  return v;
}
TQ_DEV void dp_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1,
                   const float (&c)[4]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%10,%11,%12,%13};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]),
        "f"(c[2]), "f"(c[3]));
}
// d = a * b of one 16-deep step, the small products first: a sum that starts from zero and goes on in
// float32 registers
TQ_DEV void dp_product(float (&d)[4], const uint32_t (&ah)[4], const uint32_t (&al)[4],
                       const uint32_t (&bh)[2], const uint32_t (&bl)[2]) {
  const float zero[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  dp_mma(d, al, bh[0], bh[1], zero);
  dp_mma(d, ah, bl[0], bl[1], d);
  dp_mma(d, ah, bh[0], bh[1], d);
}
TQ_DEV uint32_t dp_transpose(uint32_t v) {  // of an 8x8 matrix of 16-bit elements, a row per four lanes
  uint32_t o;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(o) : "r"(v));
  return o;
}
// 2^(top - floor(log2 x)), the power of two that takes x to [2^top, 2^(top + 1)); and its inverse.  Zero,
// denormals, infinities and NaN count as the nearest ordinary exponent.
TQ_DEV float dp_lift(float x, int top, float& inverse) {
  const int e = min(max((int)(__float_as_uint(x) >> 23 & 255u), 32), 254);
  inverse = __int_as_float((e - top) << 23);
  return __int_as_float((254 + top - e) << 23);
}
TQ_DEV void dp_cp16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}
TQ_DEV void dp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

// sequences seq0 .. seq0 + n_seqs - 1 of the layer
template <int VB>
__global__ void __launch_bounds__(DP_THREADS, 1) decode_pages_kernel(DecodeArgs a, int seq0, int n_seqs) {
  constexpr int GT = DP_GT;
  constexpr int NP = GT / 2;          // pairs of heads
  constexpr int VGB = TQ_GROUP_TOK * TQ_D * VB / 8;
  extern __shared__ __align__(128) uint8_t dp_smem[];
  DpShared<VB>& sh = *(DpShared<VB>*)dp_smem;
  const tq_geom& g = a.g;
  const int tid = threadIdx.x, lane = tid & 31, gi = tid / DP_GTH, gtid = tid % DP_GTH, warp = gtid >> 5;
  const int r = lane >> 2, c = lane & 3;
  const int G = g.group, H = g.n_kv_heads, tiles = (G + GT - 1) / GT;
  auto group_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(1 + gi), "n"(DP_GTH) : "memory"); };
  float(*q_s)[GT] = sh.q[gi];

  // ---- tables, the list of pages ---------------------------------------------------------------
  if (tid < 16) {
    sh.grid[tid] = a.tables->grid[tid];
    sh.cent[tid] = a.tables->centroids[tid];
  }
  auto pages_of = [&](int s, int& b0) -> int {
    const int nb = n_cold_blocks(a.seq_len[a.layer * g.n_seqs + seq0 + s], g.hot_window, DP_S);
    b0 = min(a.block_begin, nb);
    return (a.block_end < 0 ? nb : min(a.block_end, nb)) - b0;
  };
  int most = 0;  // pages of the longest sequence
  {
    // thread t takes sequences t * per .. + per - 1: a scan over the threads
    const int per = (n_seqs + DP_THREADS - 1) / DP_THREADS;
    int sum = 0, b0;
    for (int s = tid * per; s < min((tid + 1) * per, n_seqs); ++s) {
      const int n = pages_of(s, b0);
      sh.cum[s + 1] = n;
      sum += n;
      most = max(most, n);
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    most = __reduce_max_sync(0xffffffffu, most);
    if (lane == 31) sh.scan[tid >> 5] = incl;
    if (lane == 0) sh.most[tid >> 5] = most;
    __syncthreads();
    int before = incl - sum;
    for (int w = 0; w < DP_THREADS / 32; ++w) {
      before += w < tid >> 5 ? sh.scan[w] : 0;
      most = max(most, sh.most[w]);
    }
    if (tid == 0) sh.cum[0] = 0;
    for (int s = tid * per; s < min((tid + 1) * per, n_seqs); ++s) {
      before += sh.cum[s + 1];
      sh.cum[s + 1] = before;
    }
  }
  float inv_k, inv_v;
  {  // entries scaled to below 2^8
    float max_k = 0.0f, max_v = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      max_k = fmaxf(max_k, fabsf(sh.grid[i]));
      max_v = fmaxf(max_v, fabsf(sh.cent[i]));
    }
    const float up_k = dp_lift(max_k, 7, inv_k), up_v = dp_lift(max_v, 7, inv_v);
    for (int e = tid; e < 256 + DpShared<VB>::NV; e += DP_THREADS) {
      uint2 w;
      uint4* dst;
      if (e < 256) {
        dp_split(sh.grid[e & 15] * up_k, sh.grid[e >> 4] * up_k, w.x, w.y);
        dst = (uint4*)sh.lutk[e];
      } else {
        const int b = e - 256;
        dp_split(sh.cent[b & (VB == 4 ? 15 : 7)] * up_v, sh.cent[b >> VB] * up_v, w.x, w.y);
        dst = (uint4*)sh.lutv[b];
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) dst[(i + lane) & 7] = make_uint4(w.x, w.y, w.x, w.y);
    }
  }
  __syncthreads();

  // A sequence with n pages has n pages in the list for each of its heads and head tiles ("rows" of n
  // pages).  Shares of `share` pages; a row meets at most (n - 2) / share + 2 of them, which has to fit its
  // ns_cold partials (at least two).
  const int rows_per_seq = H * tiles, n_groups = gridDim.x * DP_GROUPS;
  const long total = (long)sh.cum[n_seqs] * rows_per_seq;
  int share = (int)((total + n_groups - 1) / n_groups);
  share = max(share, a.ns_cold > 2 ? (most + a.ns_cold - 4) / (a.ns_cold - 2) : most);
  share = max(share, 1);

  // the query rows of a tile; `log2`: times the scores' unit
  auto load_q = [&](int unit, int gt, bool log2) {
    const int seq = unit / H, head = unit - seq * H;
#pragma unroll
    for (int gg = 0; gg < GT; ++gg) {
      const int qh = gt * GT + gg;
      const size_t at = ((size_t)seq * g.n_q_heads + head * G + qh) * TQ_D + gtid;
      const float x = qh < G ? dp_ld(a.q, at, a.q_dtype) : 0.0f;
      q_s[q_row(gtid)][gg] = log2 ? tq_scaled<true>(x) : x;
    }
  };
  auto slot_of = [&](int unit, int gt, int slot) -> float* {
    return a.partials + (((size_t)unit * g.max_splits + slot) * G + gt * GT) * TQ_PART_STRIDE;
  };
  auto mark_empty = [&](int unit, int gt, int first, int end) {  // partials without sums (a sum below zero says so)
    for (int i = gtid; i < (end - first) * GT; i += DP_GTH)
      if (gt * GT + i % GT < G) {
        float* pp = slot_of(unit, gt, first + i / GT) + (i % GT) * TQ_PART_STRIDE;
        pp[0] = -INFINITY;
        pp[1] = -1.0f;
      }
  };
  if (a.ns_cold > 0)
    for (int s = blockIdx.x * DP_GROUPS + gi; s < n_seqs; s += n_groups)
      if (sh.cum[s + 1] == sh.cum[s])
        for (int row = 0; row < rows_per_seq; ++row)
          mark_empty((seq0 + s) * H + row / tiles, row % tiles, 0, a.ns_cold);

  // ---- cold pages -----------------------------------------------------------------------------
  // a page of the list: sequence, row, page of the row, pages of the row
  struct Pos {
    int seq, row, page, n;
  };
  auto advance = [&](Pos& p) {  // to the next page
    if (++p.page < p.n) return;
    p.page = 0;
    if (++p.row < rows_per_seq) return;
    p.row = 0;
    do {
      ++p.seq;
    } while (p.seq < n_seqs && sh.cum[p.seq + 1] == sh.cum[p.seq]);
    p.n = p.seq < n_seqs ? sh.cum[p.seq + 1] - sh.cum[p.seq] : 1;
  };
  const uint32_t lutk = (uint32_t)__cvta_generic_to_shared(&sh.lutk[0][lane & 15]);
  const uint32_t lutv = (uint32_t)__cvta_generic_to_shared(&sh.lutv[0][lane & 15]);
  DpStrip<VB>& st = sh.group[gi].strip[warp];
  float(*corr)[GT] = sh.corr[gi][warp];
  const int t0 = DP_STRIP * warp;  // first token of this warp's strip

  auto page_at = [&](const Pos& p) -> const uint8_t* {
    int b0;
    pages_of(p.seq, b0);
    return a.pages + page_offset(g, a.layer, seq0 + p.seq, p.row / tiles, b0 + p.page);
  };
  auto copy_keys = [&](const uint8_t* page) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      dp_cp16(st.keys + (32 * i + lane) * 16, page + t0 * (TQ_D / 2) + (32 * i + lane) * 16);
    const uint8_t* ed = page + g.hdr_off + TQ_ELL_OFF;      // 8 pieces a slot
    const uint8_t* ec = page + g.hdr_off + TQ_ELL_COL_OFF;  // 4 pieces a slot
    dp_cp16((uint8_t*)st.delta + lane * 16, ed + (lane >> 3) * (DP_S * 2) + t0 * 2 + (lane & 7) * 16);
    if (lane < 16) dp_cp16((uint8_t*)st.col + lane * 16, ec + (lane >> 2) * DP_S + t0 + (lane & 3) * 16);
    dp_cp16(&st.scale[lane >> 3][(lane & 7) * 4], page + g.scale_off + lane * 16);
    dp_cp16(&st.mean[lane >> 3][(lane & 7) * 4], page + g.mean_off + lane * 16);
    if (lane < 4) dp_cp16((uint8_t*)&st.hdr + lane * 16, page + g.hdr_off + lane * 16);
    else dp_cp16(st.ovf + (lane - 4) * 4, page + g.hdr_off + TQ_OVF_OFF + (lane - 4) * 16);
  };
  auto copy_values = [&](const uint8_t* page) {
    const uint8_t* src = page + g.v_off + (size_t)(t0 / TQ_GROUP_TOK) * VGB;
#pragma unroll
    for (int i = 0; i < 4 * VGB / 512; ++i)
      dp_cp16(st.values + (32 * i + lane) * 16, src + (32 * i + lane) * 16);
    if (lane < 16) dp_cp16(st.norms + lane * 4, page + g.norm_off + t0 * 4 + lane * 16);
  };
  static_assert(sizeof(PageHeader) == 64 && TQ_OVF_CAP * 4 == 28 * 16, "pieces of the tail");

  // this lane's heads are 2 c and 2 c + 1, its channels 16 mt + r and 16 mt + r + 8
  float acc[8][4], m_run[2], l_run[2];
  auto reset = [&]() {
#pragma unroll
    for (int mt = 0; mt < 8; ++mt)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[mt][i] = 0.0f;
    m_run[0] = m_run[1] = -INFINITY;
    l_run[0] = l_run[1] = 0.0f;
  };
  // the four warps' states become one partial
  auto flush = [&](int unit, int gt, int slot) {
#pragma unroll
    for (int x = 0; x < 2; ++x) {
#pragma unroll
      for (int o = 4; o <= 16; o <<= 1) l_run[x] += __shfl_xor_sync(0xffffffffu, l_run[x], o);
      if (r == 0) {
        sh.m[gi][warp][2 * c + x] = m_run[x];
        sh.l[gi][warp][2 * c + x] = l_run[x];
      }
    }
    group_sync();  // (and every warp is done with its corrections: the sums take their place)
    float f[2];
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      float M = -INFINITY;
#pragma unroll
      for (int w = 0; w < 4; ++w) M = fmaxf(M, sh.m[gi][w][2 * c + x]);
      f[x] = m_run[x] > -INFINITY ? tq_exp2(m_run[x] - M) : 0.0f;
    }
    float* sums = &sh.corr[gi][0][0][0];  // [8 heads][128], bits 3 and 4 of the channel by the head
    for (int w = 0; w < 4; ++w) {
      if (warp == w) {
#pragma unroll
        for (int mt = 0; mt < 8; ++mt)
#pragma unroll
          for (int y = 0; y < 2; ++y)
#pragma unroll
            for (int x = 0; x < 2; ++x) {
              float* at = &sums[(2 * c + x) * TQ_D + ((16 * mt + 8 * y + r) ^ (8 * c))];
              const float v = acc[mt][2 * y + x] * f[x];
              *at = w == 0 ? v : *at + v;
            }
      }
      group_sync();
    }
    float* pp = slot_of(unit, gt, slot);
#pragma unroll
    for (int gg = 0; gg < GT; ++gg)
      if (gt * GT + gg < G) pp[gg * TQ_PART_STRIDE + 2 + gtid] = sums[gg * TQ_D + (gtid ^ (8 * (gg >> 1)))];
    if (gtid < GT && gt * GT + gtid < G) {
      float M = -INFINITY, L = 0.0f;
#pragma unroll
      for (int w = 0; w < 4; ++w) M = fmaxf(M, sh.m[gi][w][gtid]);
#pragma unroll
      for (int w = 0; w < 4; ++w)
        L += sh.m[gi][w][gtid] > -INFINITY ? sh.l[gi][w][gtid] * tq_exp2(sh.m[gi][w][gtid] - M) : 0.0f;
      pp[gtid * TQ_PART_STRIDE] = M;
      pp[gtid * TQ_PART_STRIDE + 1] = L;
    }
  };

  // (neighbouring shares go to different SMs: where there are few, each has one to itself)
  const int me = gi * gridDim.x + blockIdx.x;
  const long n_shares = a.ns_cold > 0 ? (total + share - 1) / share : 0;
  for (long k = me; k < n_shares; k += n_groups) {
    const long lo = k * share;
    const int count = (int)min((long)share, total - lo);
    Pos p;
    {  // the sequence that holds page lo of the list: the last one that starts at or before it
      int x = 0, y = n_seqs - 1;
      while (x < y) {
        const int mid = (x + y + 1) >> 1;
        if ((long)sh.cum[mid] * rows_per_seq <= lo) x = mid;
        else y = mid - 1;
      }
      p.seq = x;
      p.n = sh.cum[x + 1] - sh.cum[x];
      const int rem = (int)(lo - (long)sh.cum[x] * rows_per_seq);
      p.row = rem / p.n;
      p.page = rem - p.row * p.n;
    }
    {
      const uint8_t* page = page_at(p);
      copy_keys(page);
      dp_commit();
      copy_values(page);
      dp_commit();
    }
    bool fresh = true;  // the row's query has to be loaded
    for (int i = 0; i < count; ++i) {
      const int unit = (seq0 + p.seq) * H + p.row / tiles, gt = p.row % tiles;
      if (fresh) {
        group_sync();  // (the queries and sums of the row before are no longer read)
        load_q(unit, gt, true);
        reset();
        group_sync();
        fresh = false;
      }
      Pos next = p;
      advance(next);
      const uint8_t* next_page = i + 1 < count ? page_at(next) : nullptr;

      asm volatile("cp.async.wait_group 1;" ::: "memory");  // the key half has landed
      __syncwarp();
      // weights: k-step j takes channels 32 c + 4 j .. + 3 of this lane, column r is head r
      uint32_t bh[8][2], bl[8][2];
      float bias2[2], inv2[2];
      {
        float w[8][4], mx = 0.0f;
        float4 b4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 s4 = *(const float4*)&st.scale[c][4 * j], m4 = *(const float4*)&st.mean[c][4 * j];
          const int d = 32 * c + 4 * j;
          const float q0 = q_s[q_row(d)][r], q1 = q_s[q_row(d + 1)][r], q2 = q_s[q_row(d + 2)][r],
                      q3 = q_s[q_row(d + 3)][r];
          w[j][0] = q0 * s4.x, w[j][1] = q1 * s4.y, w[j][2] = q2 * s4.z, w[j][3] = q3 * s4.w;
          b4.x += q0 * m4.x, b4.y += q1 * m4.y, b4.z += q2 * m4.z, b4.w += q3 * m4.w;
#pragma unroll
          for (int x = 0; x < 4; ++x) mx = fmaxf(mx, fabsf(w[j][x]));
        }
        float bias = (b4.x + b4.y) + (b4.z + b4.w);
        bias += __shfl_xor_sync(0xffffffffu, bias, 1);
        bias += __shfl_xor_sync(0xffffffffu, bias, 2);
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        float inv;
        const float up = dp_lift(mx, 13, inv);
        inv *= inv_k;
#pragma unroll
        for (int x = 0; x < 2; ++x) {  // of heads 2 c + x
          bias2[x] = __shfl_sync(0xffffffffu, bias, 8 * c + 4 * x);
          inv2[x] = __shfl_sync(0xffffffffu, inv, 8 * c + 4 * x);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 s4 = *(const float4*)&st.scale[c][4 * j];  // (again: w is rounded)
          const int d = 32 * c + 4 * j;
          dp_split_products(q_s[q_row(d)][r] * up, s4.x, q_s[q_row(d + 1)][r] * up, s4.y, bh[j][0], bl[j][0]);
          dp_split_products(q_s[q_row(d + 2)][r] * up, s4.z, q_s[q_row(d + 3)][r] * up, s4.w, bh[j][1], bl[j][1]);
        }
      }

      float s[4][4];  // tile h: (token r, heads 2 c, 2 c + 1), (token r + 8, ...)
      const bool spilled = (st.hdr.flags & TQ_PAGE_SPILLED) != 0;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        {  // outlier corrections of 32 tokens, a lane per token
          const int tok = 32 * half + lane;  // of the strip
          float e8[GT];
#pragma unroll
          for (int x = 0; x < GT; ++x) e8[x] = 0.0f;
          auto add = [&](float delta, int row) {
            const float4 qa = *(const float4*)&q_s[row][0], qb = *(const float4*)&q_s[row][4];
            e8[0] += qa.x * delta, e8[1] += qa.y * delta, e8[2] += qa.z * delta, e8[3] += qa.w * delta;
            e8[4] += qb.x * delta, e8[5] += qb.y * delta, e8[6] += qb.z * delta, e8[7] += qb.w * delta;
          };
          if (g.outlier_k > 0 && !spilled) {
#pragma unroll
            for (int j = 0; j < TQ_ELL_SLOTS; ++j)
              add(__half2float(__ushort_as_half(st.delta[j][tok])), st.col[j][tok]);
          }
          __syncwarp();  // (the tiles of the half before have been read)
          *(float4*)&corr[lane][0] = make_float4(e8[0], e8[1], e8[2], e8[3]);
          *(float4*)&corr[lane][4] = make_float4(e8[4], e8[5], e8[6], e8[7]);
          __syncwarp();
          if (g.outlier_k > 0) {
            // the rest of the list, ordered by token: the lane with a token's first entry adds up all of
            // them, so the sum does not depend on timing
            const uint32_t* list = st.ovf;
            int e0 = st.hdr.ovf_start[warp], e1 = st.hdr.ovf_start[warp + 1];
            if (spilled) {
              const size_t slab = unit_index(g, a.layer, seq0 + p.seq, p.row / tiles) * (size_t)g.pool_entries;
              list = a.pool_dec + slab + st.hdr.off;
              e0 = 0, e1 = (int)st.hdr.cnt;
            }
            for (int e = e0 + lane; e < e1; e += 32) {
              uint32_t v = list[e];
              const int tk = (int)(v >> 24);
              if (tk >> 5 != (t0 >> 5) + half || (e > e0 && (int)(list[e - 1] >> 24) == tk)) continue;
#pragma unroll
              for (int x = 0; x < GT; ++x) e8[x] = corr[tk & 31][x];
              for (int j = e;;) {
                add(__half2float(__ushort_as_half((unsigned short)(v & 0xffffu))),
                    q_row((v >> 16) & 127));
                if (++j >= e1) break;
                v = list[j];
                if ((int)(v >> 24) != tk) break;
              }
#pragma unroll
              for (int x = 0; x < GT; ++x) corr[tk & 31][x] = e8[x];
            }
            __syncwarp();
          }
        }
#pragma unroll
        for (int h2 = 0; h2 < 2; ++h2) {
          const int h = 2 * half + h2;
          uint32_t kw[2][4];
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const uint4 v = *(const uint4*)(st.keys + (16 * h + 8 * x + r) * (TQ_D / 2) + c * 16);
            kw[x][0] = v.x, kw[x][1] = v.y, kw[x][2] = v.z, kw[x][3] = v.w;
          }
          // hi * hi a step at a time, the products with a low part in one sum of their own
          float sum[2][4], low[4] = {0.0f, 0.0f, 0.0f, 0.0f};
          const float zero[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            uint32_t ah[4], al[4];
#pragma unroll
            for (int x = 0; x < 4; ++x) {  // tokens r, r + 8; bytes 2 j, 2 j + 1
              const uint32_t b = __byte_perm(kw[x & 1][j >> 1], 0, 0x4440 + 2 * (j & 1) + (x >> 1));
              const uint2 t = dp_lut(lutk + b * 128);
              ah[x] = t.x, al[x] = t.y;
            }
            float d[4];
            dp_mma(d, ah, bh[j][0], bh[j][1], zero);
            dp_mma(low, al, bh[j][0], bh[j][1], low);
            dp_mma(low, ah, bl[j][0], bl[j][1], low);
#pragma unroll
            for (int x = 0; x < 4; ++x) sum[j & 1][x] = j < 2 ? d[x] : sum[j & 1][x] + d[x];
          }
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const float2 e2 = *(const float2*)&corr[16 * h2 + 8 * x + r][2 * c];
            s[h][2 * x] = fmaf(sum[0][2 * x] + (sum[1][2 * x] + low[2 * x]), inv2[0], bias2[0]) + e2.x;
            s[h][2 * x + 1] = fmaf(sum[0][2 * x + 1] + (sum[1][2 * x + 1] + low[2 * x + 1]), inv2[1], bias2[1]) + e2.y;
          }
        }
      }
      __syncwarp();  // the key half has been read
      if (next_page != nullptr) copy_keys(next_page);
      dp_commit();
      asm volatile("cp.async.wait_group 1;" ::: "memory");  // the value half has landed
      __syncwarp();

      // softmax over the strip, times the norms; a head's largest product sets the scale of its column of
      // the value operand (the largest norm would not do: the probability in front of it may be
      // any amount smaller, where a token of another strip dominates)
      float nv[4][2], f[2], up_n[2], inv_n[2];
#pragma unroll
      for (int h = 0; h < 4; ++h)
#pragma unroll
        for (int x = 0; x < 2; ++x) nv[h][x] = st.norms[16 * h + 8 * x + r];
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        float mx = -INFINITY;
#pragma unroll
        for (int h = 0; h < 4; ++h) mx = fmaxf(mx, fmaxf(s[h][x], s[h][2 + x]));
#pragma unroll
        for (int o = 4; o <= 16; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float m_new = fmaxf(m_run[x], mx);
        const bool any = m_new > -INFINITY;
        f[x] = any ? tq_exp2(m_run[x] - m_new) : 1.0f;
        float sum = 0.0f, most = 0.0f;
#pragma unroll
        for (int h = 0; h < 4; ++h)
#pragma unroll
          for (int y = 0; y < 2; ++y) {
            const float e = any ? tq_exp2(s[h][2 * y + x] - m_new) : 0.0f;
            sum += e;
            s[h][2 * y + x] = e;
            most = fmaxf(most, fabsf(e * nv[h][y]));
          }
#pragma unroll
        for (int o = 4; o <= 16; o <<= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
        up_n[x] = dp_lift(most, 13, inv_n[x]);
        inv_n[x] *= inv_v;
        l_run[x] = l_run[x] * f[x] + sum;
        m_run[x] = m_new;
      }
#pragma unroll
      for (int mt = 0; mt < 8; ++mt) {
        acc[mt][0] *= f[0], acc[mt][1] *= f[1];
        acc[mt][2] *= f[0], acc[mt][3] *= f[1];
      }

#pragma unroll
      for (int h = 0; h < 4; ++h) {
        uint32_t ph[2], pl[2];
#pragma unroll
        for (int x = 0; x < 2; ++x) {  // tokens 0-7, 8-15 of the tile
          uint32_t hi, lo2;
          dp_split_products(s[h][2 * x] * up_n[0], nv[h][x], s[h][2 * x + 1] * up_n[1], nv[h][x], hi, lo2);
          ph[x] = dp_transpose(hi);
          pl[x] = dp_transpose(lo2);
        }
        const uint8_t* grp = st.values + h * VGB;
        uint32_t rec[9];
        if (VB == 4) {
          const uint4 x = *(const uint4*)(grp + lane * 16), y = *(const uint4*)(grp + 512 + lane * 16);
          rec[0] = x.x, rec[1] = x.y, rec[2] = x.z, rec[3] = x.w;
          rec[4] = y.x, rec[5] = y.y, rec[6] = y.z, rec[7] = y.w;
        } else {
#pragma unroll
          for (int x = 0; x < 3; ++x) {
            const uint2 v = *(const uint2*)(grp + 256 * x + lane * 8);
            rec[2 * x] = v.x, rec[2 * x + 1] = v.y;
          }
          rec[6] = 0u;
        }
#pragma unroll
        for (int mt = 0; mt < 8; ++mt) {
          uint32_t ah[4], al[4];
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            // channels r, r + 8; tokens 0-7, 8-15: pairs 4 mt, 4 mt + 2, 4 mt + 1, 4 mt + 3 of the record
            const int pr = 4 * mt + 2 * (x & 1) + (x >> 1);
            uint32_t at;
            if (VB == 4) {
              at = __byte_perm(rec[pr >> 2], 0, 0x4440 + (pr & 3)) * 128u;
            } else {  // the 6-bit field at bit 6 pr, moved to bits 7 .. 12
              const int bit = 6 * pr, wd = bit >> 5, b = bit & 31;
              const uint32_t v = b < 7    ? rec[wd] << (7 - b)
                                 : b > 26 ? __funnelshift_r(rec[wd], rec[wd + 1], b - 7)
                                          : rec[wd] >> (b - 7);
              at = v & 0x1f80u;
            }
            const uint2 t = dp_lut(lutv + at);
            ah[x] = t.x, al[x] = t.y;
          }
          float d[4];
          dp_product(d, ah, al, ph, pl);
#pragma unroll
          for (int x = 0; x < 4; ++x) acc[mt][x] = fmaf(d[x], inv_n[x & 1], acc[mt][x]);
        }
      }
      __syncwarp();  // the value half has been read
      if (next_page != nullptr) copy_values(next_page);
      dp_commit();

      if (next.page == 0 || i + 1 == count) {  // the share leaves the row, or ends
        const long row0 = (long)sh.cum[p.seq] * rows_per_seq + (long)p.row * p.n;  // the row's first page
        const int slot = (int)(k - row0 / share);
        flush(unit, gt, slot);
        if (next.page == 0) mark_empty(unit, gt, slot + 1, a.ns_cold);
        fresh = true;
      }
      p = next;
    }
  }

  // ---- the uncompressed window -------------------------------------------------------------------
  asm volatile("cp.async.wait_all;" ::: "memory");
  DpHot& ht = sh.group[gi].hot;
  const int dt = g.kv_dtype, esz = elem_size(dt), row_bytes = TQ_D * esz, row_step = row_bytes + 16;
  // (the splits start with the groups that have the least of the pages)
  for (int item = n_groups - 1 - me; item < n_seqs * rows_per_seq * a.ns_hot; item += n_groups) {
    const int split = item % a.ns_hot, row = item / a.ns_hot % rows_per_seq;
    const int seq = seq0 + item / a.ns_hot / rows_per_seq, head = row / tiles, gt = row % tiles;
    const int unit = seq * H + head;
    const int N = a.seq_len[a.layer * g.n_seqs + seq];
    const int hot_start = n_cold_blocks(N, g.hot_window, DP_S) * DP_S;
    const int hot_len = a.with_hot ? N - hot_start : 0;
    const int ng = (hot_len + TQ_GROUP_TOK - 1) / TQ_GROUP_TOK;
    const int t_lo = (int)((long)ng * split / a.ns_hot) * TQ_GROUP_TOK;
    const int t_hi = min((int)((long)ng * (split + 1) / a.ns_hot) * TQ_GROUP_TOK, hot_len);
    if (t_lo >= t_hi) {
      mark_empty(unit, gt, a.ns_cold + split, a.ns_cold + split + 1);
      continue;
    }
    const size_t ring = hot_offset_elems(g, a.layer, seq, head) * esz;
    const int slot0 = (hot_start + t_lo) % g.hot_cap;
    // rows [t, t + n) of a ring into shared memory
    auto copy_rows = [&](const void* from, int t, int n) {
      const int pieces = row_bytes / 16;
      for (int i = gtid; i < n * pieces; i += DP_GTH) {
        const int x = i / pieces, pc = i - x * pieces;
        int slot = slot0 + (t - t_lo) + x;
        while (slot >= g.hot_cap) slot -= g.hot_cap;
        dp_cp16(ht.rows + x * row_step + pc * 16, (const uint8_t*)from + ring + (size_t)slot * row_bytes + pc * 16);
      }
    };
    group_sync();  // (what the group did before in this memory is over)
    copy_rows(a.hot_k, t_lo, min(DP_HOT, t_hi - t_lo));
    load_q(unit, gt, false);  // (products of 16-bit numbers are exact: the sum is scaled)
    float m_h[2], l_h[2];  // of heads 2 warp + i, the same in every lane
    unsigned long long av[NP];  // channel gtid
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      m_h[i] = -INFINITY;
      l_h[i] = 0.0f;
    }
#pragma unroll
    for (int x = 0; x < NP; ++x) av[x] = 0ull;
    for (int t = t_lo; t < t_hi; t += DP_HOT) {
      const int n_tok = min(DP_HOT, t_hi - t);
      asm volatile("cp.async.wait_all;" ::: "memory");
      group_sync();
      {  // scores: thread (token, four heads)
        const int tok = gtid & (DP_HOT - 1), h4 = gtid / DP_HOT * 4;
        if (tok < n_tok) {
          const uint8_t* kr = ht.rows + tok * row_step;
          unsigned long long dot[2] = {0ull, 0ull}, low[2] = {0ull, 0ull}, sub[2];
#pragma unroll 2
          for (int d0 = 0; d0 < TQ_D; d0 += 8) {
            float kv[8];
            if (dt == TQ_F32) {
              const float4 x = *(const float4*)(kr + 4 * d0), y = *(const float4*)(kr + 4 * d0 + 16);
              kv[0] = x.x; kv[1] = x.y; kv[2] = x.z; kv[3] = x.w;
              kv[4] = y.x; kv[5] = y.y; kv[6] = y.z; kv[7] = y.w;
            } else {
              const uint4 x = *(const uint4*)(kr + 2 * d0);
              const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                if (dt == TQ_F16) {
                  const float2 e = __half22float2(*(const __half2*)&w[i]);
                  kv[2 * i] = e.x; kv[2 * i + 1] = e.y;
                } else {
                  kv[2 * i] = __uint_as_float(w[i] << 16);
                  kv[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
                }
              }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const unsigned long long k2 = dp_pack(kv[i], kv[i]);
              const ulonglong2 qv = *(const ulonglong2*)&q_s[q_row(d0 + i)][h4];
              sub[0] = i == 0 ? dp_mul2(k2, qv.x) : dp_fma2(k2, qv.x, sub[0]);
              sub[1] = i == 0 ? dp_mul2(k2, qv.y) : dp_fma2(k2, qv.y, sub[1]);
            }
#pragma unroll
            for (int x = 0; x < 2; ++x) {
              if (d0 == TQ_D / 2) {  // (the halves add up separately)
                low[x] = dot[x];
                dot[x] = 0ull;
              }
              dot[x] = dp_add2(dot[x], sub[x]);
            }
          }
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const float2 e = dp_unpack(dp_add2(low[x], dot[x]));
            ht.s[h4 + 2 * x][tok] = tq_scaled<true>(e.x);
            ht.s[h4 + 2 * x + 1][tok] = tq_scaled<true>(e.y);
          }
        }
      }
      group_sync();
      copy_rows(a.hot_v, t, n_tok);  // (over the keys)
#pragma unroll
      for (int i = 0; i < 2; ++i) {  // softmax: a warp takes two heads
        const int gg = warp * 2 + i;
        float sc[2], mx = -INFINITY;
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          sc[x] = lane + 32 * x < n_tok ? ht.s[gg][lane + 32 * x] : -INFINITY;
          mx = fmaxf(mx, sc[x]);
        }
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float m_new = fmaxf(m_h[i], mx);
        const bool any = m_new > -INFINITY;
        const float fo = any ? tq_exp2(m_h[i] - m_new) : 1.0f;
        float sum = 0.0f;
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          const float pv = any && lane + 32 * x < n_tok ? tq_exp2(sc[x] - m_new) : 0.0f;
          sum += pv;
          ht.p[lane + 32 * x][gg] = pv;
        }
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        l_h[i] = l_h[i] * fo + sum;
        m_h[i] = m_new;
        if (lane == 0) sh.f[gi][gg] = fo;
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      group_sync();
#pragma unroll
      for (int x = 0; x < NP; ++x)
        av[x] = dp_mul2(av[x], dp_pack(sh.f[gi][2 * x], sh.f[gi][2 * x + 1]));
      for (int tb = 0; tb < n_tok; tb += 8) {  // eight tokens, then their sum
        unsigned long long sub[NP];
#pragma unroll
        for (int x = 0; x < NP; ++x) sub[x] = 0ull;
#pragma unroll
        for (int y = 0; y < 8; ++y) {
          if (tb + y < n_tok) {
            const float v = dp_ld(ht.rows + (tb + y) * row_step, gtid, dt);
            const unsigned long long v2 = dp_pack(v, v);
#pragma unroll
            for (int x = 0; x < NP; x += 2) {
              const ulonglong2 pv = *(const ulonglong2*)&ht.p[tb + y][2 * x];
              sub[x] = dp_fma2(v2, pv.x, sub[x]);
              sub[x + 1] = dp_fma2(v2, pv.y, sub[x + 1]);
            }
          }
        }
#pragma unroll
        for (int x = 0; x < NP; ++x) av[x] = dp_add2(av[x], sub[x]);
      }
      group_sync();  // the rows, probabilities and factors have been read
      if (t + DP_HOT < t_hi) copy_rows(a.hot_k, t + DP_HOT, min(DP_HOT, t_hi - t - DP_HOT));
    }
    float* pp = slot_of(unit, gt, a.ns_cold + split);
#pragma unroll
    for (int x = 0; x < NP; ++x) {
      const float2 v = dp_unpack(av[x]);
      if (gt * GT + 2 * x < G) pp[(2 * x) * TQ_PART_STRIDE + 2 + gtid] = v.x;
      if (gt * GT + 2 * x + 1 < G) pp[(2 * x + 1) * TQ_PART_STRIDE + 2 + gtid] = v.y;
    }
    if (lane == 0) {
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (gt * GT + warp * 2 + i < G) {
          pp[(warp * 2 + i) * TQ_PART_STRIDE] = m_h[i];
          pp[(warp * 2 + i) * TQ_PART_STRIDE + 1] = l_h[i];
        }
    }
  }
}

template <int VB>
int launch_pages(const DecodeArgs& a, int ctas, cudaStream_t st) {
  static_assert(sizeof(DpShared<VB>) <= 227 * 1024, "shared memory of one CTA");
  int device = 0;
  TQ_CUDA(cudaGetDevice(&device));
  static bool attr_set[16] = {};  // per device: the attribute belongs to the device's context
  if (!attr_set[device & 15]) {
    TQ_CUDA(cudaFuncSetAttribute(decode_pages_kernel<VB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(DpShared<VB>)));
    attr_set[device & 15] = true;
  }
  for (int s0 = 0; s0 < a.g.n_seqs; s0 += DP_SEQS)
    decode_pages_kernel<VB><<<ctas, DP_THREADS, sizeof(DpShared<VB>), st>>>(
        a, s0, a.g.n_seqs - s0 < DP_SEQS ? a.g.n_seqs - s0 : DP_SEQS);
  return TQ_OK;
}

}  // namespace

// Tiles of eight heads; a group of five to seven leaves up to three idle, one of nine to fifteen up to
// seven of its second tile.  Microseconds of a decode call, general kernel / this one, merge included
// (K4/V3, bf16; 64 units of 700 to 12 000 tokens, 64 of 6 000, 8 of 32 768, 32 of 900, 4 of 600):
//   5 heads   258 / 80   269 / 72   199 / 54   44 / 23   40 / 21
//   7 heads   260 / 80   271 / 72   200 / 54   44 / 24   40 / 22
//   9 heads   558 / 128  562 / 119  390 / 80   75 / 34   65 / 23
//  16 heads   557 / 137  560 / 121  387 / 81   79 / 35   66 / 23
// What bounds it: the look-ups (shared memory 56 %) and the issue slots (50 %) of splits and products.
int tq_launch_decode_pages(const DecodeArgs& a, int sm_count, cudaStream_t st) {
  return a.g.value_bits == 3 ? launch_pages<3>(a, sm_count, st) : launch_pages<4>(a, sm_count, st);
}
