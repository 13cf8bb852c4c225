// Decode-on-codes attention in float32 for 256-token blocks and query groups the tensor-core kernel
// has no tile for (5, 6, 7 and 9 to 16 query heads per KV head), and for larger groups wherever the
// general-shape kernel is asked for.  Same arithmetic as decode_generic.cu: float32 products and sums
// throughout; the partials have its layout and go through its combine kernel.
//
// Bound by latency, not by issue.  Counters of one launch (160 units of seven heads, 700 to 12 000
// tokens, 422 us): 32 % of the issue slots, 2.5 warps per scheduler of which 0.4 can issue; of 7.9
// cycles between two instructions of a warp 3.6 wait for global memory (codes, scales, norms and outlier
// lists are fetched where they are used, between the page's four barriers); and the splits are uneven, the
// busiest SM works 822 000 cycles, the average one 633 000.  168 registers hold it at three CTAs an
// SM, with 40 bytes spilled.  decode_generic.cu looks every code up once per tile of four heads, a
// 16-token group at a time; here a code is looked up once for eight heads and feeds packed
// multiply-adds (two heads an instruction), sixteen instructions per code and lane in all:
//   scores   a lane owns two tokens and walks their channels; the weights w = q * scale of a channel
//            lie side by side for the heads, two broadcast loads for both tokens;
//   softmax  once per page: a warp takes a head's 256 scores, so there is one rescaling a page;
//   values   a warp takes half the channels of every second 16-token group (one 12- or 16-byte load
//            per lane), its tokens' probabilities come as four-head vectors.
// The uncompressed window: a thread per token for the scores, a thread per channel for the values.
#include "decode_generic.cuh"

namespace {

constexpr int DP_THREADS = 128;
constexpr int DP_GT = 8;           // query heads a CTA takes
constexpr int DP_S = 256;
constexpr int DP_SROW = DP_S + 4;  // scores of a head
constexpr int DP_HOT = 128;        // hot tokens per round

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

// GT query heads of one KV head per CTA; grid = (splits, units, head tiles)
__global__ void __launch_bounds__(DP_THREADS, 3) decode_pages_kernel(DecodeArgs a) {
  constexpr int GT = DP_GT;
  constexpr int NP = GT / 2;          // pairs of heads
  constexpr int PROW = GT + 4;        // floats per token of the probabilities
  constexpr int HW = GT / 4;          // heads per warp in the softmax
  const tq_geom& g = a.g;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int split = blockIdx.x, unit = blockIdx.y, gt = blockIdx.z;
  const int seq = unit / g.n_kv_heads, head = unit % g.n_kv_heads;
  const int G = g.group, vb = g.value_bits;
  const int N = a.seq_len[a.layer * g.n_seqs + seq];
  const int nb = n_cold_blocks(N, g.hot_window, DP_S);
  const bool cold = split < a.ns_cold;

  __shared__ __align__(16) float q_s[TQ_D][GT], w_s[TQ_D][GT];
  __shared__ float s_s[GT][DP_SROW];  // outlier corrections, then scores
  __shared__ __align__(16) float p_s[DP_S][PROW];
  __shared__ float bias_w[4][GT], f_s[GT];
  __shared__ float nf4_s[16], cent_s[16];
  if (tid < 16) {
    nf4_s[tid] = a.tables->grid[tid];
    cent_s[tid] = a.tables->centroids[tid];
  }
#pragma unroll
  for (int gg = 0; gg < GT; ++gg) {
    const int qh = gt * GT + gg;
    q_s[tid][gg] = qh < G ? dp_ld(a.q, ((size_t)seq * g.n_q_heads + head * G + qh) * TQ_D + tid,
                                  a.q_dtype)
                          : 0.0f;
  }
  float m_run[HW], l_run[HW];  // of heads warp * HW + i, the same in every lane
#pragma unroll
  for (int i = 0; i < HW; ++i) {
    m_run[i] = -INFINITY;
    l_run[i] = 0.0f;
  }
  __syncthreads();

  // the softmax of a round's scores: probabilities times `wgt`, and the factor for what was
  // accumulated before
  auto softmax = [&](int n_tok, auto wgt) {
#pragma unroll
    for (int i = 0; i < HW; ++i) {
      const int gg = warp * HW + i;
      float mx = -INFINITY;
      for (int t = lane; t < n_tok; t += 32) mx = fmaxf(mx, s_s[gg][t]);
      __syncwarp();
#pragma unroll
      for (int o = 16; o >= 1; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      const float m_new = fmaxf(m_run[i], mx);
      const bool any = m_new > -INFINITY;
      const float f = any ? __expf(m_run[i] - m_new) : 1.0f;
      float sum = 0.0f;
      for (int t = lane; t < n_tok; t += 32) {
        const float p = any ? __expf(s_s[gg][t] - m_new) : 0.0f;
        sum += p;
        p_s[t][gg] = p * wgt(t);
      }
      __syncwarp();
#pragma unroll
      for (int o = 16; o >= 1; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      l_run[i] = l_run[i] * f + sum;
      m_run[i] = m_new;
      if (lane == 0) f_s[gg] = f;
    }
  };

  const size_t out0 = ((size_t)unit * g.max_splits + split) * G + gt * GT;
  if (cold) {
    unsigned long long acc[8][NP];  // channels 64 (warp & 1) + 8 k + lane / 4
#pragma unroll
    for (int k = 0; k < 8; ++k)
#pragma unroll
      for (int x = 0; x < NP; ++x) acc[k][x] = 0ull;
    const int b0 = min(a.block_begin, nb), b1 = a.block_end < 0 ? nb : min(a.block_end, nb);
    const int nbr = max(b1 - b0, 0);
    const int p_lo = b0 + (int)((long)nbr * split / a.ns_cold);
    const int p_hi = b0 + (int)((long)nbr * (split + 1) / a.ns_cold);
    const size_t u_idx = unit_index(g, a.layer, seq, head);
    for (int pg = p_lo; pg < p_hi; ++pg) {
      const uint8_t* page = a.pages + page_offset(g, a.layer, seq, head, pg);
      // the two tokens' code rows, on their way while the weights are formed
      uint4 row[2][4];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int v = 0; v < 4; ++v)
          row[h][v] = ((const uint4*)(page + (64 * warp + 32 * h + lane) * (TQ_D / 2)))[v];
      {
        const float sc = ((const float*)(page + g.scale_off))[tid];
        const float mu = ((const float*)(page + g.mean_off))[tid];
#pragma unroll
        for (int gg = 0; gg < GT; ++gg) {
          const float qv = q_s[tid][gg];
          w_s[tid][gg] = qv * sc;
          float b = qv * mu;
#pragma unroll
          for (int o = 16; o >= 1; o >>= 1) b += __shfl_xor_sync(0xffffffffu, b, o);
          if (lane == 0) bias_w[warp][gg] = b;
          s_s[gg][tid] = 0.0f;
          s_s[gg][tid + 128] = 0.0f;
        }
      }
      __syncthreads();
      if (g.outlier_k > 0) {
        // ordered by token, then channel: the thread with a token's first entry adds up all of
        // them, so the sum does not depend on timing
        const PageMeta pm = a.page_meta[u_idx * g.max_blocks + pg];
        const uint32_t* ent = a.pool_dec + u_idx * (size_t)g.pool_entries + pm.off;
        for (uint32_t e = tid; e < pm.cnt; e += DP_THREADS) {
          const int tk = (int)(ent[e] >> 24);
          if (e > 0 && (int)(ent[e - 1] >> 24) == tk) continue;
          float sum[GT];
#pragma unroll
          for (int gg = 0; gg < GT; ++gg) sum[gg] = 0.0f;
          for (uint32_t j = e; j < pm.cnt; ++j) {
            const uint32_t wv = ent[j];
            if ((int)(wv >> 24) != tk) break;
            const float delta = __half2float(__ushort_as_half((unsigned short)(wv & 0xffff)));
            const float* qr = q_s[(wv >> 16) & 127];
#pragma unroll
            for (int gg = 0; gg < GT; ++gg) sum[gg] += qr[gg] * delta;
          }
#pragma unroll
          for (int gg = 0; gg < GT; ++gg) s_s[gg][tk] = sum[gg];
        }
      }
      __syncthreads();
      {
        // eight channels at a time, then those sums: shorter chains of rounding than one of 128
        unsigned long long dot[2][NP], sub[2][NP];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int x = 0; x < NP; ++x) dot[h][x] = sub[h][x] = 0ull;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const uint32_t cw[2][4] = {{row[0][v].x, row[0][v].y, row[0][v].z, row[0][v].w},
                                     {row[1][v].x, row[1][v].y, row[1][v].z, row[1][v].w}};
#pragma unroll
          for (int n = 0; n < 32; ++n) {
            unsigned long long w2[NP];
#pragma unroll
            for (int x = 0; x < NP; x += 2) {
              const ulonglong2 t = *(const ulonglong2*)&w_s[32 * v + n][2 * x];
              w2[x] = t.x;
              w2[x + 1] = t.y;
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const float lv = nf4_s[(cw[h][n >> 3] >> (4 * (n & 7))) & 15];
              const unsigned long long l2 = dp_pack(lv, lv);
#pragma unroll
              for (int x = 0; x < NP; ++x) {
                sub[h][x] = (n & 7) == 0 ? dp_mul2(l2, w2[x]) : dp_fma2(l2, w2[x], sub[h][x]);
                if ((n & 7) == 7) dot[h][x] = dp_add2(dot[h][x], sub[h][x]);
              }
            }
          }
          if (v == 1) {  // the first half of the channels joins the corrections
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int x = 0; x < NP; ++x) {
                const float2 e = dp_unpack(dot[h][x]);
                s_s[2 * x][64 * warp + 32 * h + lane] += e.x;
                s_s[2 * x + 1][64 * warp + 32 * h + lane] += e.y;
                dot[h][x] = 0ull;
              }
          }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int t = 64 * warp + 32 * h + lane;
#pragma unroll
          for (int x = 0; x < NP; ++x) {
            const float2 e = dp_unpack(dot[h][x]);
            const float d2[2] = {e.x, e.y};
#pragma unroll
            for (int y = 0; y < 2; ++y) {
              const int gg = 2 * x + y;
              const float bias = bias_w[0][gg] + bias_w[1][gg] + bias_w[2][gg] + bias_w[3][gg];
              s_s[gg][t] = (d2[y] + bias + s_s[gg][t]) * a.scale;
            }
          }
        }
      }
      __syncthreads();
      const float* norms = (const float*)(page + g.norm_off);
      softmax(DP_S, [&](int t) { return norms[t]; });
      __syncthreads();
      {
        const int half = warp & 1;
#pragma unroll
        for (int x = 0; x < NP; ++x) {
          const unsigned long long f2 = dp_pack(f_s[2 * x], f_s[2 * x + 1]);
#pragma unroll
          for (int k = 0; k < 8; ++k) acc[k][x] = dp_mul2(acc[k][x], f2);
        }
        const int c4 = lane & 3;
#pragma unroll 1
        for (int gq = warp >> 1; gq < DP_S / TQ_GROUP_TOK; gq += 2) {
          const uint8_t* grp = page + g.v_off + (size_t)gq * v_group_bytes(vb);
          uint32_t rec[4];
          if (vb == 4) {
            const uint4 r = *(const uint4*)(grp + half * 512 + lane * 16);
            rec[0] = r.x; rec[1] = r.y; rec[2] = r.z; rec[3] = r.w;
          } else {
            // bytes 12 half .. + 11 of the lane's 24-byte record (parts of 8 bytes)
            const uint2 mid = *(const uint2*)(grp + 256 + lane * 8);
            const uint2 end = *(const uint2*)(grp + half * 512 + lane * 8);
            rec[0] = half ? mid.y : end.x;
            rec[1] = half ? end.x : end.y;
            rec[2] = half ? end.y : mid.x;
            rec[3] = 0u;
          }
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {  // tokens 2 c4, 2 c4 + 1 of the group's lower, upper eight
            unsigned long long pr[2][NP];
#pragma unroll
            for (int o = 0; o < 2; ++o)
#pragma unroll
              for (int x = 0; x < NP; x += 2) {
                const ulonglong2 t =
                    *(const ulonglong2*)&p_s[16 * gq + 8 * hh + 2 * c4 + o][2 * x];
                pr[o][x] = t.x;
                pr[o][x + 1] = t.y;
              }
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const int p = 2 * k + hh;
              uint32_t ca, cb;
              if (vb == 4) {
                const uint32_t b = rec[p >> 2] >> (8 * (p & 3));
                ca = b & 15;
                cb = (b >> 4) & 15;
              } else {
                const int bit = 6 * p;
                const uint32_t b = __funnelshift_r(rec[bit >> 5], rec[(bit >> 5) + 1], bit & 31);
                ca = b & 7;
                cb = (b >> 3) & 7;
              }
              const float va = cent_s[ca], vc = cent_s[cb];
              const unsigned long long a2 = dp_pack(va, va), c2 = dp_pack(vc, vc);
#pragma unroll
              for (int x = 0; x < NP; ++x)  // (two tokens, then the sum: half the chain)
                acc[k][x] = dp_add2(acc[k][x], dp_fma2(c2, pr[1][x], dp_mul2(a2, pr[0][x])));
            }
          }
        }
      }
      // (no barrier: what the next page writes first is not read by the value phase)
    }
    // lanes of a quad hold different tokens of the same channels, and so do warps w and w + 2
    __syncthreads();
    float* mrg = &p_s[0][0];  // [GT][D]
    static_assert(GT * TQ_D <= DP_S * PROW, "merge area");
    for (int part = 0; part < 2; ++part) {
      if (warp >> 1 == part) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
#pragma unroll
          for (int x = 0; x < NP; ++x) {
            const float2 v = dp_unpack(acc[k][x]);
            float vv[2] = {v.x, v.y};
#pragma unroll
            for (int y = 0; y < 2; ++y) {
              vv[y] += __shfl_xor_sync(0xffffffffu, vv[y], 1);
              vv[y] += __shfl_xor_sync(0xffffffffu, vv[y], 2);
              if ((lane & 3) == 0) {
                float* dst = mrg + (2 * x + y) * TQ_D + 64 * (warp & 1) + 8 * k + (lane >> 2);
                *dst = part == 0 ? vv[y] : *dst + vv[y];
              }
            }
          }
      }
      __syncthreads();
    }
#pragma unroll
    for (int gg = 0; gg < GT; ++gg)
      if (gt * GT + gg < G) a.partials[(out0 + gg) * TQ_PART_STRIDE + 2 + tid] = mrg[gg * TQ_D + tid];
  } else {
    unsigned long long acc[NP];  // channel tid
#pragma unroll
    for (int x = 0; x < NP; ++x) acc[x] = 0ull;
    const int j = split - a.ns_cold, dt = g.kv_dtype;
    const int hot_start = nb * DP_S, hot_len = a.with_hot ? N - hot_start : 0;
    const int ng = (hot_len + TQ_GROUP_TOK - 1) / TQ_GROUP_TOK;
    const int t_lo = (int)((long)ng * j / a.ns_hot) * TQ_GROUP_TOK;
    const int t_hi = min((int)((long)ng * (j + 1) / a.ns_hot) * TQ_GROUP_TOK, hot_len);
    const size_t ring = hot_offset_elems(g, a.layer, seq, head);
    for (int t0 = t_lo; t0 < t_hi; t0 += DP_HOT) {
      const int n_tok = min(DP_HOT, t_hi - t0);
      if (tid < n_tok) {
        const size_t at = ring + (size_t)((hot_start + t0 + tid) % g.hot_cap) * TQ_D;
        unsigned long long dot[NP], sub[NP], low[NP];
#pragma unroll
        for (int x = 0; x < NP; ++x) dot[x] = sub[x] = low[x] = 0ull;
#pragma unroll 2
        for (int d0 = 0; d0 < TQ_D; d0 += 8) {
          float kv[8];
          if (dt == TQ_F32) {
            const float4 x = *(const float4*)((const float*)a.hot_k + at + d0);
            const float4 y = *(const float4*)((const float*)a.hot_k + at + d0 + 4);
            kv[0] = x.x; kv[1] = x.y; kv[2] = x.z; kv[3] = x.w;
            kv[4] = y.x; kv[5] = y.y; kv[6] = y.z; kv[7] = y.w;
          } else {
            const uint4 x = *(const uint4*)((const uint16_t*)a.hot_k + at + d0);
            const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              if (dt == TQ_F16) {
                const float2 f = __half22float2(*(const __half2*)&w[i]);
                kv[2 * i] = f.x; kv[2 * i + 1] = f.y;
              } else {
                kv[2 * i] = __uint_as_float(w[i] << 16);
                kv[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
              }
            }
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const unsigned long long k2 = dp_pack(kv[i], kv[i]);
#pragma unroll
            for (int x = 0; x < NP; x += 2) {
              const ulonglong2 t = *(const ulonglong2*)&q_s[d0 + i][2 * x];
              sub[x] = i == 0 ? dp_mul2(k2, t.x) : dp_fma2(k2, t.x, sub[x]);
              sub[x + 1] = i == 0 ? dp_mul2(k2, t.y) : dp_fma2(k2, t.y, sub[x + 1]);
            }
          }
#pragma unroll
          for (int x = 0; x < NP; ++x) {
            if (d0 == TQ_D / 2) {  // (the halves add up separately)
              low[x] = dot[x];
              dot[x] = 0ull;
            }
            dot[x] = dp_add2(dot[x], sub[x]);
          }
        }
#pragma unroll
        for (int x = 0; x < NP; ++x) {
          const float2 e = dp_unpack(dp_add2(low[x], dot[x]));
          s_s[2 * x][tid] = e.x * a.scale;
          s_s[2 * x + 1][tid] = e.y * a.scale;
        }
      }
      __syncthreads();
      softmax(n_tok, [](int) { return 1.0f; });
      __syncthreads();
#pragma unroll
      for (int x = 0; x < NP; ++x) acc[x] = dp_mul2(acc[x], dp_pack(f_s[2 * x], f_s[2 * x + 1]));
      int slot = (hot_start + t0) % g.hot_cap;
      for (int tb = 0; tb < n_tok; tb += 8) {  // eight tokens, then their sum
        unsigned long long sub[NP];
#pragma unroll
        for (int x = 0; x < NP; ++x) sub[x] = 0ull;
        const int m = min(8, n_tok - tb);
#pragma unroll
        for (int t = 0; t < 8; ++t) {
          if (t < m) {
            const float v = dp_ld(a.hot_v, ring + (size_t)slot * TQ_D + tid, dt);
            if (++slot == g.hot_cap) slot = 0;
            const unsigned long long v2 = dp_pack(v, v);
#pragma unroll
            for (int x = 0; x < NP; x += 2) {
              const ulonglong2 p = *(const ulonglong2*)&p_s[tb + t][2 * x];
              sub[x] = dp_fma2(v2, p.x, sub[x]);
              sub[x + 1] = dp_fma2(v2, p.y, sub[x + 1]);
            }
          }
        }
#pragma unroll
        for (int x = 0; x < NP; ++x) acc[x] = dp_add2(acc[x], sub[x]);
      }
      // (no barrier: the next round's scores are not read here, its probabilities come after two)
    }
#pragma unroll
    for (int x = 0; x < NP; ++x) {
      const float2 v = dp_unpack(acc[x]);
      if (gt * GT + 2 * x < G) a.partials[(out0 + 2 * x) * TQ_PART_STRIDE + 2 + tid] = v.x;
      if (gt * GT + 2 * x + 1 < G) a.partials[(out0 + 2 * x + 1) * TQ_PART_STRIDE + 2 + tid] = v.y;
    }
  }
  if (lane == 0) {
#pragma unroll
    for (int i = 0; i < HW; ++i) {
      const int gg = warp * HW + i;
      if (gt * GT + gg < G) {
        a.partials[(out0 + gg) * TQ_PART_STRIDE] = m_run[i];
        a.partials[(out0 + gg) * TQ_PART_STRIDE + 1] = l_run[i];
      }
    }
  }
}

}  // namespace

void tq_launch_decode_pages(const DecodeArgs& a, int n_units, cudaStream_t st) {
  // Tiles of eight heads; a group of five to seven leaves up to three idle, one of nine to fifteen
  // up to seven of its second tile.  Microseconds a layer, general kernel / this one (K4/V3, bf16; 64
  // units of 700 to 12 000 tokens, 64 of 6 000, 8 of 32 768, 32 of 900):
  //   5 heads   252 / 203   264 / 192   191 / 110   39 / 31
  //   7 heads   254 / 203   266 / 192   192 / 110   39 / 31
  //   8 heads   310 / 203   311 / 193   232 / 110   52 / 31   (where the general kernel is asked for)
  //   9 heads   553 / 256   557 / 256   382 / 170   70 / 36
  //  16 heads   552 / 257   555 / 256   379 / 170   74 / 36
  const dim3 grid(a.ns_cold + a.ns_hot, n_units, (a.g.group + DP_GT - 1) / DP_GT);
  decode_pages_kernel<<<grid, DP_THREADS, 0, st>>>(a);
}
