// Dequantised read-back of a token range (the get_keys / get_values getters, and the restore of a
// stored request into an engine's pages).  The result is bit-identical to the reference decoders:
// keys are fl(fl(scale * NF4[code]) + mean) with outlier positions overwritten by their fp16
// values; values are (centroid[code] @ Pi) * norm with the rotation accumulated sequentially and
// unfused.
//
// One kernel serves all of it.  The values are bound by the FP32 pipe (128 multiplications and 128
// additions per element that may not be fused), keys and hot tokens by memory: the CTAs share out
// both kinds of jobs, every second CTA beginning with the memory-bound ones, so that the two
// overlap on an SM.
//   values  a job is 64 tokens of one page and head: the codes are expanded into shared memory
//           channel by channel ([channel][token]), then a thread accumulates 4 tokens x 8 channels
//           with packed multiplications and additions (two channels an instruction).  Pi lies in
//           shared memory (64 KB) for the life of the CTA.
//   keys    a job is 64 tokens of one page and head: a warp per token row, a lane per four
//           channels; the block's outliers that fall on these tokens are written over them after a
//           barrier (their list is loaded before the rows are, so the latencies overlap).
//   hot     a job is 32 tokens of the uncompressed window of one head.
// Results go to dense float32 tensors or, in the cache's or another element type, straight to the
// rows of an engine's paged tensor.
#include <algorithm>

#include "common.cuh"

namespace {

constexpr int DQ_THREADS = 256;
constexpr int DQ_VT = 64;              // tokens of a value job
constexpr int DQ_KT = 64;              // tokens of a key job
constexpr int DQ_HT = 32;              // tokens of a hot job
constexpr int DQ_STRIDE = DQ_VT + 8;   // floats per channel of the expanded codes: the pairs that
                                       // half a warp stores fall on different banks
constexpr int DQ_SMEM = (TQ_D * TQ_D + TQ_D * DQ_STRIDE) * 4;  // 100 KB: two CTAs per SM
constexpr int DQ_PRE = 3;              // outliers a thread loads ahead (256 x 3 cover the usual list)

struct DequantArgs {
  tq_geom g;
  const uint8_t* pages;
  const void* hot_k;
  const void* hot_v;
  const uint32_t* pool_dec;
  const uint16_t* pool_val;
  const PageMeta* page_meta;
  const Tables* tables;
  int layer, seq, start, end, n_total;
  void* k_out;
  void* v_out;
  // row of (position, head): dense, head_stride * head + row_stride * (position - start); paged,
  // ids[position / page_tokens] * page_stride + (position % page_tokens) * row_stride + head_stride * head,
  // nothing (and a status bit) where the id is outside [0, pages)
  const int64_t* ids;
  int64_t pages_out;
  int32_t* status;
  int page_tokens;
  int64_t page_stride, row_stride, head_stride;
  float one;    // 1.0f (see dq_add2)
  int aligned;  // every row takes vector stores
  int blk0, n_pages, v_tiles, k_tiles;
  int n_v, n_polar, n_k, n_h;  // jobs: values, PolarQuant keys (decoded like values), keys, hot
};

TQ_DEV unsigned long long dq_pack(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
TQ_DEV void dq_unpack(unsigned long long v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
// two products
TQ_DEV unsigned long long dq_mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// two sums a + b, as b * 1 + a with a one the compiler cannot see through: it fuses the packed
// mul.rn and add.rn of a product and a sum (the scalar ones it leaves alone), which would round once
// where the reference rounds twice
TQ_DEV unsigned long long dq_add2(unsigned long long a, unsigned long long b, unsigned long long one) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(b), "l"(one), "l"(a));
  return r;
}

template <int OT>
TQ_DEV typename Elem<OT>::type to_out(float x);
template <>
TQ_DEV float to_out<TQ_F32>(float x) { return x; }
template <>
TQ_DEV __half to_out<TQ_F16>(float x) { return __float2half_rn(x); }
template <>
TQ_DEV __nv_bfloat16 to_out<TQ_BF16>(float x) { return __float2bfloat16_rn(x); }

// four neighbouring elements of a row
template <int OT>
TQ_DEV void store4(typename Elem<OT>::type* p, float a, float b, float c, float d, int aligned) {
  using T = typename Elem<OT>::type;
  struct alignas(4 * sizeof(T)) V4 { T v[4]; } q;
  q.v[0] = to_out<OT>(a); q.v[1] = to_out<OT>(b); q.v[2] = to_out<OT>(c); q.v[3] = to_out<OT>(d);
  if (aligned) {
    *(V4*)p = q;
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) p[i] = q.v[i];
  }
}

// (null: the row has no place)
template <int OT, bool PAGED>
TQ_DEV typename Elem<OT>::type* out_row(const DequantArgs& a, void* base, int pos, int head) {
  int64_t o;
  if constexpr (PAGED) {
    const int64_t id = a.ids[pos / a.page_tokens];
    if ((uint64_t)id >= (uint64_t)a.pages_out) return nullptr;
    o = id * a.page_stride + (pos % a.page_tokens) * a.row_stride + head * a.head_stride;
  } else {
    o = (int64_t)head * a.head_stride + (int64_t)(pos - a.start) * a.row_stride;
  }
  return (typename Elem<OT>::type*)base + o;
}

// four neighbouring elements of a hot row (rows start on 256-byte boundaries)
TQ_DEV void ld4_any(const void* p, size_t i, int dt, float (&x)[4]) {
  if (dt == TQ_F32) {
    const float4 v = *(const float4*)((const float*)p + i);
    x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
    return;
  }
  const uint2 v = *(const uint2*)((const uint16_t*)p + i);
  const uint32_t w[2] = {v.x, v.y};
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    if (dt == TQ_F16) {
      const float2 f = __half22float2(*(const __half2*)&w[k]);
      x[2 * k] = f.x; x[2 * k + 1] = f.y;
    } else {
      x[2 * k] = __uint_as_float(w[k] << 16);
      x[2 * k + 1] = __uint_as_float(w[k] & 0xffff0000u);
    }
  }
}

template <int OT, bool PAGED>
__global__ void __launch_bounds__(DQ_THREADS, 2) dequant_kernel(DequantArgs a) {
  const tq_geom& g = a.g;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int S = g.block_tokens;
  extern __shared__ __align__(16) float dq_smem[];
  float* pi_s = dq_smem;                 // [D][D]
  float* us = dq_smem + TQ_D * TQ_D;     // [D][DQ_STRIDE]
  __shared__ float cent_s[16], grid_s[16];
  if (tid < 16) {
    cent_s[tid] = a.tables->centroids[tid];
    grid_s[tid] = a.tables->grid[tid];
  }
  const int first = blockIdx.x, step = gridDim.x;
  const int nv_all = a.n_v + a.n_polar, nm_all = a.n_k + a.n_h;
  if (first < nv_all) {  // Pi, on its way while the CTA does something else
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(pi_s);
    for (int i = tid; i < TQ_D * TQ_D / 4; i += DQ_THREADS)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * i),
                   "l"(a.tables->pi + 4 * i)
                   : "memory");
  }
  __syncthreads();
  // (a page without a place is reported once, at the end: no atomic among the loads and stores)
  bool missed = false;
  auto has_place = [&](const void* row) -> bool {
    if (!PAGED || row != nullptr) return true;
    missed = true;
    return false;
  };

  auto key_job = [&](int job) {
    const int kt = job % a.k_tiles, pg = job / a.k_tiles % a.n_pages,
              head = job / a.k_tiles / a.n_pages;
    const int blk = a.blk0 + pg, t0 = kt * DQ_KT;
    const int lo = max(t0, a.start - blk * S), hi = min(min(t0 + DQ_KT, S), a.end - blk * S);
    if (lo >= hi) return;  // (uniform over the CTA)
    const uint8_t* page = a.pages + page_offset(g, a.layer, a.seq, head, blk);
    const size_t unit = unit_index(g, a.layer, a.seq, head);
    PageMeta pm = {0, 0};
    if (g.outlier_k > 0) pm = a.page_meta[unit * g.max_blocks + blk];
    const size_t slab = unit * (size_t)g.pool_entries + pm.off;
    uint32_t ent[DQ_PRE];
#pragma unroll
    for (int i = 0; i < DQ_PRE; ++i) {
      const uint32_t e = tid + i * DQ_THREADS;
      ent[i] = e < pm.cnt ? a.pool_dec[slab + e] : 0u;
    }
    const float4 sc = *(const float4*)(page + g.scale_off + 16 * lane);
    const float4 mu = *(const float4*)(page + g.mean_off + 16 * lane);
    constexpr int WARPS = DQ_THREADS / 32;
    for (int t4 = lo + warp; t4 < hi; t4 += 4 * WARPS) {  // four rows: their loads, then their stores
      typename Elem<OT>::type* row[4];
      uint32_t w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = min(t4 + i * WARPS, hi - 1);
        row[i] = out_row<OT, PAGED>(a, a.k_out, blk * S + t, head);
        w[i] = *(const uint16_t*)(page + t * (TQ_D / 2) + 2 * lane);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        // symmetric NF4 stores mean 0, uniform keys are fl(fl(code * scale) + zero): one form
        if (t4 + i * WARPS < hi && has_place(row[i]))
          store4<OT>(row[i] + 4 * lane,
                     __fadd_rn(__fmul_rn(sc.x, grid_s[w[i] & 15]), mu.x),
                     __fadd_rn(__fmul_rn(sc.y, grid_s[(w[i] >> 4) & 15]), mu.y),
                     __fadd_rn(__fmul_rn(sc.z, grid_s[(w[i] >> 8) & 15]), mu.z),
                     __fadd_rn(__fmul_rn(sc.w, grid_s[w[i] >> 12]), mu.w), a.aligned);
      }
    }
    if (pm.cnt == 0) return;
    __syncthreads();  // the rows are written; the outliers go over them
    auto put = [&](uint32_t w, uint32_t e) {
      const int col = (w >> 16) & 255, t = (int)(w >> 24);
      if (t < lo || t >= hi) return;
      auto* row = out_row<OT, PAGED>(a, a.k_out, blk * S + t, head);
      if (has_place(row)) row[col] = to_out<OT>(__half2float(__ushort_as_half(a.pool_val[slab + e])));
    };
#pragma unroll
    for (int i = 0; i < DQ_PRE; ++i) {
      const uint32_t e = tid + i * DQ_THREADS;
      if (e < pm.cnt) put(ent[i], e);
    }
    for (uint32_t e = tid + DQ_PRE * DQ_THREADS; e < pm.cnt; e += DQ_THREADS)
      put(a.pool_dec[slab + e], e);
  };

  const int cold_end = n_cold_blocks(a.n_total, g.hot_window, S) * S;
  auto hot_job = [&](int job) {
    const int h0 = max(a.start, cold_end), n_tiles = a.n_h / g.n_kv_heads;
    const int head = job / n_tiles, p0 = h0 + job % n_tiles * DQ_HT;
    const size_t ring = hot_offset_elems(g, a.layer, a.seq, head);
#pragma unroll 4
    for (int pos = p0 + warp; pos < min(p0 + DQ_HT, a.end); pos += DQ_THREADS / 32) {
      const size_t i = ring + (size_t)(pos % g.hot_cap) * TQ_D + 4 * lane;
      float x[4];
      auto move = [&](const void* ring_of, void* to) {
        if (to == nullptr) return;
        auto* row = out_row<OT, PAGED>(a, to, pos, head);
        ld4_any(ring_of, i, g.kv_dtype, x);
        if (has_place(row)) store4<OT>(row + 4 * lane, x[0], x[1], x[2], x[3], a.aligned);
      };
      move(a.hot_k, a.k_out);
      move(a.hot_v, a.v_out);
    }
  };

  auto value_job = [&](int job) {
    const bool polar = job >= a.n_v;  // PolarQuant keys: codes and norms in the key fields
    if (polar) job -= a.n_v;
    const int vt = job % a.v_tiles, pg = job / a.v_tiles % a.n_pages,
              head = job / a.v_tiles / a.n_pages;
    const int blk = a.blk0 + pg, t0 = vt * DQ_VT;
    const int lo = max(t0, a.start - blk * S), hi = min(min(t0 + DQ_VT, S), a.end - blk * S);
    if (lo >= hi) return;  // (uniform over the CTA)
    const uint8_t* page = a.pages + page_offset(g, a.layer, a.seq, head, blk);
    {
      // warp w expands pairs 16 (w & 1) .. + 15 of every lane record of the tile's group w >> 1
      const int grp = warp >> 1, half = warp & 1;
      const int gq = (t0 >> 4) + grp;
      if (gq * TQ_GROUP_TOK < g.block_tokens_pad) {
        const uint8_t* src =
            page + (polar ? 0 : g.v_off) + (size_t)gq * v_group_bytes(g.value_bits);
        float* dst = us + (64 * half + (lane >> 2)) * DQ_STRIDE + 16 * grp + 2 * (lane & 3);
        if (g.value_bits == 4) {
          const uint4 q = *(const uint4*)(src + half * 512 + lane * 16);
          const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const uint32_t b = w[i >> 2] >> (8 * (i & 3));
            *(float2*)(dst + 8 * (i >> 1) * DQ_STRIDE + 8 * (i & 1)) =
                make_float2(cent_s[b & 15], cent_s[(b >> 4) & 15]);
          }
        } else {
          // the record's 24 bytes; this half's sixteen 6-bit pairs are words 3 half .. + 2
          const uint2 r0 = *(const uint2*)(src + lane * 8), r1 = *(const uint2*)(src + 256 + lane * 8),
                      r2 = *(const uint2*)(src + 512 + lane * 8);
          const uint32_t w[4] = {half ? r1.y : r0.x, half ? r2.x : r0.y, half ? r2.y : r1.x, 0u};
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int bit = 6 * i;
            const uint32_t b = __funnelshift_r(w[bit >> 5], w[(bit >> 5) + 1], bit & 31);
            *(float2*)(dst + 8 * (i >> 1) * DQ_STRIDE + 8 * (i & 1)) =
                make_float2(cent_s[b & 7], cent_s[(b >> 3) & 7]);
          }
        }
      }
    }
    __syncthreads();
    // thread: tokens 4 ty .. + 3, channels 4 tx .. + 3 and 64 + 4 tx .. + 3
    const int tx = tid & 15, ty = tid >> 4;
    unsigned long long acc[4][4];
    const unsigned long long one = dq_pack(a.one, a.one);
    const float* up = us + 4 * ty;
    const float* pp = pi_s + 4 * tx;
    {
      const float4 u = *(const float4*)up;
      const ulonglong2 p0 = *(const ulonglong2*)pp, p1 = *(const ulonglong2*)(pp + 64);
      const float uv[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const unsigned long long uu = dq_pack(uv[t], uv[t]);
        acc[t][0] = dq_mul2(uu, p0.x);
        acc[t][1] = dq_mul2(uu, p0.y);
        acc[t][2] = dq_mul2(uu, p1.x);
        acc[t][3] = dq_mul2(uu, p1.y);
      }
    }
#pragma unroll 8
    for (int d = 1; d < TQ_D; ++d) {
      const float4 u = *(const float4*)(up + d * DQ_STRIDE);
      const ulonglong2 p0 = *(const ulonglong2*)(pp + d * TQ_D),
                       p1 = *(const ulonglong2*)(pp + d * TQ_D + 64);
      const float uv[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const unsigned long long uu = dq_pack(uv[t], uv[t]);
        acc[t][0] = dq_add2(acc[t][0], dq_mul2(uu, p0.x), one);
        acc[t][1] = dq_add2(acc[t][1], dq_mul2(uu, p0.y), one);
        acc[t][2] = dq_add2(acc[t][2], dq_mul2(uu, p1.x), one);
        acc[t][3] = dq_add2(acc[t][3], dq_mul2(uu, p1.y), one);
      }
    }
    const float* norms = (const float*)(page + (polar ? g.scale_off : g.norm_off));
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int tt = t0 + 4 * ty + t;
      if (tt >= lo && tt < hi) {
        const float nrm = norms[tt];
        float x[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          dq_unpack(acc[t][j], x[2 * j], x[2 * j + 1]);
          x[2 * j] = __fmul_rn(x[2 * j], nrm);
          x[2 * j + 1] = __fmul_rn(x[2 * j + 1], nrm);
        }
        auto* row = out_row<OT, PAGED>(a, polar ? a.k_out : a.v_out, blk * S + tt, head);
        if (has_place(row)) {
          store4<OT>(row + 4 * tx, x[0], x[1], x[2], x[3], a.aligned);
          store4<OT>(row + 64 + 4 * tx, x[4], x[5], x[6], x[7], a.aligned);
        }
      }
    }
    __syncthreads();  // the expanded codes make room for the next job's
  };

  const bool memory_first = (first & 1) != 0;
  for (int part = 0; part < 2; ++part) {
    if ((part == 0) == memory_first) {
      for (int j = first; j < nm_all; j += step) {
        if (j < a.n_k) key_job(j); else hot_job(j - a.n_k);
      }
    } else if (first < nv_all) {
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();
      for (int j = first; j < nv_all; j += step) value_job(j);
    }
  }
  if (missed) atomicOr(a.status, TQ_STATUS_BAD_PAGE);
}

template <int OT, bool PAGED>
int launch_t(const DequantArgs& a, int device, cudaStream_t st) {
  static bool attr_set[64] = {};  // per device: the attribute belongs to the device's context
  if (device >= 64 || !attr_set[device]) {
    TQ_CUDA(cudaFuncSetAttribute(dequant_kernel<OT, PAGED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 DQ_SMEM));
    if (device < 64) attr_set[device] = true;
  }
  int sm_count = 148;
  cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, device);
  // one wave of resident CTAs: Pi is fetched once per CTA
  const int jobs = std::max(a.n_v + a.n_polar, a.n_k + a.n_h);
  dequant_kernel<OT, PAGED><<<std::min(jobs, 2 * sm_count), DQ_THREADS, DQ_SMEM, st>>>(a);
  TQ_CUDA(cudaGetLastError());
  return TQ_OK;
}

int launch(tq_ctx* ctx, DequantArgs& a, int layer, int seq, int start, int end, int dtype,
           cudaStream_t st) {
  const tq_geom& g = ctx->g;
  a.g = g;
  a.one = 1.0f;
  a.pages = (const uint8_t*)ctx->b.pages;
  a.hot_k = ctx->b.hot_k;
  a.hot_v = ctx->b.hot_v;
  a.pool_dec = (const uint32_t*)ctx->b.pool_dec;
  a.pool_val = (const uint16_t*)ctx->b.pool_val;
  a.page_meta = (const PageMeta*)ctx->b.page_meta;
  a.tables = (const Tables*)ctx->b.tables;
  a.status = (int32_t*)((uint8_t*)ctx->b.state + state_status_off(g));
  a.layer = layer;
  a.seq = seq;
  a.start = start;
  a.end = end;
  a.n_total = ctx->len[(size_t)layer * g.n_seqs + seq];
  // vector stores take four elements: the bases and every stride on that grid
  const size_t v4 = 4 * (size_t)elem_size(dtype);
  a.aligned = (((uintptr_t)a.k_out | (uintptr_t)a.v_out) % v4) == 0 &&
              ((a.page_stride | a.row_stride | a.head_stride) & 3) == 0;
  const int S = g.block_tokens;
  const int cold_end = n_cold_blocks(a.n_total, g.hot_window, S) * S;
  const int cend = std::min(end, cold_end), hbeg = std::max(start, cold_end);
  a.blk0 = start / S;
  a.n_pages = start < cend ? (cend - 1) / S - a.blk0 + 1 : 0;
  a.v_tiles = (g.block_tokens_pad + DQ_VT - 1) / DQ_VT;
  a.k_tiles = (S + DQ_KT - 1) / DQ_KT;
  const bool polar = g.key_mode == TQ_KEYS_POLAR;
  a.n_v = a.v_out != nullptr ? g.n_kv_heads * a.n_pages * a.v_tiles : 0;
  // (PolarQuant keys: TurboQuantKV.decompress on the key codes, core.py:619-654)
  a.n_polar = a.k_out != nullptr && polar ? g.n_kv_heads * a.n_pages * a.v_tiles : 0;
  a.n_k = a.k_out != nullptr && !polar ? g.n_kv_heads * a.n_pages * a.k_tiles : 0;
  a.n_h = end > hbeg ? g.n_kv_heads * ((end - hbeg + DQ_HT - 1) / DQ_HT) : 0;
  if (a.ids == nullptr) return launch_t<TQ_F32, false>(a, ctx->device, st);
  switch (dtype) {
    case TQ_F32: return launch_t<TQ_F32, true>(a, ctx->device, st);
    case TQ_F16: return launch_t<TQ_F16, true>(a, ctx->device, st);
    default: return launch_t<TQ_BF16, true>(a, ctx->device, st);
  }
}

}  // namespace

int tq_launch_dequant(tq_ctx* ctx, int layer, int seq, int start, int end, float* k_out,
                      float* v_out, cudaStream_t st) {
  DequantArgs a = {};
  a.k_out = k_out;
  a.v_out = v_out;
  a.row_stride = TQ_D;
  a.head_stride = (int64_t)(end - start) * TQ_D;
  return launch(ctx, a, layer, seq, start, end, TQ_F32, st);
}

int tq_launch_dequant_paged(tq_ctx* ctx, int layer, int seq, int n_tokens, void* k_pages,
                            void* v_pages, int dtype, const int64_t* page_ids, int64_t n_pages,
                            int page_tokens, int64_t page_stride, int64_t row_stride,
                            int64_t head_stride, cudaStream_t st) {
  DequantArgs a = {};
  a.k_out = k_pages;
  a.v_out = v_pages;
  a.ids = page_ids;
  a.pages_out = n_pages;
  a.page_tokens = page_tokens;
  a.page_stride = page_stride;
  a.row_stride = row_stride;
  a.head_stride = head_stride;
  return launch(ctx, a, layer, seq, 0, n_tokens, dtype, st);
}
