// Cold blocks to and from the reference's container layout, many blocks at a time, on the device.
// tq_export_block / tq_import_block do the same for one block with loops on the host (about 1 ms a
// block of eight heads, most of it single codes); here a CTA converts the page of one KV head, and
// the containers of all blocks travel in one copy.  Bound by latency: a block's page and containers
// are 70 KB, its conversion shuffles bits through shared memory.
//
// Layout of a block in the staging buffer (every part 16-byte aligned, as the sizes show):
//   key codes (H x S x 64 B; PolarQuant keys: H x S x 16 key_bits B) | scale (H x 128 floats;
//   PolarQuant keys: the H x S norms) | mean (H x 128 floats) | value codes (H x S x 16 value_bits
//   B) | value norms (H x S floats)
// and for all blocks together the outliers: int32 flat indices, then uint16 fp16 bits, block after
// block, head after head, ascending.
#include <algorithm>

#include "common.cuh"

namespace {

constexpr int WIRE_THREADS = 256;
// Dynamic shared memory a launch may ask for: the largest page (256 tokens, 4-bit values: 38 KB) and
// its value codes as a bit stream (16 KB).  The limit belongs to the kernel on a device, not to a
// context: it is set once, to the same value whoever comes first, so that no thread's small geometry
// can take it away between another's look and launch.
constexpr int WIRE_SMEM = 64 * 1024;

struct WireParts {
  int64_t key, scale, mean, val, norm, bytes;  // offsets of a block's parts, bytes of a block
};

WireParts wire_parts(const tq_geom& g) {
  const int64_t H = g.n_kv_heads, S = g.block_tokens;
  const bool polar = g.key_mode == TQ_KEYS_POLAR;
  WireParts p;
  p.key = 0;
  p.scale = align_up(polar ? H * S * 16 * g.key_bits : H * S * 64, 16);
  p.mean = align_up(p.scale + (polar ? H * S : H * TQ_D) * 4, 16);
  p.val = p.mean + H * TQ_D * 4;
  p.norm = p.val + H * S * 16 * g.value_bits;
  p.bytes = align_up(p.norm + H * S * 4, 16);
  return p;
}

struct WireArgs {
  tq_geom g;
  WireParts parts;
  uint8_t* pages;
  uint32_t* pool_dec;
  uint16_t* pool_val;
  PageMeta* page_meta;
  uint32_t* cursor;  // of the sequence's heads
  const Tables* tables;
  uint8_t* staging;
  int32_t* out_idx;
  uint16_t* out_val;
  const int32_t* first;  // import: first outlier of (block, head), and the end
  int32_t* short_flag;   // import: set when the outlier pool could not take everything
  int layer, seq, blk0, n_blocks;
  int64_t n_out;  // export: outliers the buffers take
};

// every byte's bits in reverse order: the container keeps bit-reversed nibbles, the first channel
// of a pair on top
TQ_DEV uint32_t rev_bytes(uint32_t w) { return __byte_perm(__brev(w), 0, 0x0123); }

// value-layout codes -> LSB-first bit stream: a thread packs 32 channels of a token
TQ_DEV void stream_from_records(const uint8_t* rec, uint8_t* dst, int S, int bits, int tid) {
  uint32_t* out = (uint32_t*)dst;
  for (int i = tid; i < S * 4; i += WIRE_THREADS) {
    const int t = i >> 2, d0 = (i & 3) * 32;
    const uint8_t* grp = rec + (size_t)(t / TQ_GROUP_TOK) * v_group_bytes(bits);
    unsigned long long acc = 0;
    int have = 0, w = 0;
    for (int d = d0; d < d0 + 32; ++d) {
      acc |= (unsigned long long)v_get_code(grp, bits, t % TQ_GROUP_TOK, d) << have;
      have += bits;
      if (have >= 32) {
        out[i * bits + w++] = (uint32_t)acc;
        acc >>= 32;
        have -= 32;
      }
    }
  }
}

// code (t, d) of a bit stream
TQ_DEV uint32_t stream_code(const uint8_t* src, int bits, int t, int d) {
  const int bit = (t * TQ_D + d) * bits;
  uint32_t w = src[bit >> 3];
  if ((bit & 7) + bits > 8) w |= (uint32_t)src[(bit >> 3) + 1] << 8;
  return (w >> (bit & 7)) & ((1u << bits) - 1);
}

TQ_DEV void copy_words(const void* src, void* dst, int words, int tid) {
  for (int i = tid; i < words; i += WIRE_THREADS) ((uint32_t*)dst)[i] = ((const uint32_t*)src)[i];
}

// grid = (heads, blocks)
__global__ void __launch_bounds__(WIRE_THREADS) export_kernel(WireArgs a) {
  const tq_geom& g = a.g;
  const int tid = threadIdx.x, head = blockIdx.x, b = blockIdx.y, blk = a.blk0 + b;
  const int S = g.block_tokens, H = g.n_kv_heads;
  const bool polar = g.key_mode == TQ_KEYS_POLAR;
  extern __shared__ __align__(16) uint8_t pg[];  // the page up to its tail
  const uint8_t* page = a.pages + page_offset(g, a.layer, a.seq, head, blk);
  for (int i = tid; i < g.hdr_off / 16; i += WIRE_THREADS) ((uint4*)pg)[i] = ((const uint4*)page)[i];
  // where this page's outliers go: behind those of all blocks and heads before it
  __shared__ int s_off;
  if (tid == 0) s_off = 0;
  __syncthreads();
  const size_t unit0 = unit_index(g, a.layer, a.seq, 0);
  if (g.outlier_k > 0) {
    int before = 0;
    for (int i = tid; i < b * H + head; i += WIRE_THREADS)
      before += (int)a.page_meta[(unit0 + i % H) * g.max_blocks + a.blk0 + i / H].cnt;
    if (before) atomicAdd(&s_off, before);
  }
  uint8_t* dst = a.staging + b * a.parts.bytes;
  if (polar) {
    stream_from_records(pg, dst + a.parts.key + (size_t)head * S * 16 * g.key_bits, S, g.key_bits, tid);
    copy_words(pg + g.scale_off, (float*)(dst + a.parts.scale) + head * S, S, tid);
  } else {
    uint32_t* kd = (uint32_t*)(dst + a.parts.key + (size_t)head * S * 64);
    for (int i = tid; i < S * 16; i += WIRE_THREADS) kd[i] = rev_bytes(((const uint32_t*)pg)[i]);
    copy_words(pg + g.scale_off, (float*)(dst + a.parts.scale) + head * TQ_D, TQ_D, tid);
    copy_words(pg + g.mean_off, (float*)(dst + a.parts.mean) + head * TQ_D, TQ_D, tid);
  }
  stream_from_records(pg + g.v_off, dst + a.parts.val + (size_t)head * S * 16 * g.value_bits, S,
                      g.value_bits, tid);
  copy_words(pg + g.norm_off, (float*)(dst + a.parts.norm) + head * S, S, tid);
  if (g.outlier_k > 0) {
    __syncthreads();
    const PageMeta pm = a.page_meta[(unit0 + head) * g.max_blocks + blk];
    const size_t slab = (unit0 + head) * (size_t)g.pool_entries + pm.off;
    for (uint32_t e = tid; e < pm.cnt; e += WIRE_THREADS) {
      const int64_t o = (int64_t)s_off + e;
      if (o >= a.n_out) break;  // (the counts grew since they were read: never past the buffers)
      const uint32_t w = a.pool_dec[slab + e];
      // the list is ordered by token, then channel, as the flat indices are
      a.out_idx[o] = (head * S + (int)(w >> 24)) * TQ_D + (int)((w >> 16) & 255);
      a.out_val[o] = a.pool_val[slab + e];
    }
  }
}

// Writes the pages, metadata and pool entries of the blocks: what tq_import_block writes, bit for
// bit.  grid = (heads, blocks)
__global__ void __launch_bounds__(WIRE_THREADS) import_kernel(WireArgs a) {
  const tq_geom& g = a.g;
  const int tid = threadIdx.x, head = blockIdx.x, b = blockIdx.y, blk = a.blk0 + b;
  const int S = g.block_tokens, H = g.n_kv_heads, vb = g.value_bits;
  extern __shared__ __align__(16) uint8_t pg[];  // the page image, then the value bit stream
  uint8_t* stream = pg + g.page_bytes;
  __shared__ int s_tok[256], s_ovf[257];  // outliers per token; overflow entries before a token
  for (int i = tid; i < g.page_bytes / 16; i += WIRE_THREADS) ((uint4*)pg)[i] = make_uint4(0, 0, 0, 0);
  s_tok[tid] = 0;
  const uint8_t* src = a.staging + b * a.parts.bytes;
  copy_words(src + a.parts.val + (size_t)head * S * 16 * vb, stream, S * 4 * vb, tid);
  const int first = a.first[b * H + head], n = a.first[b * H + head + 1] - first;
  __syncthreads();
  for (int i = tid; i < n; i += WIRE_THREADS)
    atomicAdd(&s_tok[(a.out_idx[first + i] - head * S * TQ_D) / TQ_D], 1);
  const uint32_t* ks = (const uint32_t*)(src + a.parts.key + (size_t)head * S * 64);
  for (int i = tid; i < S * 16; i += WIRE_THREADS) ((uint32_t*)pg)[i] = rev_bytes(ks[i]);
  float* scale = (float*)(pg + g.scale_off);
  float* mean = (float*)(pg + g.mean_off);
  copy_words((const float*)(src + a.parts.scale) + head * TQ_D, scale, TQ_D, tid);
  copy_words((const float*)(src + a.parts.mean) + head * TQ_D, mean, TQ_D, tid);
  copy_words((const float*)(src + a.parts.norm) + head * S, pg + g.norm_off, S, tid);
  // a lane record of a 16-token group per step: pair p holds tokens (2 (l & 3), + 1) + 8 (p & 1)
  // of channel 8 (p / 2) + l / 4
  for (int i = tid; i < g.block_tokens_pad / TQ_GROUP_TOK * 32; i += WIRE_THREADS) {
    const int gq = i >> 5, l = i & 31;
    uint8_t* grp = pg + g.v_off + (size_t)gq * v_group_bytes(vb);
    unsigned long long acc = 0;
    int have = 0, byte = 0;
    for (int p = 0; p < 32; ++p) {
      const int t = gq * TQ_GROUP_TOK + 8 * (p & 1) + 2 * (l & 3), d = 8 * (p >> 1) + (l >> 2);
      uint32_t pr = t < S ? stream_code(stream, vb, t, d) : 0u;
      if (t + 1 < S) pr |= stream_code(stream, vb, t + 1, d) << vb;
      acc |= (unsigned long long)pr << have;
      have += 2 * vb;
      if (have >= 32) {  // whole words: a record's parts are 8 or 16 bytes
        *(uint32_t*)(grp + v_record_byte_off(vb, l, byte)) = (uint32_t)acc;
        acc >>= 32;
        have -= 32;
        byte += 4;
      }
    }
  }
  __syncthreads();
  // header: the four widest channels (largest scale first, ties to the lower channel)
  PageHeader* hdr = (PageHeader*)(pg + g.hdr_off);
  if (tid < TQ_D) {
    const float mine = scale[tid];
    int rank = 0;
    for (int o = 0; o < TQ_D; ++o) rank += (scale[o] > mine || (scale[o] == mine && o < tid)) ? 1 : 0;
    if (rank < TQ_WIDE) hdr->wide[rank] = (uint8_t)tid;
  }
  // overflow entries before every token
  if (tid < 32) {
    int sum = 0;
    for (int t = 8 * tid; t < 8 * tid + 8; ++t) sum += max(s_tok[t] - TQ_ELL_SLOTS, 0);
    int run = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, run, o);
      if (tid >= o) run += v;
    }
    if (tid == 31) s_ovf[256] = run;
    run -= sum;
    for (int t = 8 * tid; t < 8 * tid + 8; ++t) {
      s_ovf[t] = run;
      run += max(s_tok[t] - TQ_ELL_SLOTS, 0);
    }
  }
  // this page's slice of the pool slab, allocated like the encoder does, block after block
  __shared__ int s_before;
  if (tid == 0) s_before = 0;
  __syncthreads();
  {
    int before = 0;
    for (int i = tid; i < b; i += WIRE_THREADS)
      before += (a.first[i * H + head + 1] - a.first[i * H + head] + 3) & ~3;
    if (before) atomicAdd(&s_before, before);
  }
  if (tid < S) {
    uint32_t side = 0;
#pragma unroll
    for (int rk = 0; rk < TQ_WIDE; ++rk) {
      const int d = hdr->wide[rk];
      side |= (uint32_t)((pg[tid * (TQ_D / 2) + (d >> 1)] >> (4 * (d & 1))) & 15) << (4 * rk);
    }
    ((uint16_t*)(pg + g.hdr_off + TQ_SIDE_OFF))[tid] = (uint16_t)side;
  }
  __syncthreads();
  const size_t unit = unit_index(g, a.layer, a.seq, head);
  uint32_t off = 0;
  int alloc = 0;
  bool lacking = false;
  if (n > 0) {
    const int n4 = (n + 3) & ~3;
    off = a.cursor[head] + (uint32_t)s_before;
    if (off >= (uint32_t)g.pool_entries) off = 0;
    else alloc = min(n4, g.pool_entries - (int)off);
    lacking = alloc < n4;
  }
  const int kept = min(n, alloc);
  const size_t slab = unit * (size_t)g.pool_entries + off;
  uint16_t* ell_delta = (uint16_t*)(pg + g.hdr_off + TQ_ELL_OFF);
  uint8_t* ell_col = pg + g.hdr_off + TQ_ELL_COL_OFF;
  uint32_t* ovf = (uint32_t*)(pg + g.hdr_off + TQ_OVF_OFF);
  for (int i = tid; i < n; i += WIRE_THREADS) {
    const int flat = a.out_idx[first + i] - head * S * TQ_D;
    const int t = flat / TQ_D, d = flat % TQ_D;
    int in_tok = 0;  // entries of the token before this one
    while (in_tok < i && (a.out_idx[first + i - in_tok - 1] - head * S * TQ_D) / TQ_D == t) ++in_tok;
    const int code = (pg[t * (TQ_D / 2) + (d >> 1)] >> (4 * (d & 1))) & 15;
    const float sl = __fmul_rn(scale[d], a.tables->grid[code]);
    const float dense = g.key_mode == TQ_KEYS_NF4 ? sl : __fadd_rn(mean[d], sl);
    const uint16_t hv = a.out_val[first + i];
    const uint16_t delta =
        __half_as_ushort(__float2half_rn(__fsub_rn(__half2float(__ushort_as_half(hv)), dense)));
    const uint32_t ent = (uint32_t)delta | ((uint32_t)d << 16) | ((uint32_t)t << 24);
    if (i < kept) {
      a.pool_dec[slab + i] = ent;
      a.pool_val[slab + i] = hv;
    }
    if (in_tok < TQ_ELL_SLOTS) {
      ell_delta[in_tok * 256 + t] = delta;
      ell_col[in_tok * 256 + t] = (uint8_t)q_row(d);
    } else {
      const int o = s_ovf[t] + in_tok - TQ_ELL_SLOTS;
      if (o < TQ_OVF_CAP) ovf[o] = ent;
    }
  }
  if (tid == 0) {
    const int n_ovf = s_ovf[256];
    for (int q4 = 0; q4 < 5; ++q4) hdr->ovf_start[q4] = (uint16_t)min(s_ovf[64 * q4], TQ_OVF_CAP);
    hdr->ovf_n = (uint16_t)min(n_ovf, TQ_OVF_CAP);
    hdr->off = off;
    hdr->cnt = (uint32_t)kept;
    hdr->flags = (n_ovf > TQ_OVF_CAP || alloc < n) ? TQ_PAGE_SPILLED : 0;
    a.page_meta[unit * g.max_blocks + blk] = {off, (uint32_t)kept};
    if (lacking) atomicOr(a.short_flag, 1);
  }
  __syncthreads();
  uint4* page = (uint4*)(a.pages + page_offset(g, a.layer, a.seq, head, blk));
  for (int i = tid; i < g.page_bytes / 16; i += WIRE_THREADS) page[i] = ((const uint4*)pg)[i];
}

// after the pages: the pool cursors move past the blocks' slices (the pages read the old ones)
__global__ void import_cursor_kernel(WireArgs a) {
  const int head = threadIdx.x + blockIdx.x * blockDim.x, H = a.g.n_kv_heads;
  if (head >= H) return;
  uint32_t add = 0;
  for (int b = 0; b < a.n_blocks; ++b)
    add += (uint32_t)((a.first[b * H + head + 1] - a.first[b * H + head] + 3) & ~3);
  a.cursor[head] += add;
}

WireArgs wire_args(tq_ctx* ctx, int layer, int seq, int blk0, int n_blocks) {
  WireArgs a = {};
  a.g = ctx->g;
  a.parts = wire_parts(ctx->g);
  a.pages = (uint8_t*)ctx->b.pages;
  a.pool_dec = (uint32_t*)ctx->b.pool_dec;
  a.pool_val = (uint16_t*)ctx->b.pool_val;
  a.page_meta = (PageMeta*)ctx->b.page_meta;
  a.cursor = (uint32_t*)((uint8_t*)ctx->b.state + state_cursor_off(ctx->g)) +
             unit_index(ctx->g, layer, seq, 0);
  a.tables = (const Tables*)ctx->b.tables;
  a.layer = layer;
  a.seq = seq;
  a.blk0 = blk0;
  a.n_blocks = n_blocks;
  return a;
}

bool range_ok(const tq_ctx* ctx, int layer, int seq) {
  return ctx != nullptr && layer >= 0 && layer < ctx->g.n_layers && seq >= 0 && seq < ctx->g.n_seqs;
}

template <class K>
int allow_smem(K kernel, int bytes, int device, bool (&set)[64]) {
  TQ_REQUIRE(bytes <= WIRE_SMEM, TQ_ERR_UNSUPPORTED, "a page larger than the wire kernels take");
  if (device >= 64 || !set[device]) {
    TQ_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, WIRE_SMEM));
    if (device < 64) set[device] = true;
  }
  return TQ_OK;
}

}  // namespace

extern "C" {

int32_t tq_wire_parts(const tq_geom* g, int64_t* offsets) {
  TQ_REQUIRE(g != nullptr && offsets != nullptr, TQ_ERR_INVALID, "null argument");
  TQ_REQUIRE(g->page_bytes > 0, TQ_ERR_INVALID, "call tq_geom_finish first");
  const WireParts p = wire_parts(*g);
  const int64_t v[6] = {p.key, p.scale, p.mean, p.val, p.norm, p.bytes};
  for (int i = 0; i < 6; ++i) offsets[i] = v[i];
  return TQ_OK;
}

int32_t tq_outlier_counts(tq_ctx* ctx, int32_t layer, int32_t seq, int32_t block, int32_t n_blocks,
                          int32_t* counts, void* stream) {
  TQ_REQUIRE(range_ok(ctx, layer, seq) && counts != nullptr, TQ_ERR_INVALID, "bad argument");
  const tq_geom& g = ctx->g;
  const int nb = n_cold_blocks(ctx->len[(size_t)layer * g.n_seqs + seq], g.hot_window, g.block_tokens);
  TQ_REQUIRE(block >= 0 && n_blocks >= 0 && block + n_blocks <= nb, TQ_ERR_INVALID,
             "block index out of range");
  for (int b = 0; b < n_blocks; ++b) counts[b] = 0;
  if (n_blocks == 0 || g.outlier_k == 0) return TQ_OK;
  TQ_CUDA(cudaSetDevice(ctx->device));
  cudaStream_t st = (cudaStream_t)stream;
  const int H = g.n_kv_heads;
  std::vector<PageMeta> meta((size_t)H * n_blocks);
  TQ_CUDA(cudaMemcpy2DAsync(
      meta.data(), n_blocks * sizeof(PageMeta),
      (const PageMeta*)ctx->b.page_meta + unit_index(g, layer, seq, 0) * g.max_blocks + block,
      g.max_blocks * sizeof(PageMeta), n_blocks * sizeof(PageMeta), H, cudaMemcpyDeviceToHost, st));
  TQ_CUDA(cudaStreamSynchronize(st));
  for (int h = 0; h < H; ++h)
    for (int b = 0; b < n_blocks; ++b) counts[b] += (int32_t)meta[(size_t)h * n_blocks + b].cnt;
  return TQ_OK;
}

int32_t tq_export_blocks(tq_ctx* ctx, int32_t layer, int32_t seq, int32_t block, int32_t n_blocks,
                         void* staging, int32_t* outlier_idx, uint16_t* outlier_val,
                         int64_t n_outliers, void* stream) {
  TQ_REQUIRE(range_ok(ctx, layer, seq) && staging != nullptr, TQ_ERR_INVALID, "bad argument");
  const tq_geom& g = ctx->g;
  const int nb = n_cold_blocks(ctx->len[(size_t)layer * g.n_seqs + seq], g.hot_window, g.block_tokens);
  TQ_REQUIRE(block >= 0 && n_blocks >= 0 && n_blocks <= 65535 && block + n_blocks <= nb,
             TQ_ERR_INVALID, "block index out of range");
  TQ_REQUIRE(((uintptr_t)staging & 15) == 0, TQ_ERR_INVALID, "staging must be 16-byte aligned");
  TQ_REQUIRE(n_outliers == 0 || (outlier_idx && outlier_val), TQ_ERR_INVALID,
             "outlier buffers missing");
  if (n_blocks == 0) return TQ_OK;
  TQ_CUDA(cudaSetDevice(ctx->device));
  WireArgs a = wire_args(ctx, layer, seq, block, n_blocks);
  a.staging = (uint8_t*)staging;
  a.out_idx = outlier_idx;
  a.out_val = outlier_val;
  a.n_out = n_outliers;
  static bool attr_set[64] = {};  // per device
  const int rc = allow_smem(export_kernel, g.hdr_off, ctx->device, attr_set);
  if (rc != TQ_OK) return rc;
  export_kernel<<<dim3(g.n_kv_heads, n_blocks), WIRE_THREADS, g.hdr_off, (cudaStream_t)stream>>>(a);
  TQ_CUDA(cudaGetLastError());
  return TQ_OK;
}

int32_t tq_import_blocks(tq_ctx* ctx, int32_t layer, int32_t seq, int32_t block, int32_t n_blocks,
                         void* staging, const int32_t* outlier_idx, const uint16_t* outlier_val,
                         const int32_t* first, int32_t* short_flag, void* stream) {
  TQ_REQUIRE(range_ok(ctx, layer, seq), TQ_ERR_INVALID, "bad context, layer or sequence");
  const tq_geom& g = ctx->g;
  TQ_REQUIRE(g.key_mode != TQ_KEYS_POLAR, TQ_ERR_UNSUPPORTED,
             "import of PolarQuant-key blocks is not implemented");
  TQ_REQUIRE(ctx->len[(size_t)layer * g.n_seqs + seq] == 0, TQ_ERR_INVALID,
             "blocks are imported into a cleared cache, before tq_restore_hot sets its length");
  TQ_REQUIRE(block >= 0 && n_blocks >= 0 && n_blocks <= 65535 && block + n_blocks <= g.max_blocks,
             TQ_ERR_CAPACITY, "block index out of range");
  TQ_REQUIRE(staging && first && short_flag && ((uintptr_t)staging & 15) == 0, TQ_ERR_INVALID,
             "null or misaligned argument");
  if (n_blocks == 0) return TQ_OK;
  TQ_CUDA(cudaSetDevice(ctx->device));
  cudaStream_t st = (cudaStream_t)stream;
  WireArgs a = wire_args(ctx, layer, seq, block, n_blocks);
  a.staging = (uint8_t*)staging;
  a.out_idx = const_cast<int32_t*>(outlier_idx);
  a.out_val = const_cast<uint16_t*>(outlier_val);
  a.first = first;
  a.short_flag = short_flag;
  const int smem = g.page_bytes + g.block_tokens * 16 * g.value_bits;
  static bool attr_set[64] = {};  // per device
  const int rc = allow_smem(import_kernel, smem, ctx->device, attr_set);
  if (rc != TQ_OK) return rc;
  TQ_CUDA(cudaMemsetAsync(short_flag, 0, 4, st));
  import_kernel<<<dim3(g.n_kv_heads, n_blocks), WIRE_THREADS, smem, st>>>(a);
  TQ_CUDA(cudaGetLastError());  // (no page written: the cursors stay)
  import_cursor_kernel<<<(g.n_kv_heads + 127) / 128, 128, 0, st>>>(a);
  TQ_CUDA(cudaGetLastError());
  int32_t lacking = 0;
  TQ_CUDA(cudaMemcpyAsync(&lacking, short_flag, 4, cudaMemcpyDeviceToHost, st));
  TQ_CUDA(cudaStreamSynchronize(st));
  TQ_REQUIRE(!lacking, TQ_ERR_CAPACITY, "the outlier pool of this sequence is full");
  return TQ_OK;
}

}  // extern "C"
