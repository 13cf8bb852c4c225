// Value encoder for blocks of 128 or 256 tokens, the rotation on the fifth-generation tensor cores.
// It writes the pages that encode_values_kernel and encode_values_tc5_kernel (encode.cu) write, bit
// for bit:
//   norm = sqrt(pairwise sum of fl(x*x))      (numpy's 8-accumulator order for n = 128)
//   y_ch = sequential, unfused sum over d of fl(x_d / max(norm, 1e-30)) * Pi[ch][d]
//   code = #{ j : boundary_j < y_ch }
//
// One persistent CTA per SM, warps by role.  The roles meet through mbarriers and the counts of the lists, and
// those waits are bounded.  Three others are not: the loaders' named barrier (its eight warps run the same
// loop, whose length follows from the sequence lengths alone), the block barrier at the end (every role
// gets there: its loops are over tiles or bounded waits), and the allocation of tensor memory, which
// waits for other CTAs of this kernel or of encode_values_tc5_kernel on the SM; those free it without
// waiting for any other kernel, and shared memory has room for one of them at a time anyway.
// Warp-wide operations stand only where all lanes decided alike (votes, or one lane's reading).
//
//
// * Eight loader warps copy a tile of 128 tokens (64 for float32) into shared memory with cp.async,
//   two tiles ahead, straight into the tensor cores' operand layout, [16-byte piece][token], which two
//   threads a token also read without bank conflicts for the norm.  16-bit rows are an operand as
//   they are: the product is Pi . X^T and the norm is divided out behind it, so nothing is
//   converted.  (float32 rows are scaled by 4096 / norm and split into two fp16 parts.)
// * One of their threads issues the tcgen05.mma of a tile (M = 128 channels, N = its tokens) into the
//   tile's own columns of tensor memory.
// * Twelve epilogue warps turn the products into codes: lane = channel, column = token.  The rows
//   of Pi are permuted so that a warp's 32 channels fill whole 8-byte pieces of the page's
//   records: no image of the group in shared memory and no barrier, a warp packs 16 tokens x 32
//   channels with four shuffles and stores them itself.
//
// A code takes one table look-up.  z = y scaled to [0, 1) becomes a 23-bit integer Z (the mantissa of
// 1 + z); its top five bits pick one of 32 bins, none of which holds more than one boundary B.  The
// bin's entry (a shuffle: entry k sits in lane k) is ((j + 1) << (32 - bits)) - B, so the sum
// Z + entry has the code in its top bits (the borrow of Z - B takes one off below the boundary) and the
// distance to the boundary in the bits under it: one funnel shift appends the code, one compare
// finds the distances within the slack.
//
// Those products (see VALUE_SLACK) go on a list of the warp's own: (row, destination, norm, channel,
// token, code).  Four more warps take them from there, compute them again in the reference's order, a
// lane per entry, and flip the bits of a code that differs in the page.  (The epilogue warps must not
// do it themselves: a batch takes as long as several tiles, and the other warps would wait at the
// ring of slots.)
//
// What bounds it (8 x 16 384 tokens x 8 heads): at 3 bits (246 us) the logic pipe and the chains of the
// epilogue, 49 % of the issue slots, six warps a scheduler; at 4 bits (328 us in bfloat16) the warps that
// recompute, which wait for rows in global memory and divide.  (With a slack of 1.4e-5, 3 bits, 224 us; of
// that 165 without lists and their recomputation, 124 without codes, products and norms, too, 83 without the
// copies.)
#include <algorithm>
#include <climits>
#include <cmath>

#include "encode.cuh"

namespace {

// The exact dot product lies within 127 * 2^-25 + 2^-23 < 4.0e-6 of the reference's sum (the running
// sum stays below 1: the absolute values of the terms add up to at most |u| |row of Pi| = 1).
// Here Pi is two fp16 parts (what is left is below 2^-23 of a term; of float32 rows likewise) or, for
// bfloat16 rows, three bfloat16 parts (2^-26).  The products with a low part come
// first; their sums stay below 2^-8 and lose next to nothing.  Then the accumulator takes eight steps of
// 16 terms; a step that aligns its 17 addends to the largest of them and cuts them off 24 bits below
// loses at most 17 * 2^-24, 8.2e-6 in all.  Together 1.24e-5.
// How the tensor cores align and cut is not documented, so the slack is two and a half times that, as in
// the other encoders.  (Measured, on 1.1e9 products whose partial sums are large and cancel: a slack of
// zero gives other codes up to 2.2e-7 from a boundary, 7.3e-7 where Pi had two bfloat16 parts.)  Microseconds of an
// append of 8 x 16 384 tokens x 8 heads: fp16, 3 bits, 451 with 1.13 times the bound and 477 with this;
// bfloat16, 4 bits, 617 with two parts of Pi and two and a half times their bound, 563 with three parts.
constexpr float VALUE_SLACK = 3.1e-5f;

constexpr int EV_LOADERS = 256;              // threads of the loader warps
constexpr int EV_EPI_WARPS = 12;
constexpr int EV_REDO_WARPS = 4;
constexpr int EV_THREADS = EV_LOADERS + 32 * (EV_EPI_WARPS + EV_REDO_WARPS);
constexpr int EV_PER_REDO = EV_EPI_WARPS / EV_REDO_WARPS;  // lists a redo warp takes from
constexpr int EV_LIST = 64;                  // entries of a list (a ring)
constexpr int EV_PI_PART = TQ_D * TQ_D * 2;  // bytes of one part of Pi
constexpr int EV_TILE_BYTES = 33280;         // rows of a tile: 128 x 256 or 64 x 512 bytes, and the pads
constexpr int EV_WAIT = 1 << 20;             // probes of a barrier (2 us each at most) before a wait gives up
constexpr int EV_WITHHOLD = 1 << 20;         // test hook: a.withhold_row of tile 0 of the first CTA

template <int DT>
struct EvShape {
  static constexpr bool F32 = DT == TQ_F32;
  static constexpr int T = F32 ? 64 : 128;      // tokens of a tile
  static constexpr int PS = 16 * T + 16;        // bytes from one piece of the rows to the next (padded)
  // Parts of Pi: two of fp16 or three of bfloat16 hold 22 and 24 bits.  (Where there are three, shared memory
  // has room for three tiles.)
  static constexpr int PARTS = DT == TQ_BF16 ? 3 : 2;
  static constexpr int SLOTS = F32 ? 2 : PARTS == 3 ? 3 : 4;  // tiles between loader and epilogue
  static constexpr int RAW = SLOTS;             // row buffers (16-bit: they are the operands)
  static constexpr int TILES = F32 ? 4 : SLOTS; // tile buffers
  static constexpr int COLS = F32 ? 128 : 512;  // columns of tensor memory: SLOTS * T, a power of two
};

struct EvInfo {            // what the epilogue needs to know about a tile
  uint8_t* dst;            // the codes of its first group; null: no more tiles
  float* nrm_dst;
  const void* in0;         // where the row of its token 0 is (or would be) in the caller's tensor
  const void* ring;        // the sequence's and head's ring
  int n_ring, ring0;       // the first n_ring tokens lie in the ring, from slot ring0 on
};

struct EvList {
  const void* row[EV_LIST];
  uint32_t dst[EV_LIST];   // the group's codes, in units of 128 bytes from the first page
  float norm[EV_LIST];
  uint32_t meta[EV_LIST];  // channel | token << 8 | code << 12
};

template <int DT>
struct EvShared {
  alignas(16) uint8_t pi[EvShape<DT>::PARTS * EV_PI_PART];  // Pi as A operand: [hi | lo ...][K / 8][128 rows][8]
  alignas(16) uint8_t tile[EvShape<DT>::TILES][EV_TILE_BYTES];  // rows; float32: two row buffers, two operand buffers
  // per slot and token: z = product * mul + 1/2; -1: no usable norm; -2: a row of zeros
  alignas(16) float mul[4][128];
  float norm[4][128];
  EvList list[EV_EPI_WARPS];
  int put[EV_EPI_WARPS], got[EV_EPI_WARPS], fin[EV_EPI_WARPS];  // entries listed, taken; no more to come
  EvInfo info[4];
  unsigned long long odd[4];  // per slot, a byte per loader warp: it has a token without a usable norm
  unsigned long long full[4], done[4], empty[4];
  uint32_t tmem;
  int lost;  // first tile whose codes or norms are not all there: a wait ran out
};
static_assert(sizeof(EvShared<TQ_F32>) <= 227 * 1024 && sizeof(EvShared<TQ_F16>) <= 227 * 1024 &&
                  sizeof(EvShared<TQ_BF16>) <= 227 * 1024,
              "shared memory of one CTA");

TQ_DEV void ev_cp16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
TQ_DEV void ev_mma(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
      "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
TQ_DEV void ev_tmem_ld16(uint32_t addr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
      "[%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
        "=r"(r[15])
      : "r"(addr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
// a.xy = b.xy * b.xy + a.xy
TQ_DEV void ev_sq2(float2& a, float2 b) {
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %3};\n\t"
      "fma.rn.f32x2 x, y, y, x;\n\tmov.b64 {%0, %1}, x;\n\t}\n"
      : "+f"(a.x), "+f"(a.y)
      : "f"(b.x), "f"(b.y));
}
template <int DT>
TQ_DEV float2 ev_pair(uint32_t h) {
  if (DT == TQ_BF16) return make_float2(__uint_as_float(h << 16), __uint_as_float(h & 0xffff0000u));
  return __half22float2(*(const __half2*)&h);
}
// two neighbouring elements as one word of the hi part and one of the lo part
template <int DT>
TQ_DEV void ev_split(float2 p, uint32_t& hi, uint32_t& lo) {
  if (DT == TQ_BF16) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(p.x, p.y);
    const float2 f = __bfloat1622float2(h);
    const __nv_bfloat162 l = __floats2bfloat162_rn(p.x - f.x, p.y - f.y);
    hi = *(const uint32_t*)&h, lo = *(const uint32_t*)&l;
  } else {
    const __half2 h = __floats2half2_rn(p.x, p.y);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(p.x - f.x, p.y - f.y);
    hi = *(const uint32_t*)&h, lo = *(const uint32_t*)&l;
  }
}

// The products are scaled by powers of two so that the fp16 low parts keep their bits: Pi by 2^8,
// float32 rows to a norm of 2^12.  bfloat16 parts need none.
template <int DT>
TQ_HD float ev_pi_scale() { return DT == TQ_BF16 ? 1.0f : 256.0f; }
constexpr float EV_ROW_NORM = 4096.0f;

template <int DT, int VB>
__global__ void __launch_bounds__(EV_THREADS, 1)
    encode_values_tile_kernel(EncodeArgs a, ValueTable vt) {
  using T_ = typename Elem<DT>::type;
  using Sh = EvShape<DT>;
  constexpr bool F32 = Sh::F32;
  constexpr int T = Sh::T, PS = Sh::PS, SLOTS = Sh::SLOTS;
  constexpr int EPC = 16 / (int)sizeof(T_), CH = TQ_D / EPC;  // elements of a piece, pieces of a row
  constexpr int VGB = TQ_GROUP_TOK * TQ_D * VB / 8;
  const tq_geom& g = a.g;
  extern __shared__ __align__(128) uint8_t ev_smem[];
  using Shared = EvShared<DT>;
  Shared& sh = *(Shared*)ev_smem;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float* pi_rows = a.tables->pi;
  const bool keys = a.polar_keys_pass != 0;
  const void* in_base = keys ? a.k : a.v;
  const void* ring_base = keys ? a.hot_k : a.hot_v;
  const int out_off = keys ? 0 : g.v_off, nrm_off = keys ? g.scale_off : g.norm_off;
  const bool rows_aligned = ((uintptr_t)in_base & 15) == 0 &&
                            ((a.seq_stride | a.tok_stride | a.head_stride) & (EPC - 1)) == 0;

  // Row m of the A operand is channel 8 * (m % 16) + m / 16: element (m, d) of part p at
  // p * 32 KB + (d / 8) * 2 KB + m * 16 + (d % 8) * 2 bytes.  (All loads before the first use.)
  {
    constexpr int N = (TQ_D * TQ_D / 2 + EV_THREADS - 1) / EV_THREADS;
    float2 p[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const int i = min((int)threadIdx.x + k * EV_THREADS, TQ_D * TQ_D / 2 - 1);
      const int m = i >> 6, ch = 8 * (m & 15) + (m >> 4);
      p[k] = *(const float2*)&pi_rows[ch * TQ_D + (i & 63) * 2];
    }
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const int i = min((int)threadIdx.x + k * EV_THREADS, TQ_D * TQ_D / 2 - 1);
      const int m = i >> 6, d = (i & 63) * 2;
      uint32_t hi, lo;
      ev_split<DT>(make_float2(p[k].x * ev_pi_scale<DT>(), p[k].y * ev_pi_scale<DT>()), hi, lo);
      uint32_t* at = (uint32_t*)(sh.pi + (d >> 3) * 2048 + m * 16 + (d & 7) * 2);
      at[0] = hi;
      at[EV_PI_PART / 4] = lo;
      if constexpr (Sh::PARTS == 3) {
        const float2 h = ev_pair<DT>(hi), l = ev_pair<DT>(lo);
        const __nv_bfloat162 r = __floats2bfloat162_rn(p[k].x - h.x - l.x, p[k].y - h.y - l.y);
        at[EV_PI_PART / 2] = *(const uint32_t*)&r;
      }
    }
  }
  if (threadIdx.x < SLOTS) {
    const int s = threadIdx.x;
    mbar_init(enc_smem(&sh.full[s]), EV_LOADERS);
    mbar_init(enc_smem(&sh.done[s]), 1);
    mbar_init(enc_smem(&sh.empty[s]), EV_EPI_WARPS);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x < EV_EPI_WARPS)
    sh.put[threadIdx.x] = sh.got[threadIdx.x] = sh.fin[threadIdx.x] = 0;
  if (threadIdx.x == 0) sh.lost = INT_MAX;
  if (warp == 0) {
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     enc_smem(&sh.tmem)),
                 "r"(Sh::COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // Pi is read by the tensor cores
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *(volatile uint32_t*)&sh.tmem;

  const int limit = a.wait_limit > 0 ? min(a.wait_limit, 1 << 26) : EV_WAIT;
  auto lose = [&](int i) {  // a wait for tile i ran out
    atomicOr(a.status, TQ_STATUS_WAIT_TIMEOUT);
    atomicMin(&sh.lost, i);
  };
  bool gave_up = false;  // (no later wait of this thread probes again)
  // bounded wait for the phase of `bars` that tile i completes
  auto wait = [&](unsigned long long* bars, int i) {
    if (gave_up) return;
    const uint32_t bar = enc_smem(&bars[i % SLOTS]);
    const unsigned parity = (unsigned)((i / SLOTS) & 1);
    for (int n = 0; !mbar_try_wait(bar, parity);) {
      if (++n >= limit) {
        lose(i);
        gave_up = true;
        break;
      }
    }
    gave_up = __any_sync(0xffffffffu, gave_up);  // (a warp's lanes stay together)
  };

  if (warp < EV_LOADERS / 32) {
    // ---- loaders ---------------------------------------------------------------------------
    const int tl = threadIdx.x;
    auto sync = [&]() { asm volatile("bar.sync 1, %0;" ::"n"(EV_LOADERS) : "memory"); };
    // tiles w = ((seq * heads + head) * blocks + jb) * parts + part, w = first, first + grid, ...:
    // the four indices are stepped with carries; tiles of blocks this call does not flush are
    // skipped
    const int parts = g.block_tokens / T;
    int part_n, jb_n, head_n, seq_n, step[4];
    auto digits = [&](int w, int& p, int& j, int& h, int& s) {
      p = w % parts, w /= parts;
      j = w % a.max_new_blocks, w /= a.max_new_blocks;
      h = w % g.n_kv_heads, s = w / g.n_kv_heads;
    };
    digits(blockIdx.x, part_n, jb_n, head_n, seq_n);
    digits(gridDim.x, step[0], step[1], step[2], step[3]);
    int seq_known = -1, n0 = 0, nb0 = 0, nb1 = 0;
    // finds tile i, notes it in info[i % 4] and starts the copies of its rows; false when there is none
    auto fetch = [&](int i) -> bool {
      while (seq_n < a.seq_count) {
        const int part = part_n, jb = jb_n, head = head_n, seq = a.seq_begin + seq_n;
        part_n += step[0];
        int c = part_n >= parts ? 1 : 0;
        part_n -= c ? parts : 0;
        jb_n += step[1] + c;
        c = jb_n >= a.max_new_blocks ? 1 : 0;
        jb_n -= c ? a.max_new_blocks : 0;
        head_n += step[2] + c;
        c = head_n >= g.n_kv_heads ? 1 : 0;
        head_n -= c ? g.n_kv_heads : 0;
        seq_n += step[3] + c;
        if (seq != seq_known) {
          n0 = a.seq_len[a.layer * g.n_seqs + seq];
          nb0 = n_cold_blocks(n0, g.hot_window, g.block_tokens);
          nb1 = n_cold_blocks(n0 + a.n_tokens, g.hot_window, g.block_tokens);
          seq_known = seq;
        }
        const int blk = nb0 + jb;
        if (blk >= nb1) continue;
        const TokenSource<DT> src = make_source<DT>(a, ring_base, in_base, seq, head, n0);
        const int pos0 = blk * g.block_tokens + part * T;
        const int n_ring = min(max(n0 - pos0, 0), T), ring0 = n_ring > 0 ? pos0 % src.cap : 0;
        const T_* in0 = (const T_*)src.in + (int64_t)(pos0 - n0) * src.tok_stride;
        if (!F32 && i >= SLOTS) wait(sh.empty, i - SLOTS);  // (float32: the row buffer is free)
        if (tl == 0) {
          uint8_t* page = a.pages + page_offset(g, a.layer, seq, head, blk);
          EvInfo& nf = sh.info[i & 3];
          nf.dst = page + out_off + (size_t)part * (T / TQ_GROUP_TOK) * VGB;
          nf.nrm_dst = (float*)(page + nrm_off) + part * T;
          nf.in0 = in0, nf.ring = src.ring;
          nf.n_ring = n_ring, nf.ring0 = ring0;
        }
        // Piece p of token t goes to p * PS + t * 16; a half warp (float32: a warp) copies a whole row.
        // (The pad spreads the pieces of a row over the banks.)
        constexpr int RPI = EV_LOADERS / CH;  // rows of an iteration
        const int p = tl % CH, t8 = tl / CH;
        uint8_t* buf = sh.tile[i % Sh::RAW] + p * PS + t8 * 16;
        if (rows_aligned && n_ring == 0) {
          const T_* row = in0 + (int64_t)t8 * src.tok_stride + p * EPC;
          const int64_t next = (int64_t)RPI * src.tok_stride;
          const uint32_t to = enc_smem(buf);
#pragma unroll
          for (int it = 0; it < T / RPI; ++it) {
            ev_cp16(to + it * (16 * RPI), row);
            row += next;
          }
        } else {
#pragma unroll 1
          for (int it = 0; it < T / RPI; ++it, buf += 16 * RPI) {
            const int t = t8 + it * RPI;
            int slot = ring0 + t;
            slot -= slot >= src.cap ? src.cap : 0;
            const T_* row = (t < n_ring ? (const T_*)src.ring + (size_t)slot * TQ_D
                                        : in0 + (int64_t)t * src.tok_stride) + p * EPC;
            if (rows_aligned) {
              ev_cp16(enc_smem(buf), row);
            } else {
              alignas(16) T_ x[EPC];
#pragma unroll
              for (int q = 0; q < EPC; ++q) x[q] = row[q];
              *(uint4*)buf = *(const uint4*)x;
            }
          }
        }
        return true;
      }
      return false;
    };
    auto commit = [&]() { asm volatile("cp.async.commit_group;" ::: "memory"); };

    // products of tile i: columns (i % SLOTS) * T on
    constexpr uint32_t fmt = DT == TQ_BF16 ? 1u : 0u;
    constexpr uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(T >> 3) << 17) |
                               ((128u >> 4) << 24);
    auto issue = [&](int i) {
      if (blockIdx.x == 0 && a.withhold_row - EV_WITHHOLD == i) return;  // test hook
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t d = tmem + (uint32_t)((i % SLOTS) * T);
      const uint64_t a_hi0 = umma_desc_k_major(enc_smem(sh.pi), 2048, 128);
      const uint64_t a_lo0 = umma_desc_k_major(enc_smem(sh.pi) + EV_PI_PART, 2048, 128);
      const uint64_t b0 = umma_desc_k_major(
          enc_smem(sh.tile[F32 ? 2 + i % 2 : i % Sh::TILES]), PS, 128);
      constexpr uint64_t KA = 4096 >> 4, KB = 2 * PS >> 4;  // a step of 16 input channels
      // the small products first (see VALUE_SLACK)
      if constexpr (Sh::PARTS == 3) {
        const uint64_t a_rest0 = umma_desc_k_major(enc_smem(sh.pi) + 2 * EV_PI_PART, 2048, 128);
#pragma unroll
        for (int kb = 0; kb < 8; ++kb) ev_mma(d, a_rest0 + kb * KA, b0 + kb * KB, idesc, kb > 0);
      }
#pragma unroll
      for (int kb = 0; kb < 8; ++kb) {
        ev_mma(d, a_lo0 + kb * KA, b0 + kb * KB, idesc, kb > 0 || Sh::PARTS == 3);
        if (F32) ev_mma(d, a_hi0 + kb * KA, b0 + kb * KB + (EV_TILE_BYTES / 2 >> 4), idesc, 1u);
      }
#pragma unroll
      for (int kb = 0; kb < 8; ++kb) ev_mma(d, a_hi0 + kb * KA, b0 + kb * KB, idesc, 1u);
      umma_commit(enc_smem(&sh.done[i % SLOTS]));
    };

    int n = 0;  // tiles started
    bool more = true;
    for (int i = 0; i < 2; ++i) {
      if (more && fetch(n)) ++n;
      else more = false;
      commit();
    }
    for (int i = 0; i < n; ++i) {
      const int slot = i % SLOTS;
      if (!F32) {
        // With three slots the next copies start behind this tile's products: they wait for the epilogue of
        // the tile before it.
        if (SLOTS > 3) {
          if (more && fetch(n)) ++n;
          else more = false;
          commit();
          asm volatile("cp.async.wait_group 2;" ::: "memory");
        } else {
          asm volatile("cp.async.wait_group 1;" ::: "memory");
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        sync();
        if (tl == 0) issue(i);
        // the norm, two threads a token: accumulators 4h .. 4h + 3 (j takes elements j, j + 8, ...)
        const int t = tl >> 1, h = tl & 1;
        const uint8_t* buf = sh.tile[i % Sh::RAW] + t * 16 + h * 8;
        float2 r[2] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
        // (the square of a 16-bit number is exact in float32, so the fused form rounds as the
        // unfused one does - above the denormals: see below)
#pragma unroll 4
        for (int p = 0; p < CH; ++p) {
          const uint2 v = *(const uint2*)(buf + p * PS);
          ev_sq2(r[0], ev_pair<DT>(v.x));
          ev_sq2(r[1], ev_pair<DT>(v.y));
        }
        auto total = [&]() {
          const float s = __fadd_rn(__fadd_rn(r[0].x, r[0].y), __fadd_rn(r[1].x, r[1].y));
          return __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, 1));
        };
        float sq = total();
        uint32_t any = 1u;  // an element that is not zero
        if (__any_sync(0xffffffffu, sq < 1e-27f)) {  // (bfloat16) squares below 2^-126 are rounded: unfused
          any = 0u;
          r[0] = r[1] = make_float2(0.0f, 0.0f);
          for (int p = 0; p < CH; ++p) {
            const uint2 v = *(const uint2*)(buf + p * PS);
            any |= (v.x | v.y) & 0x7fff7fffu;
            const float2 f0 = ev_pair<DT>(v.x), f1 = ev_pair<DT>(v.y);
            r[0].x = __fadd_rn(r[0].x, __fmul_rn(f0.x, f0.x));
            r[0].y = __fadd_rn(r[0].y, __fmul_rn(f0.y, f0.y));
            r[1].x = __fadd_rn(r[1].x, __fmul_rn(f1.x, f1.x));
            r[1].y = __fadd_rn(r[1].y, __fmul_rn(f1.y, f1.y));
          }
          sq = total();
          any |= __shfl_xor_sync(0xffffffffu, any, 1);
        }
        const float nrm = __fsqrt_rn(sq);
        // A tiny, huge or unordered norm is marked: every channel goes on the list.  A row of zeros (all
        // its sums are zero) is marked, too.
        const bool sane = nrm > 0x1p-40f && nrm < 0x1p+60f;
        if (h == 0) {
          sh.info[i & 3].nrm_dst[t] = nrm;
          sh.norm[slot][t] = nrm;
          sh.mul[slot][t] =
              sane ? __fdividef(vt.scale / ev_pi_scale<DT>(), nrm) : any == 0u ? -2.0f : -1.0f;
        }
        const bool all_sane = __all_sync(0xffffffffu, sane);
        if (lane == 0) ((uint8_t*)&sh.odd[slot])[warp] = all_sane ? 0 : 1;
        if (SLOTS == 3) {
          mbar_arrive(enc_smem(&sh.full[slot]));
          if (more && fetch(n)) ++n;
          else more = false;
          commit();
          continue;
        }
      } else {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        sync();
        // four threads a token: accumulators 2u and 2u + 1, elements 8p + 2u and 8p + 2u + 1 of its row
        const int t = 8 * warp + ((lane >> 1) & 7), u = 2 * (lane >> 4) + (lane & 1);
        const uint8_t* buf = sh.tile[i % Sh::RAW] + (u >> 1) * PS + t * 16 + (u & 1) * 8;
        float2 x[CH / 2], r;
#pragma unroll
        for (int p = 0; p < CH / 2; ++p) x[p] = *(const float2*)(buf + p * 2 * PS);
        uint32_t any = 0u;  // an element that is not zero
#pragma unroll
        for (int p = 0; p < CH / 2; ++p) {
          const float2 q = make_float2(__fmul_rn(x[p].x, x[p].x), __fmul_rn(x[p].y, x[p].y));
          r = p == 0 ? q : make_float2(__fadd_rn(r.x, q.x), __fadd_rn(r.y, q.y));
          any |= __float_as_uint(x[p].x) | __float_as_uint(x[p].y);
        }
        float sq = __fadd_rn(r.x, r.y);
        sq = __fadd_rn(sq, __shfl_xor_sync(0xffffffffu, sq, 1));
        sq = __fadd_rn(sq, __shfl_xor_sync(0xffffffffu, sq, 16));
        any |= __shfl_xor_sync(0xffffffffu, any, 1);
        any |= __shfl_xor_sync(0xffffffffu, any, 16);
        const float nrm = __fsqrt_rn(sq);
        const bool sane = nrm > 0x1p-40f && nrm < 0x1p+60f;
        const float up = sane ? EV_ROW_NORM / nrm : 0.0f;
        if (i >= SLOTS) wait(sh.empty, i - SLOTS);  // operand buffer, slot and columns are free
        uint8_t* op = sh.tile[2 + i % 2] + t * 16 + u * 4;
#pragma unroll
        for (int p = 0; p < CH / 2; ++p)
          ev_split<DT>(make_float2(x[p].x * up, x[p].y * up), *(uint32_t*)(op + p * PS),
                       *(uint32_t*)(op + EV_TILE_BYTES / 2 + p * PS));
        if (u == 0) {
          sh.info[i & 3].nrm_dst[t] = nrm;
          sh.norm[slot][t] = nrm;
          sh.mul[slot][t] = sane ? vt.scale / (ev_pi_scale<DT>() * EV_ROW_NORM)
                            : (any & 0x7fffffffu) == 0u ? -2.0f : -1.0f;
        }
        const bool all_sane = __all_sync(0xffffffffu, sane);
        if (lane == 0) ((uint8_t*)&sh.odd[slot])[warp] = all_sane ? 0 : 1;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        sync();  // (every thread is done with the row buffer, too)
        if (tl == 0) issue(i);
        if (more && fetch(n)) ++n;
        else more = false;
        commit();
      }
      mbar_arrive(enc_smem(&sh.full[slot]));
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (n >= SLOTS) wait(sh.empty, n - SLOTS);
    if (tl == 0) sh.info[n & 3].dst = nullptr;
    mbar_arrive(enc_smem(&sh.full[n % SLOTS]));
    for (int i = max(n - SLOTS, 0); i < n; ++i) {  // no product is under way when the tensor memory goes back
      gave_up = false;
      wait(sh.done, i);
    }
  } else if (warp < EV_LOADERS / 32 + EV_EPI_WARPS) {
    // ---- epilogue --------------------------------------------------------------------------
    // tensor-memory lanes 32 wq on; of the groups of all tiles every third
    constexpr int WGS = EV_EPI_WARPS / 4, NG = T / TQ_GROUP_TOK;
    const int wq = warp & 3;
    int first = (warp - EV_LOADERS / 32) >> 2;  // this warp's first group of the tile
    const int i16 = lane & 15, qd = i16 >> 2, s4 = i16 & 3;
    const int rr = 2 * wq + (lane >> 4), ch = 8 * i16 + rr;  // this lane's channel
    const int tab = vt.off[lane];
    const uint32_t near_add = vt.slack << VB, near_lim = 2u * near_add;
    const int ew = warp - EV_LOADERS / 32;
    EvList& li = sh.list[ew];
    // entries written, told to the warp that takes them, and taken by it as far as this warp knows (the
    // same in every lane)
    int put = 0, told = 0, seen = 0;
    auto publish = [&]() {
      __syncwarp();
      if (lane == 0) {  // (a group's codes are in the page before its entries are seen)
        __threadfence_block();
        *(volatile int*)&sh.put[ew] = put;
      }
      told = put;
    };
    // selectors of the transpose (below)
    const uint32_t sel1 = s4 & 1 ? 0x7632u : 0x5410u;
    const uint32_t sel_lo = (s4 & 1 ? 0x1054u : 0x5410u) ^ (s4 & 2 ? 0x2222u : 0u);
    // where this lane's piece of a group's records goes
    const int l_out = rr * 4 + s4;
    const int out = VB == 4 ? (qd >> 1) * 512 + l_out * 16 + (qd & 1) * 8 : qd * 256 + l_out * 8;

    for (int i = 0;; ++i) {
      const int slot = i % SLOTS;
      wait(sh.full, i);
      if (gave_up) break;
      const EvInfo& nf = sh.info[i & 3];
      uint8_t* const tile_dst = nf.dst;
      if (tile_dst == nullptr) break;
      wait(sh.done, i);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const bool odd = sh.odd[slot] != 0ull;
#pragma unroll 1
      for (; first < NG; first += WGS) {
        const int gq = first;
        float y[16];
        ev_tmem_ld16(tmem + (uint32_t)(slot * T + gq * TQ_GROUP_TOK) + ((uint32_t)(32 * wq) << 16), y);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        const float* mul = &sh.mul[slot][gq * TQ_GROUP_TOK];
        // the word of record lanes 2k, 2k + 1 takes, from the top, tokens 2c + 9, 2c + 8, 2c + 1, 2c
        // of c = 2k + 1, then of c = 2k
        uint32_t word[2], near = 0u;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          uint32_t acc = 0u;
          const float4 m0 = *(const float4*)(mul + 4 * k), m1 = *(const float4*)(mul + 8 + 4 * k);
          const float mu[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};  // tokens 4k .., 8 + 4k ..
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int c = 2 * k + (j < 4 ? 1 : 0);
            const int t = 2 * c + ((j & 1) ^ 1) + ((j & 3) < 2 ? 8 : 0);
            const float z = __saturatef(fmaf(y[t], mu[(t & 3) + (t >> 3) * 4], 0.5f));
            const float m = fmaf(z, VALUE_SPAN, 1.0f);
            const int bin = __float_as_int(__fadd_rz(m, 262144.0f));  // (its low five bits)
            const uint32_t w = __float_as_uint(m) + (uint32_t)__shfl_sync(0xffffffffu, tab, bin);
            if (VB == 3 && j == 4) acc <<= 4;
            acc = __funnelshift_l(w, acc, VB);
            if ((w << VB) + near_add < near_lim) near |= 1u << (8 * k + j);
          }
          word[k] = acc;
        }
        if (odd) {
#pragma unroll
          for (int b = 0; b < 16; ++b) {
            const int j = b & 7, c = 2 * (b >> 3) + (j < 4 ? 1 : 0);
            const int t = 2 * c + ((j & 1) ^ 1) + ((j & 3) < 2 ? 8 : 0);
            const int at = VB == 4 ? 28 - 4 * j : (j < 4 ? 16 : 0) + 9 - 3 * (j & 3);
            const float mt = mul[t];
            if (mt == -1.0f) near |= 1u << b;
            if (mt == -2.0f) {
              near &= ~(1u << b);
              word[b >> 3] = (word[b >> 3] & ~(((1u << VB) - 1u) << at)) | (vt.zero_code << at);
            }
          }
        }
        // Lane i16 has the fields c = 0..3 of channel group i16; record (rr, c) wants them of all 16.
        // Transposed in quads of lanes: lane 4 qd + c gets fields c of channel groups 4 qd .. 4 qd + 3.
        const uint32_t keep = s4 & 2 ? word[1] : word[0], give = s4 & 2 ? word[0] : word[1];
        const uint32_t got = __shfl_xor_sync(0xffffffffu, give, 2);
        const uint32_t own = __byte_perm(keep, got, sel1);
        const uint32_t oth = __shfl_xor_sync(0xffffffffu, __byte_perm(keep, got, sel1 ^ 0x2222u), 1);
        uint32_t lo = __byte_perm(own, oth, sel_lo), hi = __byte_perm(own, oth, sel_lo ^ 0x2222u);
        uint8_t* dst = tile_dst + gq * VGB;
        if (VB == 4) {
          *(uint2*)(dst + out) = make_uint2(lo, hi);
        } else {
          // four fields of 12 bits: 48 bits, and from the next quad what completes 64
          lo = (lo & 0xfffu) | ((lo >> 4) & 0xfff000u);
          hi = (hi & 0xfffu) | ((hi >> 4) & 0xfff000u);
          const uint64_t mine = (uint64_t)(lo | (hi << 24)) | ((uint64_t)(hi >> 8) << 32);
          const uint64_t next = __shfl_down_sync(0xffffffffu, mine, 4);
          if (qd < 3) *(uint64_t*)(dst + out) = (mine >> (16 * qd)) | (next << (48 - 16 * qd));
        }
        // products near a boundary go on the list
        unsigned todo = __ballot_sync(0xffffffffu, near != 0u);
        while (todo) {
          const int n = __popc(todo);
          if (put + n - seen > EV_LIST) {
            if (put != told) publish();
            for (int k = 0;; ++k) {
              // (one lane's reading, so that the warp decides as one: the taking warp writes it meanwhile)
              seen = __shfl_sync(0xffffffffu, *(volatile int*)&sh.got[ew], 0);
              if (gave_up || put + n - seen <= EV_LIST) break;
              if (k >= 16 * limit) {
                if (lane == 0) lose(i);
                gave_up = true;
              }
              __nanosleep(100);
            }
            __threadfence_block();  // (what those entries held has been read)
          }
          if (gave_up) break;
          if (near) {
            const int b = __ffs((int)near) - 1, j = b & 7, jj = j & 3;
            near &= near - 1;
            const int c = 2 * (b >> 3) + ((j >> 2) ^ 1);
            const int t = 2 * c + ((jj & 1) ^ 1) + (jj < 2 ? 8 : 0), tt = gq * TQ_GROUP_TOK + t;
            const uint32_t wd = b & 8 ? word[1] : word[0];
            const uint32_t code = VB == 4 ? wd >> (28 - 4 * j) & 15u
                                          : wd >> ((j < 4 ? 16 : 0) + 9 - 3 * jj) & 7u;
            int sl = nf.ring0 + tt;
            sl -= sl >= g.hot_cap ? g.hot_cap : 0;
            const int at = (put + __popc(todo & ((1u << lane) - 1u))) & (EV_LIST - 1);
            li.row[at] = tt < nf.n_ring ? (const void*)((const T_*)nf.ring + (size_t)sl * TQ_D)
                                        : (const void*)((const T_*)nf.in0 + (int64_t)tt * a.tok_stride);
            li.dst[at] = (uint32_t)((size_t)(dst - a.pages) >> 7);
            li.norm[at] = sh.norm[slot][tt];
            li.meta[at] = (uint32_t)ch | ((uint32_t)t << 8) | (code << 12);
          }
          put += n;
          todo = __ballot_sync(0xffffffffu, near != 0u);
        }
      }
      first -= NG;
      if (put != told) publish();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(enc_smem(&sh.empty[slot]));
    }
    __syncwarp();
    if (lane == 0) {
      __threadfence_block();
      *(volatile int*)&sh.fin[ew] = 1;
    }
  } else {
    // ---- listed products -------------------------------------------------------------------
    const int rw = warp - EV_LOADERS / 32 - EV_EPI_WARPS, p0 = rw * EV_PER_REDO;
    constexpr int n_bnd = (1 << VB) - 1;
    const float* bnd = a.tables->boundaries;
    auto fix = [&](uint32_t dst, uint32_t meta, int cd) {  // code cd for the one that was stored
      const int c2 = (int)(meta & 255u), t2 = (int)((meta >> 8) & 15u);
      const uint32_t delta = (uint32_t)cd ^ (meta >> 12);
      if (delta) {
        const int l = v_lane(t2, c2), bit = 2 * VB * v_pair(t2, c2) + VB * (t2 & 1);
        const uint32_t v = delta << (bit & 7);
        uint32_t* d32 = (uint32_t*)(a.pages + (size_t)dst * 128);
        const int off0 = v_record_byte_off(VB, l, bit >> 3);
        if (v & 255u) atomicXor(&d32[off0 >> 2], (v & 255u) << ((off0 & 3) * 8));
        if (v >> 8) {
          const int off1 = v_record_byte_off(VB, l, (bit >> 3) + 1);
          atomicXor(&d32[off1 >> 2], (v >> 8) << ((off1 & 3) * 8));
        }
      }
    };
    auto load8 = [&](const T_* row, int d0, float (&x)[8]) {
      if (rows_aligned) {
        uint4 rw4[8 / EPC];
#pragma unroll
        for (int k = 0; k < 8 / EPC; ++k) rw4[k] = *(const uint4*)(row + d0 + k * EPC);
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = Elem<DT>::ld((const T_*)rw4, k);
      } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = Elem<DT>::ld(row, d0 + k);
      }
    };
    auto load_pi8 = [&](const float* pr, int d0, float (&pv)[8]) {
      const float4 x = __ldg((const float4*)(pr + d0)), y = __ldg((const float4*)(pr + d0 + 4));
      pv[0] = x.x, pv[1] = x.y, pv[2] = x.z, pv[3] = x.w, pv[4] = y.x, pv[5] = y.y, pv[6] = y.z, pv[7] = y.w;
    };
    int got[EV_PER_REDO];
#pragma unroll
    for (int k = 0; k < EV_PER_REDO; ++k) got[k] = 0;
    for (int idle = 0;;) {
      // what the lists hold: a batch of up to 32 entries in list order (the ends are read before the
      // counts, so a count read after the last end is final)
      bool all_fin = true;
      int avail[EV_PER_REDO], total = 0;
#pragma unroll
      for (int k = 0; k < EV_PER_REDO; ++k) all_fin &= *(volatile int*)&sh.fin[p0 + k] != 0;
      all_fin = __all_sync(0xffffffffu, all_fin);
      __threadfence_block();
#pragma unroll
      for (int k = 0; k < EV_PER_REDO; ++k) {
        avail[k] = __shfl_sync(0xffffffffu, *(volatile int*)&sh.put[p0 + k], 0) - got[k];
        total += avail[k];
      }
      __threadfence_block();
      if (total < 32 && !all_fin) {
        if (++idle >= 4 * limit) {
          if (lane == 0) lose(0);
          break;
        }
        __nanosleep(2000);
        continue;
      }
      if (total == 0) break;  // (and nothing more to come)
      idle = 0;
      // lane i takes the i-th of them
      int list = -1, at = lane;
#pragma unroll
      for (int k = 0; k < EV_PER_REDO; ++k) {
        if (list < 0 && at < avail[k]) {
          list = p0 + k;
          at += got[k];
        } else if (list < 0) {
          at -= avail[k];
        }
      }
      const T_* row = nullptr;
      uint32_t dst = 0u, meta = 0u;
      float safe = 1.0f;
      if (list >= 0) {
        const EvList& li = sh.list[list];
        at &= EV_LIST - 1;
        row = (const T_*)li.row[at];
        dst = li.dst[at];
        meta = li.meta[at];
        safe = fmaxf(li.norm[at], 1e-30f);
      }
      __syncwarp();
      int left = 32;
#pragma unroll
      for (int k = 0; k < EV_PER_REDO; ++k) {  // the entries have been read
        const int n = min(avail[k], left);
        left -= n;
        got[k] += n;
        if (lane == 0 && n > 0) {
          __threadfence_block();
          *(volatile int*)&sh.got[p0 + k] = got[k];
        }
      }
      if (list >= 0) {
        // the exact sum in the reference's order: the quotients and products rounded one by one,
        // added up in sequence
        const float* pr = pi_rows + (meta & 255u) * TQ_D;
        float yy = 0.0f;
#pragma unroll 2
        for (int d0 = 0; d0 < TQ_D; d0 += 8) {
          float x[8], pv[8], pd[8];
          load8(row, d0, x);
          load_pi8(pr, d0, pv);
#pragma unroll
          for (int k = 0; k < 8; ++k) pd[k] = __fmul_rn(__fdiv_rn(x[k], safe), pv[k]);
          // ((p0 + p1) + p2) + ... : the first product starts the sum
          yy = d0 == 0 ? pd[0] : __fadd_rn(yy, pd[0]);
#pragma unroll
          for (int k = 1; k < 8; ++k) yy = __fadd_rn(yy, pd[k]);
        }
        int cd = 0;
        for (int j = 0; j < n_bnd; ++j) cd += (bnd[j] < yy) ? 1 : 0;
        fix(dst, meta, cd);
      }
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Sh::COLS)
                 : "memory");
  }
  if (sh.lost != INT_MAX) {
    // What a wait gave up on, and this CTA's tiles after it, are stored as rows of zeros: the pages may hold
    // anything where no codes were written.
    int i = 0;
    for (long w = blockIdx.x;; w += gridDim.x) {
      const int parts = g.block_tokens / T, part = (int)(w % parts), jb = (int)(w / parts % a.max_new_blocks);
      const long unit = w / parts / a.max_new_blocks;
      if (unit >= (long)a.seq_count * g.n_kv_heads) break;
      const int head = (int)(unit % g.n_kv_heads), seq = a.seq_begin + (int)(unit / g.n_kv_heads);
      const int n0 = a.seq_len[a.layer * g.n_seqs + seq];
      const int blk = n_cold_blocks(n0, g.hot_window, g.block_tokens) + jb;
      if (blk >= n_cold_blocks(n0 + a.n_tokens, g.hot_window, g.block_tokens) || i++ < sh.lost) continue;
      uint8_t* page = a.pages + page_offset(g, a.layer, seq, head, blk);
      uint4* codes = (uint4*)(page + out_off + (size_t)part * (T / TQ_GROUP_TOK) * VGB);
      for (int k = threadIdx.x; k < T / TQ_GROUP_TOK * VGB / 16; k += EV_THREADS) codes[k] = make_uint4(0, 0, 0, 0);
      if (threadIdx.x < T) ((float*)(page + nrm_off))[part * T + threadIdx.x] = 0.0f;
    }
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");  // (the kernel before this one, see the launch)
}

// Microseconds of the value encoder, groups of 16 tokens (encode_values_tc5_kernel) / this one: 8 x 16 384 fp16
// tokens x 8 heads, 3 bits, 561 / 246; bf16, 4 bits, 616 / 328, 3 bits 563 / 250.  Of a whole append, where this
// one starts under the key encoder: 814 / 477, 870 / 563, 819 / 485; 4 001 float32 tokens x 32 heads, 4 bits,
// 164 / 131; 3 333 bf16 tokens x 8 heads, 4 bits, 58 / 46; 4 x 1 010, 3 bits, 58 / 46; one block of 8 heads 48 / 31.
template <int DT, int VB>
int launch_tiles(const EncodeArgs& a, const ValueTable& vt, bool after_keys, int sm_count, int device,
                 cudaStream_t st) {
  static bool attr_set[16] = {};  // per device: the attribute belongs to the device's context
  if (!attr_set[device & 15]) {
    TQ_CUDA(cudaFuncSetAttribute(encode_values_tile_kernel<DT, VB>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(EvShared<DT>)));
    attr_set[device & 15] = true;
  }
  const long total = (long)a.seq_count * a.g.n_kv_heads * a.max_new_blocks *
                     (a.g.block_tokens / EvShape<DT>::T);
  // It may start while the key encoder before it in the stream drains (they share no output); it ends
  // after that kernel has, so that the ring writer, which waits for this one, follows both.
  // (An append of 3 333 bf16 tokens x 8 heads 53 -> 47 us, 4 001 float32 tokens x 32 heads 138 -> 132, 8 x 16 384
  // fp16 tokens 484 -> 475, with the slack that was smaller then.)
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)std::min<long>(total, sm_count));
  cfg.blockDim = dim3(EV_THREADS);
  cfg.dynamicSmemBytes = sizeof(EvShared<DT>);
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = after_keys ? 1 : 0;
  TQ_CUDA(cudaLaunchKernelEx(&cfg, encode_values_tile_kernel<DT, VB>, a, vt));
  return TQ_OK;
}

}  // namespace

void tq_value_table(const float* boundaries, int bits, ValueTable* vt) {
  // the widest range of y that holds all boundaries and whose 32 bins hold at most one each, with the slack
  // on both sides
  const int n = (1 << bits) - 1;
  vt->ok = false;
  for (int i = 0; i < n; ++i)
    if (!(std::fabs(boundaries[i]) < 1.0f) || (i > 0 && !(boundaries[i] > boundaries[i - 1]))) return;
  for (double range = 1.0; range > 0.02 && !vt->ok; range *= 0.99) {
    const double unit = VALUE_SPAN * 8388608.0 / (2.0 * range);  // Z per y
    const long slack = (long)std::ceil(VALUE_SLACK * unit) + 2;
    long at[15];
    int touched = 0;  // last bin the boundaries so far can lie in; the first and the last bin have none
    bool fits = slack < (1 << 17);
    for (int i = 0; i < n && fits; ++i) {
      at[i] = std::lround((boundaries[i] + range) * unit);
      const long first = ((at[i] - 2 * slack + (1 << 18) - 1) >> 18) - 1;
      fits = first > touched;
      touched = (int)((at[i] + 2 * slack) >> 18);
    }
    if (!fits || touched > 30) continue;
    const int sh = 32 - bits;
    for (int k = 0; k < 32; ++k) {
      const long lo = (long)k << 18, hi = lo + (1 << 18);
      int below = 0, which = -1;
      for (int i = 0; i < n; ++i) {
        if (at[i] >= lo - 2 * slack && at[i] <= hi + 2 * slack) which = i;
        else if (at[i] < lo) ++below;
      }
      const int64_t base = which >= 0 ? ((int64_t)(which + 1) << sh) - at[which]
                                      : ((int64_t)below << sh) + (1ll << (sh - 1)) - lo;
      vt->off[k] = (int32_t)(uint32_t)(base - 0x3F800000ll);
    }
    vt->ok = true;
    vt->slack = (uint32_t)slack;
    vt->scale = (float)(1.0 / (2.0 * range));
    vt->zero_code = 0u;
    for (int i = 0; i < n; ++i) vt->zero_code += boundaries[i] < 0.0f ? 1u : 0u;
  }
}

extern "C" float tq_debug_value_slack() { return VALUE_SLACK; }

int tq_launch_encode_values_tiles(const EncodeArgs& a, const ValueTable& vt, bool after_keys,
                                  int sm_count, int device, cudaStream_t st) {
  const bool three = a.g.value_bits == 3;
  switch (a.g.kv_dtype) {
    case TQ_F32:
      return three ? launch_tiles<TQ_F32, 3>(a, vt, after_keys, sm_count, device, st)
                   : launch_tiles<TQ_F32, 4>(a, vt, after_keys, sm_count, device, st);
    case TQ_F16:
      return three ? launch_tiles<TQ_F16, 3>(a, vt, after_keys, sm_count, device, st)
                   : launch_tiles<TQ_F16, 4>(a, vt, after_keys, sm_count, device, st);
    default:
      return three ? launch_tiles<TQ_BF16, 3>(a, vt, after_keys, sm_count, device, st)
                   : launch_tiles<TQ_BF16, 4>(a, vt, after_keys, sm_count, device, st);
  }
}
