// Archives of stored .npy members (what np.savez writes, and the container format of a cold block): host
// code, one pass over the data.  The records are those of PKWARE's APPNOTE 4.3: a local header with 64-bit
// sizes in an extra field before each member, a central directory, an end record; stored, dated
// 1980-01-01, no comments.
//
// The checksum (CRC-32, polynomial 0xEDB88320 reflected) folds four 128-bit words at a time with carry-less
// multiplications (V. Gopal et al., "Fast CRC computation for generic polynomials using the PCLMULQDQ
// instruction", 2009); what is left, 16 bytes and a tail, goes through a table.  A block of 0.5 MB: 70 us
// to write and 57 us to read, Python's share included; with the records packed in Python and zlib's
// checksum 143 and 171 us.  What is left is the copy into fresh pages.
#include <cstring>

#include "common.cuh"

#if defined(__x86_64__)
#include <immintrin.h>
#endif

namespace {

struct CrcTables {
  uint32_t t[8][256];     // t[k][b]: byte b followed by k zero bytes
  uint64_t k512[2], k128[2];  // factors that move the low and high half of a word 512 and 128 bits on
  bool clmul;
  CrcTables() {
    for (uint32_t b = 0; b < 256; ++b) {
      uint32_t v = b;
      for (int i = 0; i < 8; ++i) v = step(v);
      t[0][b] = v;
    }
    for (uint32_t b = 0; b < 256; ++b)
      for (int k = 1; k < 8; ++k) t[k][b] = t[0][t[k - 1][b] & 255] ^ (t[k - 1][b] >> 8);
    // A word of 128 bits in memory order is a polynomial whose first bit has the highest degree; the product
    // of two reflected 64-bit halves comes out one degree too high.
    k512[0] = power(512 + 63), k512[1] = power(511);
    k128[0] = power(128 + 63), k128[1] = power(127);
#if defined(__x86_64__)
    clmul = __builtin_cpu_supports("pclmul") && __builtin_cpu_supports("sse4.1");
#else
    clmul = false;
#endif
  }
  static uint32_t step(uint32_t v) { return (v >> 1) ^ (v & 1 ? 0xEDB88320u : 0u); }
  static uint64_t power(int n) {  // x^n modulo the polynomial, as a reflected 64-bit half
    uint32_t v = 0x80000000u;
    for (int i = 0; i < n; ++i) v = step(v);
    return (uint64_t)v << 32;
  }
};
const CrcTables& crc_tables() {
  static const CrcTables tables;
  return tables;
}

// (the state without the inversions at both ends)
uint32_t crc_table(const CrcTables& c, uint32_t s, const uint8_t* p, size_t n) {
  for (; n >= 8; p += 8, n -= 8) {
    uint64_t w;
    memcpy(&w, p, 8);
    w ^= s;
    s = c.t[7][w & 255] ^ c.t[6][w >> 8 & 255] ^ c.t[5][w >> 16 & 255] ^ c.t[4][w >> 24 & 255] ^
        c.t[3][w >> 32 & 255] ^ c.t[2][w >> 40 & 255] ^ c.t[1][w >> 48 & 255] ^ c.t[0][w >> 56];
  }
  for (; n > 0; ++p, --n) s = c.t[0][(s ^ *p) & 255] ^ (s >> 8);
  return s;
}

#if defined(__x86_64__)
__attribute__((target("pclmul,sse4.1"))) inline __m128i crc_fold(__m128i x, __m128i k, __m128i next) {
  return _mm_xor_si128(_mm_xor_si128(_mm_clmulepi64_si128(x, k, 0x00), _mm_clmulepi64_si128(x, k, 0x11)), next);
}
// whole words of n >= 64 bytes; to != null: copied on the way
__attribute__((target("pclmul,sse4.1"))) uint32_t crc_words(const CrcTables& c, uint32_t s, const uint8_t* p,
                                                            size_t n, uint8_t* to) {
  auto load = [&](size_t at) __attribute__((target("pclmul,sse4.1"))) {
    const __m128i v = _mm_loadu_si128((const __m128i*)(p + at));
    if (to != nullptr) _mm_storeu_si128((__m128i*)(to + at), v);
    return v;
  };
  const __m128i k4 = _mm_set_epi64x((long long)c.k512[1], (long long)c.k512[0]);
  const __m128i k1 = _mm_set_epi64x((long long)c.k128[1], (long long)c.k128[0]);
  __m128i x0 = _mm_xor_si128(load(0), _mm_cvtsi32_si128((int)s));
  __m128i x1 = load(16), x2 = load(32), x3 = load(48);
  size_t at = 64;
  for (; at + 64 <= n; at += 64) {
    x0 = crc_fold(x0, k4, load(at));
    x1 = crc_fold(x1, k4, load(at + 16));
    x2 = crc_fold(x2, k4, load(at + 32));
    x3 = crc_fold(x3, k4, load(at + 48));
  }
  x0 = crc_fold(crc_fold(crc_fold(x0, k1, x1), k1, x2), k1, x3);
  for (; at + 16 <= n; at += 16) x0 = crc_fold(x0, k1, load(at));
  alignas(16) uint8_t last[16];
  _mm_store_si128((__m128i*)last, x0);
  return crc_table(c, 0, last, 16);
}
#endif

// checksum state after n more bytes, which are copied to `to` where it is not null
uint32_t crc_update(uint32_t s, const void* data, size_t n, uint8_t* to) {
  const CrcTables& c = crc_tables();
  const uint8_t* p = (const uint8_t*)data;
#if defined(__x86_64__)
  if (c.clmul && n >= 64) {
    const size_t whole = n & ~(size_t)15;
    s = crc_words(c, s, p, whole, to);
    p += whole, n -= whole;
    if (to != nullptr) to += whole;
  }
#endif
  if (n > 0 && to != nullptr) memcpy(to, p, n);
  return crc_table(c, s, p, n);
}

void put(uint8_t*& p, uint64_t v, int bytes) {  // little-endian
  for (int i = 0; i < bytes; ++i) *p++ = (uint8_t)(v >> (8 * i));
}
uint64_t get(const uint8_t* p, int bytes) {
  uint64_t v = 0;
  for (int i = 0; i < bytes; ++i) v |= (uint64_t)p[i] << (8 * i);
  return v;
}
constexpr int64_t LOCAL = 30, EXTRA = 20, CENTRAL = 46, END = 22;

}  // namespace

extern "C" int64_t tq_npz_write(int32_t n, const int64_t* parts, const char* text, void* out, int64_t out_bytes) {
  int64_t total = END;
  for (int i = 0; i < n; ++i) {
    if (parts[4 * i] < 0 || parts[4 * i] > 0xffff || parts[4 * i + 1] < 0 || parts[4 * i + 3] < 0) return -1;
    total += LOCAL + EXTRA + CENTRAL + 2 * parts[4 * i] + parts[4 * i + 1] + parts[4 * i + 3];
  }
  if (n < 0 || n >= 0xffff || total != out_bytes || total > INT32_MAX) return -1;
  uint8_t* p = (uint8_t*)out;
  int64_t central = out_bytes - END;
  for (int i = 0; i < n; ++i) central -= CENTRAL + parts[4 * i];
  uint8_t* c = p + central;
  for (int i = 0; i < n; ++i) {
    const int64_t n_name = parts[4 * i], n_head = parts[4 * i + 1], n_data = parts[4 * i + 3];
    const int64_t size = n_head + n_data, at = p - (uint8_t*)out;
    uint8_t* local = p;
    uint8_t* body = p + LOCAL + n_name + EXTRA;
    uint32_t crc = crc_update(0xffffffffu, text + n_name, (size_t)n_head, body);
    crc = ~crc_update(crc, (const void*)(intptr_t)parts[4 * i + 2], (size_t)n_data, body + n_head);
    // version 4.5 (64-bit sizes in the extra field), stored
    put(local, 0x04034b50u, 4), put(local, 45, 2), put(local, 0, 2), put(local, 0, 2), put(local, 0, 2);
    put(local, 33, 2), put(local, crc, 4), put(local, 0xffffffffu, 4), put(local, 0xffffffffu, 4);
    put(local, (uint64_t)n_name, 2), put(local, EXTRA, 2);
    memcpy(local, text, (size_t)n_name);
    local += n_name;
    put(local, 1, 2), put(local, 16, 2), put(local, (uint64_t)size, 8), put(local, (uint64_t)size, 8);
    // (written on a Unix system, readable and writable by the owner)
    put(c, 0x02014b50u, 4), put(c, 3 << 8 | 45, 2), put(c, 45, 2), put(c, 0, 2), put(c, 0, 2), put(c, 0, 2);
    put(c, 33, 2), put(c, crc, 4), put(c, (uint64_t)size, 4), put(c, (uint64_t)size, 4);
    put(c, (uint64_t)n_name, 2), put(c, 0, 2), put(c, 0, 2), put(c, 0, 2), put(c, 0, 2);
    put(c, 0600u << 16, 4), put(c, (uint64_t)at, 4);
    memcpy(c, text, (size_t)n_name);
    c += n_name;
    p = body + size;
    text += n_name + n_head;
  }
  const int64_t n_central = c - p;
  put(c, 0x06054b50u, 4), put(c, 0, 2), put(c, 0, 2), put(c, (uint64_t)n, 2), put(c, (uint64_t)n, 2);
  put(c, (uint64_t)n_central, 4), put(c, (uint64_t)central, 4), put(c, 0, 2);
  return c - (uint8_t*)out;
}

extern "C" int32_t tq_npz_read(const void* blob, int64_t bytes, int32_t max_members, int64_t* members) {
  const uint8_t* b = (const uint8_t*)blob;
  if (bytes < END) return -1;
  const int64_t end = bytes - END;
  const uint8_t* e = b + end;
  const int64_t total = (int64_t)get(e + 10, 2), first = (int64_t)get(e + 16, 4);
  if (get(e, 4) != 0x06054b50u || get(e + 4, 4) != 0 || (int64_t)get(e + 8, 2) != total || get(e + 20, 2) != 0 ||
      first + (int64_t)get(e + 12, 4) != end || total > max_members)
    return -1;
  int64_t at = first;
  for (int i = 0; i < total; ++i) {
    if (at + CENTRAL > end) return -1;
    const uint8_t* c = b + at;
    const uint32_t crc = (uint32_t)get(c + 16, 4);
    const int64_t size = (int64_t)get(c + 24, 4), n_name = (int64_t)get(c + 28, 2), local = (int64_t)get(c + 42, 4);
    // (flags and method, extra field and comment: none)
    if (get(c, 4) != 0x02014b50u || get(c + 8, 4) != 0 || (int64_t)get(c + 20, 4) != size || size == 0xffffffff ||
        get(c + 30, 4) != 0 || at + CENTRAL + n_name > end || local + LOCAL > first)
      return -1;
    const uint8_t* l = b + local;
    const int64_t start = local + LOCAL + n_name + (int64_t)get(l + 28, 2);
    if (get(l, 4) != 0x04034b50u || get(l + 6, 4) != 0 || (uint32_t)get(l + 14, 4) != crc ||
        (int64_t)get(l + 26, 2) != n_name || start + size > first || size < 10 ||
        memcmp(l + LOCAL, c + CENTRAL, (size_t)n_name) != 0)
      return -1;
    const int64_t n_head = 10 + (int64_t)get(b + start + 8, 2);
    if (memcmp(b + start, "\x93NUMPY\x01\x00", 8) != 0 || n_head > size ||
        ~crc_update(0xffffffffu, b + start, (size_t)size, nullptr) != crc)
      return -1;
    int64_t* m = members + 6 * i;
    m[0] = at + CENTRAL, m[1] = n_name;
    m[2] = start, m[3] = n_head;
    m[4] = start + n_head, m[5] = size - n_head;
    at += CENTRAL + n_name;
  }
  return at == end ? (int32_t)total : -1;
}
