// Fingerprint of a host buffer taken for a constant, used to notice that the constant changed.
//
// It covers the length, the first and last 512 bytes and up to 256 64-byte lines spread evenly over
// the rest, so that a change in the interior is seen too; about 17 KB are read whatever the size of
// the constant.  This runs for every constant of every inference (108 of them in ResNet-50), so its
// time is host time of every inference.  What bounds it is the fetch of 27 000 scattered cache
// lines, each on a page of its own in the large filters: sampled lines start on a cache-line
// boundary (one line each, not two) and are prefetched sixteen ahead, which overlaps the page walks,
// and the arithmetic takes 32 bytes per instruction.  ResNet-50's constants, caches warm: 78 us;
// 227 us with a multiply per eight bytes, no prefetch and lines at 8-byte boundaries.
//
// Per 64-byte line: acc += lo32(w ^ key) * hi32(w ^ key) in every 64-bit lane, plus the neighbouring
// half's words unmixed, so that no single changed word goes unseen; the key steps from line to line,
// so that exchanged lines count as a change.
//
// Published methods it builds on: the step per line is the long-input accumulation of XXH3 (Y. Collet, xxHash), the
// final mix is one round of splitmix64's (S. Vigna); the constants are odd 64-bit numbers known from these and from
// wyhash (W. Yi).  The choice of lines and their completion are this file's.
#include <cstddef>
#include <cstdint>
#include <cstring>
#if defined(__x86_64__)
#include <immintrin.h>
#endif

namespace occ {

namespace {

constexpr uint64_t KEY0[4] = {0x9e3779b97f4a7c15ull, 0xc2b2ae3d27d4eb4full, 0x165667b19e3779f9ull,
                              0x27d4eb2f165667c5ull};
constexpr uint64_t KEY_STEP[4] = {0x9fb21c651e98df25ull, 0xd6e8feb86659fd93ull, 0xa0761d6478bd642full,
                                  0xe7037ed1a0b428dbull};
constexpr int AHEAD = 16;   // sampled lines requested ahead of the one being hashed

// The covered 64-byte lines in hashing order; partial ones are completed with zeros in `pad`.
struct Lines {
  const unsigned char *at[2 * 8 + 256];
  int n = 0;
  unsigned char pad[2][64];

  Lines(const unsigned char *b, size_t bytes) {
    const size_t head = bytes < 512 ? bytes : 512;
    range(b, 0, head, pad[0]);
    if (bytes > 512) range(b, bytes - 512 > head ? bytes - 512 : head, bytes, pad[1]);
    if (bytes > 1024) {   // whole lines over the rest: all of them, or 256 from the first to the last
      const unsigned char *first = b + 512 - ((uintptr_t)(b + 512) & 63);
      const size_t count = ((size_t)(b + bytes - 513 - first) >> 6) + 1;
      const size_t take = count < 256 ? count : 256;
      const uint64_t step = take > 1 ? ((uint64_t)(count - 1) << 16) / (take - 1) : 0;
      for (size_t k = 0; k < take; ++k) at[n++] = first + 64 * (size_t)((step * k + 0xffff) >> 16);
    }
    for (int i = 0; i < AHEAD && i < n; ++i) __builtin_prefetch(at[i]);
  }
  void range(const unsigned char *b, size_t lo, size_t hi, unsigned char *rest) {
    for (; lo + 64 <= hi; lo += 64) at[n++] = b + lo;
    if (lo < hi) {
      memset(rest, 0, 64);
      memcpy(rest, b + lo, hi - lo);
      at[n++] = rest;
    }
  }
};

uint64_t finish(const uint64_t *acc, size_t bytes) {
  uint64_t h = KEY0[0] ^ bytes;
  for (int j = 0; j < 8; ++j) {
    h = (h ^ acc[j] ^ (acc[j] >> 29)) * 0xbf58476d1ce4e5b9ull;
    h ^= h >> 32;
  }
  return h;
}

#if defined(__x86_64__)
__attribute__((target("avx2"))) uint64_t fingerprint_avx2(const unsigned char *b, size_t bytes) {
  __m256i a0 = _mm256_setzero_si256(), a1 = _mm256_setzero_si256();
  __m256i key = _mm256_loadu_si256((const __m256i *)KEY0);
  const __m256i step = _mm256_loadu_si256((const __m256i *)KEY_STEP);
  const Lines lines(b, bytes);
  for (int i = 0; i < lines.n; ++i) {
    const unsigned char *p = lines.at[i];
    if (i + AHEAD < lines.n) __builtin_prefetch(lines.at[i + AHEAD]);
    const __m256i w0 = _mm256_loadu_si256((const __m256i *)p);
    const __m256i w1 = _mm256_loadu_si256((const __m256i *)(p + 32));
    const __m256i next = _mm256_add_epi64(key, step);
    const __m256i x0 = _mm256_xor_si256(w0, key), x1 = _mm256_xor_si256(w1, next);
    a0 = _mm256_add_epi64(a0, _mm256_add_epi64(_mm256_mul_epu32(x0, _mm256_srli_epi64(x0, 32)), w1));
    a1 = _mm256_add_epi64(a1, _mm256_add_epi64(_mm256_mul_epu32(x1, _mm256_srli_epi64(x1, 32)), w0));
    key = next;
  }
  uint64_t acc[8];
  _mm256_storeu_si256((__m256i *)acc, a0);
  _mm256_storeu_si256((__m256i *)(acc + 4), a1);
  return finish(acc, bytes);
}
#endif

uint64_t fingerprint_plain(const unsigned char *b, size_t bytes) {
  uint64_t acc[8] = {0, 0, 0, 0, 0, 0, 0, 0}, key[4];
  memcpy(key, KEY0, sizeof(key));
  const Lines lines(b, bytes);
  for (int i = 0; i < lines.n; ++i) {
    uint64_t w[8];
    memcpy(w, lines.at[i], 64);
    for (int j = 0; j < 4; ++j) {
      const uint64_t next = key[j] + KEY_STEP[j];
      const uint64_t x0 = w[j] ^ key[j], x1 = w[4 + j] ^ next;
      acc[j] += (x0 & 0xffffffffu) * (x0 >> 32) + w[4 + j];
      acc[4 + j] += (x1 & 0xffffffffu) * (x1 >> 32) + w[j];
      key[j] = next;
    }
  }
  return finish(acc, bytes);
}

}  // namespace

uint64_t host_hash(const void *src, size_t bytes) {
  const unsigned char *b = (const unsigned char *)src;
#if defined(__x86_64__)
  static const bool avx2 = __builtin_cpu_supports("avx2");
  if (avx2) return fingerprint_avx2(b, bytes);
#endif
  return fingerprint_plain(b, bytes);
}

// The same value without vector instructions (what a processor without AVX2 computes).
uint64_t host_hash_plain(const void *src, size_t bytes) {
  return fingerprint_plain((const unsigned char *)src, bytes);
}

}  // namespace occ
