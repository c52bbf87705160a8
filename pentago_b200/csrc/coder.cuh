// What the rANS coders (rans.cu, store.cu) share.
#pragma once
#include <cstdint>

namespace pg {

// Selects by a comparison, kept as selects: a predicated instruction waits
// about 13 cycles for a predicate that a select takes in 4 (measured), and the
// coders' chains are made of little else.
// x >= a ? u : v, and the same for a second pair of values
__device__ __forceinline__ void select_ge(uint32_t x, uint32_t a, uint32_t u0, uint32_t v0, uint32_t& r0, uint32_t u1,
                                          uint32_t v1, uint32_t& r1) {
  asm("{\n.reg .pred p;\nsetp.ge.u32 p, %2, %3;\nselp.u32 %0, %4, %5, p;\nselp.u32 %1, %6, %7, p;\n}\n"
      : "=&r"(r0), "=&r"(r1) : "r"(x), "r"(a), "r"(u0), "r"(v0), "r"(u1), "r"(v1));
}
__device__ __forceinline__ uint32_t select_ge(uint32_t x, uint32_t a, uint32_t u, uint32_t v) {
  uint32_t r;
  asm("{\n.reg .pred p;\nsetp.ge.u32 p, %1, %2;\nselp.u32 %0, %3, %4, p;\n}\n"
      : "=r"(r) : "r"(x), "r"(a), "r"(u), "r"(v));
  return r;
}

// A team of TEAM threads (this one is `rank`, `sync` their barrier) moves len
// bytes from src down to dst (dst <= src), WORDS words each at a time: whole
// words when src + len is on a word boundary, as it is in a word-aligned stream.
// A round's words are read before any of them is written, and a later round
// reads above what this one wrote.
template<int TEAM, int WORDS, class Sync>
__device__ __forceinline__ void move_down(uint8_t* dst, const uint8_t* src, uint32_t len, int rank, Sync sync) {
  if (dst == src) return;
  if (reinterpret_cast<uintptr_t>(src + len) & 3) {
    for (uint32_t i0 = 0; i0 < len; i0 += TEAM) {
      const uint8_t v = i0 + rank < len ? src[i0 + rank] : 0;
      sync();
      if (i0 + rank < len) dst[i0 + rank] = v;
      sync();
    }
    return;
  }
  const uint32_t head = min(len, uint32_t(-reinterpret_cast<uintptr_t>(dst)) & 3u);
  const uint32_t words = (len - head) >> 2, tail = len - head - 4 * words;
  const uint8_t hv = rank < head ? src[rank] : 0;
  sync();
  if (rank < head) dst[rank] = hv;
  sync();
  dst += head;
  src += head;
  const uint32_t sh = 8 * uint32_t(reinterpret_cast<uintptr_t>(src) & 3);
  const uint32_t* from = reinterpret_cast<const uint32_t*>(reinterpret_cast<uintptr_t>(src) & ~uintptr_t(3));
  uint32_t* to = reinterpret_cast<uint32_t*>(dst);
  for (uint32_t w0 = 0; w0 < words; w0 += TEAM * WORDS) {
    uint32_t v[WORDS];
#pragma unroll
    for (int q = 0; q < WORDS; q++) {
      const uint32_t w = w0 + TEAM * q + rank;
      v[q] = 0;
      if (w < words) v[q] = sh ? __funnelshift_r(from[w], from[w + 1], sh) : from[w];
    }
    sync();
#pragma unroll
    for (int q = 0; q < WORDS; q++) {
      const uint32_t w = w0 + TEAM * q + rank;
      if (w < words) to[w] = v[q];
    }
    sync();
  }
  const uint8_t tv = rank < tail ? src[4 * words + rank] : 0;
  sync();
  if (rank < tail) dst[4 * words + rank] = tv;
  sync();
}

}  // namespace pg
