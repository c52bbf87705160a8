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

// The warp moves len bytes from src down to dst (dst <= src): whole words
// when src + len is on a word boundary, as it is in a word-aligned stream.
// A round's words are read before any of them is written.
constexpr int kMoveWords = 8;
__device__ __forceinline__ void move_down(uint8_t* dst, const uint8_t* src, uint32_t len, int lane) {
  if (dst == src) return;
  if (reinterpret_cast<uintptr_t>(src + len) & 3) {
    for (uint32_t i0 = 0; i0 < len; i0 += 32) {
      const uint8_t v = i0 + lane < len ? src[i0 + lane] : 0;
      __syncwarp();
      if (i0 + lane < len) dst[i0 + lane] = v;
      __syncwarp();
    }
    return;
  }
  const uint32_t head = min(len, uint32_t(-reinterpret_cast<uintptr_t>(dst)) & 3u);
  const uint32_t words = (len - head) >> 2, tail = len - head - 4 * words;
  const uint8_t hv = lane < head ? src[lane] : 0;
  __syncwarp();
  if (lane < head) dst[lane] = hv;
  __syncwarp();
  dst += head;
  src += head;
  const uint32_t sh = 8 * uint32_t(reinterpret_cast<uintptr_t>(src) & 3);
  const uint32_t* from = reinterpret_cast<const uint32_t*>(reinterpret_cast<uintptr_t>(src) & ~uintptr_t(3));
  uint32_t* to = reinterpret_cast<uint32_t*>(dst);
  for (uint32_t w0 = 0; w0 < words; w0 += 32 * kMoveWords) {
    uint32_t v[kMoveWords];
#pragma unroll
    for (int q = 0; q < kMoveWords; q++) {
      const uint32_t w = w0 + 32 * q + lane;
      v[q] = 0;
      if (w < words) v[q] = sh ? __funnelshift_r(from[w], from[w + 1], sh) : from[w];
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < kMoveWords; q++) {
      const uint32_t w = w0 + 32 * q + lane;
      if (w < words) to[w] = v[q];
    }
    __syncwarp();
  }
  const uint8_t tv = lane < tail ? src[4 * words + lane] : 0;
  __syncwarp();
  if (lane < tail) dst[4 * words + lane] = tv;
  __syncwarp();
}

}  // namespace pg
