// Static-table rANS over ternary win/tie/loss symbols, byte-identical to the
// reference's format version 2 (pentago/shard/arithmetic.cc:20-23, 48-77,
// 366-495): 8 interleaved 32-bit rANS lanes (symbol i on lane i % 8), 14-bit
// frequency total, byte renormalization at 2^23, each lane's bytes stored in
// decode order, header = version(4) | counts(3 x 8) | stream lengths(8 x 4).
//
// A stream has only 8 sequential chains, so the GPU codes many streams at
// once: 8 threads per stream, four streams per warp.
#include "coder.cuh"
#include "runtime.h"
#include "../../include/pentago_b200.h"
#include <cstdint>

namespace pg {

constexpr uint32_t kRansTotalBits = 14;
constexpr uint32_t kRansTotal = 1u << kRansTotalBits;
constexpr uint32_t kRansLower = 1u << 23;
constexpr int kLanes = 8;
constexpr int kHeader = 4 + 24 + 32;

struct rans_freq {
  uint32_t freq[3], cum[3], xmax[3];
};

// make_freq (arithmetic.cc:48-77), in the same integer arithmetic.
__host__ __device__ inline rans_freq make_freq(const uint64_t* counts) {
  rans_freq t;
  const uint64_t sum = counts[0] + counts[1] + counts[2];
  uint32_t f[3];
  if (sum) {
    for (int i = 0; i < 3; i++) f[i] = uint32_t(counts[i] * kRansTotal / sum);
    for (int i = 0; i < 3; i++) if (!f[i]) f[i] = 1;
    const int32_t adjust = int32_t(kRansTotal) - int32_t(f[0] + f[1] + f[2]);
    int largest = 0;
    if (f[1] > f[largest]) largest = 1;
    if (f[2] > f[largest]) largest = 2;
    f[largest] = uint32_t(int32_t(f[largest]) + adjust);
  } else {
    f[0] = f[1] = f[2] = kRansTotal / 3;
    f[0] += kRansTotal - 3 * (kRansTotal / 3);
  }
  const uint32_t xm = (kRansLower >> kRansTotalBits) << 8;
  for (int i = 0; i < 3; i++) { t.freq[i] = f[i]; t.xmax[i] = xm * f[i]; }
  t.cum[0] = 0;
  t.cum[1] = f[0];
  t.cum[2] = f[0] + f[1];
  return t;
}

// Worst-case lane slot (the reference's per-lane buffer, arithmetic.cc:377).
__host__ __device__ inline int64_t lane_capacity(int64_t n) { return n / kLanes * 2 + 64; }
__host__ __device__ inline int64_t stream_bound(int64_t n) { return kHeader + kLanes * lane_capacity(n); }

__device__ inline void put_u32(uint8_t* p, uint32_t v) { for (int i = 0; i < 4; i++) p[i] = uint8_t(v >> (8 * i)); }
__device__ inline void put_u64(uint8_t* p, uint64_t v) { for (int i = 0; i < 8; i++) p[i] = uint8_t(v >> (8 * i)); }
__device__ inline uint32_t get_u32(const uint8_t* p) {
  return uint32_t(p[0]) | uint32_t(p[1]) << 8 | uint32_t(p[2]) << 16 | uint32_t(p[3]) << 24;
}
__device__ inline uint64_t get_u64(const uint8_t* p) { return uint64_t(get_u32(p)) | uint64_t(get_u32(p + 4)) << 32; }

// Encoder constants of one symbol: state / freq by a reciprocal multiply
// (x < 2^31 after renormalization, where the reciprocal is exact), as in
// F. Giesen's ryg_rans (RansEncSymbolInit / RansEncPutSymbol, after
// Alverson, "Integer division using reciprocals", 1991).  The new state is
// x + bias + q * (total - freq) = (x / freq) * total + x % freq + cum.
struct rans_enc_sym {
  uint32_t xmax, rcp, shift, bias, cmpl;
};

__host__ __device__ inline rans_enc_sym enc_sym(const rans_freq& t, int s) {
  rans_enc_sym e;
  const uint32_t f = t.freq[s];
  e.xmax = t.xmax[s];
  e.cmpl = kRansTotal - f;
  if (f < 2) {
    e.rcp = ~0u;
    e.shift = 0;
    e.bias = t.cum[s] + kRansTotal - 1;
  } else {
    uint32_t sh = 0;
    while (f > (1u << sh)) sh++;
    e.rcp = uint32_t(((uint64_t(1) << (sh + 31)) + f - 1) / f);
    e.shift = sh - 1;
    e.bias = t.cum[s];
  }
  return e;
}

// ---------------------------------------------------------------------------
// Encoding, in three launches:
//
//   rans_count_kernel   symbol counts of long streams (the frequency tables);
//   rans_encode_kernel  the coding itself, 8 lanes per stream, a warp for four
//                       streams, with the counting and packing of short ones;
//   rans_pack_kernel    the lanes' bytes of long streams moved from their slots
//                       to behind the header.
//
// The coding is bound by the latency of its 8 chains per stream: a lane's
// next symbol waits for its last (a compare and select, a multiply-high, a
// shift and a multiply-add), and 1,024 streams are only 256 warps.  So a
// warp (four streams) is a CTA of its own, which spreads the warps over all
// SMs, and little but the chain is on the chain: symbols are staged in shared
// memory a chunk ahead, a symbol's constants are one 16-byte shared load, and
// the bytes of a renormalization are always written to the lane's buffer,
// whose position then moves past them or does not; whole words leave it at a
// chunk's end.  Counting and packing of a long stream have a CTA, as its 8
// lanes would take as long for them as for the coding; for short ones such
// CTAs would cost more (14 ns a stream) than the lanes take, and bytes that fit
// the lanes' buffers never see their slots.  1,024 streams of 1 M symbols:
// 3.65 ms (coding 3.36, about 53 cycles a symbol of a lane where the chain itself
// needs 27, counting 0.17, packing 0.11); 65,536 of 512 symbols: 0.12 ms.

constexpr int kChunk = 1024;             // symbols of a stream staged at a time: 128 for each lane
constexpr int kChunkRow = kChunk + 32;   // the four streams' rows start 8 banks apart
constexpr int kWarpStreams = 32 / kLanes;
// A renormalization moves at most one byte for a symbol of this frequency:
// the encoder's state, below 2^31, is below xmax = 64 * 2^17 after one, and
// the decoder's is at least 64 * 2^9 = 2^15 before it.  One-byte forms of the inner
// loops take fewer instructions per symbol and refill or flush half as often.
constexpr uint32_t kOneByteFreq = 64;

// Ones and twos of a stream, and whether it holds a symbol above 2.
struct rans_counts {
  uint64_t one, two;
  uint32_t bad;
};

// Four symbols: ones in the low half of n, twos in the high half.
__device__ __forceinline__ void count_word(uint32_t w, uint32_t& n, uint32_t& bad) {
  n += __popc(w & 0x01010101u) + (__popc(w & 0x02020202u) << 16);
  bad |= (w & 0xfcfcfcfcu) | (w & (w >> 1) & 0x01010101u);
}

// The symbols sym[0 .. n) that thread `rank` of TEAM counts: 16-byte loads where the
// words lie inside the stream, bytes at its ends.  Eight loads are in flight
// per thread.
template<int TEAM>
__device__ __forceinline__ rans_counts count_symbols(const uint8_t* sym, int64_t n, int rank) {
  const int64_t head = min(n, int64_t(-reinterpret_cast<uintptr_t>(sym) & 15)), words = (n - head) >> 4;
  const int64_t tail = head + 16 * words;
  const uint4* W = reinterpret_cast<const uint4*>(sym + head);
  uint32_t one = 0, two = 0, bad = 0;   // (a thread has less than 2^32 of them)
  constexpr int kUnroll = 8;
  for (int64_t k0 = 0; k0 < words; k0 += kUnroll * TEAM) {
    uint4 v[kUnroll];
#pragma unroll
    for (int q = 0; q < kUnroll; q++) {
      const int64_t k = k0 + q * TEAM + rank;
      v[q] = k < words ? __ldg(W + k) : make_uint4(0, 0, 0, 0);
    }
    uint32_t m = 0;
#pragma unroll
    for (int q = 0; q < kUnroll; q++) {
      count_word(v[q].x, m, bad);
      count_word(v[q].y, m, bad);
      count_word(v[q].z, m, bad);
      count_word(v[q].w, m, bad);
    }
    one += m & 0xffff;
    two += m >> 16;
  }
  uint32_t m = 0;
  for (int i = rank; i < int(head); i += TEAM) count_word(sym[i], m, bad);
  for (int i = rank; i < int(n - tail); i += TEAM) count_word(sym[tail + i], m, bad);
  one += m & 0xffff;
  two += m >> 16;
  return rans_counts{one, two, bad};
}

// Streams longer than this, in a batch of nstreams, are left to the kernels of
// the long ones for their counts and packing.  A few streams have the chip to
// themselves (64 of 4,096 symbols 42 us with those kernels, 46 without); of many,
// those that their 8 lanes see to cost less (65,536 of 4,096: 1.24 and 0.42 ms).
constexpr int64_t kOwnOfFew = 2048, kOwnOfMany = 16384;
// A CTA of those handles streams blockIdx.x + k gridDim.x: the next 256 of them
// are looked at together, and f(s, n) called for the long ones, by all threads.
constexpr int kLongThreads = 256, kLongCtas = 8 * 148;   // (resident at once)
template<class F>
__device__ __forceinline__ void each_long(const int64_t* __restrict__ offsets, int nstreams, int64_t own,
                                          const int64_t* __restrict__ expect, F f) {
  __shared__ unsigned mask[kLongThreads / 32];
  for (int64_t k0 = 0; blockIdx.x + k0 * gridDim.x < nstreams; k0 += kLongThreads) {
    const int64_t s = blockIdx.x + (k0 + threadIdx.x) * gridDim.x;
    const int64_t n = s < nstreams ? offsets[s + 1] - offsets[s] : 0;
    const unsigned mine = __ballot_sync(0xffffffffu, n > own && !(expect && n != expect[s]));
    if ((threadIdx.x & 31) == 0) mask[threadIdx.x >> 5] = mine;
    __syncthreads();
    for (int w = 0; w < kLongThreads / 32; w++)
      for (unsigned left = mask[w]; left; left &= left - 1) {
        const int64_t t = blockIdx.x + (k0 + 32 * w + __ffs(left) - 1) * gridDim.x;
        f(t, offsets[t + 1] - offsets[t]);
      }
    __syncthreads();
  }
}

// The counts go into the header of the stream's output, with a version of 0 if
// the stream cannot be coded.
__global__ void __launch_bounds__(kLongThreads, 8)
rans_count_kernel(const uint8_t* __restrict__ symbols, const int64_t* __restrict__ offsets, int nstreams, int64_t own,
                  const int64_t* __restrict__ expect, uint8_t* __restrict__ out,
                  const int64_t* __restrict__ out_offsets) {
  __shared__ unsigned long long total[3];
  each_long(offsets, nstreams, own, expect, [&](int64_t s, int64_t n) {
    if (threadIdx.x < 3) total[threadIdx.x] = 0;
    __syncthreads();
    rans_counts C = count_symbols<kLongThreads>(symbols + offsets[s], n, threadIdx.x);
    for (int o = 16; o; o >>= 1) {
      C.one += __shfl_xor_sync(0xffffffffu, C.one, o);
      C.two += __shfl_xor_sync(0xffffffffu, C.two, o);
    }
    C.bad = __any_sync(0xffffffffu, C.bad != 0);
    if ((threadIdx.x & 31) == 0) {
      atomicAdd(&total[0], (unsigned long long)C.one);
      atomicAdd(&total[1], (unsigned long long)C.two);
      if (C.bad) atomicOr(&total[2], 1ull);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      uint8_t* base = out + out_offsets[s];
      put_u32(base, total[2] ? 0 : 2);
      put_u64(base + 4, uint64_t(n) - total[0] - total[1]);
      put_u64(base + 12, total[0]);
      put_u64(base + 20, total[1]);
    }
  });
}

// End of lane l's slot: its bytes are written downward from there in whole
// aligned words (a slot has 64 bytes more than its lane can need).
__device__ __forceinline__ uint8_t* slot_end(uint8_t* base, int64_t n, int l) {
  return reinterpret_cast<uint8_t*>(reinterpret_cast<uintptr_t>(base + kHeader + (l + 1) * lane_capacity(n)) &
                                    ~uintptr_t(3));
}

// One lane's coder: the state, and the bytes not yet stored, in the lane's
// buffer in shared memory at [pos, kTop).  A symbol's bytes are always
// written below pos, which moves down only when the state had to give them.
constexpr int kTop = 2 * kChunk / kLanes + 8;   // a chunk's bytes, three left from the last, two more written
constexpr int kLaneRow = kTop + 4;              // an odd number of words: the lanes' rows spread over the banks
static_assert(kTop % 4 == 0 && kLaneRow / 4 % 2 == 1, "words of a lane's buffer");
struct rans_enc_lane {
  uint32_t x;
  int pos;
  uint8_t* p;   // word aligned; what is stored so far is above it
  // P: the symbol's {xmax, rcp, bias, shift | cmpl << 5}.  A symbol takes at
  // most two bytes out of the state (x < 2^31, xmax >= 2^17), and at most one
  // when its frequency is kOneByteFreq or more (xmax >= 2^23).
  template<int BYTES> __device__ __forceinline__ void put(const uint4 P, uint8_t* buf) {
    const uint32_t x8 = x >> 8;
    uint32_t y, at;
    buf[pos - 1] = uint8_t(x);
    select_ge(x, P.x, x8, x, y, uint32_t(pos - 1), uint32_t(pos), at);
    if (BYTES == 2) {
      buf[pos - 2] = uint8_t(x8);
      select_ge(x8, P.x, x >> 16, y, y, uint32_t(pos - 2), at, at);
    }
    pos = int(at);
    const uint32_t q = __funnelshift_r(__umulhi(y, P.y), 0u, P.w);   // a shift by P.w mod 32
    // (y + bias is ready before q: the multiply-add ends the chain)
    asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(x) : "r"(q), "r"(P.w >> 5), "r"(y + P.z));
  }
  // A chunk that lies inside the stream: the lane's symbols row[8 j], last
  // first; constants are loaded four symbols ahead, and the symbols that name
  // them four before that.
  template<int BYTES> __device__ __forceinline__ void put_chunk(const uint8_t* row, const uint4* P, uint8_t* buf) {
    constexpr int kSteps = kChunk / kLanes;
    uint4 now[4], next[4];
    int sym[4];
#pragma unroll
    for (int i = 0; i < 4; i++) next[i] = P[row[8 * (kSteps - 1 - i)]];
#pragma unroll
    for (int i = 0; i < 4; i++) sym[i] = row[8 * (kSteps - 5 - i)];
#pragma unroll 4
    for (int j = kSteps - 1; j > 0; j -= 4) {
#pragma unroll
      for (int i = 0; i < 4; i++) {
        now[i] = next[i];
        next[i] = P[sym[i]];
      }
      // (the last two rounds load the chunk's first symbols again)
      const int ahead = max(j - 8, 3);
#pragma unroll
      for (int i = 0; i < 4; i++) sym[i] = row[8 * (ahead - i)];
#pragma unroll
      for (int i = 0; i < 4; i++) put<BYTES>(now[i], buf);
    }
  }
  // Whole words from the buffer to the slot; up to three bytes stay.
  __device__ __forceinline__ void flush(uint8_t* buf) {
    const int words = (kTop - pos) >> 2;
    const uint32_t* from = reinterpret_cast<const uint32_t*>(buf + kTop) - 1;
    for (int w = 0; w < words; w++) reinterpret_cast<uint32_t*>(p)[-1 - w] = from[-w];
    *reinterpret_cast<uint32_t*>(buf + kTop - 4) = from[-words];
    p -= 4 * words;
    pos += 4 * words;
  }
  // The bytes still held and the final state
  __device__ __forceinline__ void finish(const uint8_t* buf) {
    for (int k = kTop - 1; k >= pos; k--) *--p = buf[k];
    for (int j = 0; j < 4; j++) *--p = uint8_t(x >> (8 * j));
  }
};

// The 16 bytes at g that lie in [a, b), zero elsewhere: a whole load inside,
// single bytes at the ends.
__device__ __forceinline__ uint4 load_granule(uintptr_t g, uintptr_t a, uintptr_t b) {
  if (g >= a && g + 16 <= b) return __ldg(reinterpret_cast<const uint4*>(g));
  uint32_t w[4] = {0, 0, 0, 0};
  for (int k = 0; k < 16; k++)
    if (g + k >= a && g + k < b) w[k >> 2] |= uint32_t(__ldg(reinterpret_cast<const uint8_t*>(g + k))) << (8 * (k & 3));
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// One warp, four streams.  out_offsets[s] has room for stream_bound(n_s).
// (OWN is a constant because it costs 1.5% of the coding as a parameter)
template<int64_t OWN>
__global__ void __launch_bounds__(32)
rans_encode_kernel(const uint8_t* __restrict__ symbols, const int64_t* __restrict__ offsets, int nstreams,
                   uint8_t* out, const int64_t* __restrict__ out_offsets, int64_t* __restrict__ sizes,
                   const int64_t* __restrict__ expect) {
  __shared__ __align__(16) uint8_t stage[kWarpStreams][kChunkRow];
  __shared__ uint4 par[kWarpStreams][3];
  __shared__ __align__(16) uint8_t bytes[32][kLaneRow];
  const int g = threadIdx.x >> 3, lane = threadIdx.x & 7;
  const int64_t s = int64_t(blockIdx.x) * kWarpStreams + g;
  const unsigned group = 0xffu << (8 * g);
  int64_t n = -1;
  uintptr_t a = 0, b = 0;
  uint8_t* base = nullptr;
  uint64_t c[3] = {0, 0, 0};
  bool frequent = true;   // every symbol that occurs has kOneByteFreq or more
  if (s < nstreams) {
    n = offsets[s + 1] - offsets[s];
    a = reinterpret_cast<uintptr_t>(symbols) + uintptr_t(offsets[s]);
    b = a + uintptr_t(n);
    base = out + out_offsets[s];
    // With `expect`, a stream of another length has no room reserved: refuse it
    bool bad = n < 0 || (expect && n != expect[s]);
    if (!bad && n > OWN) {
      bad = get_u32(base) != 2;
      c[1] = get_u64(base + 12);
      c[2] = get_u64(base + 20);
    } else if (!bad) {
      rans_counts C = count_symbols<kLanes>(symbols + offsets[s], n, lane);
      for (int o = 4; o; o >>= 1) {
        C.one += __shfl_xor_sync(group, C.one, o, 8);
        C.two += __shfl_xor_sync(group, C.two, o, 8);
        C.bad |= __shfl_xor_sync(group, C.bad, o, 8);
      }
      bad = C.bad != 0;
      c[1] = C.one;
      c[2] = C.two;
    }
    if (bad) {
      if (lane == 0) sizes[s] = PG_ERR_ARG;
      n = -1;
    } else {
      c[0] = uint64_t(n) - c[1] - c[2];
      const rans_freq t = make_freq(c);
#pragma unroll
      for (int v = 0; v < 3; v++) frequent &= !c[v] || t.freq[v] >= kOneByteFreq;
      if (lane < 3) {
        const rans_enc_sym e = enc_sym(t, lane);
        par[g][lane] = make_uint4(e.xmax, e.rcp, e.bias, e.shift | e.cmpl << 5);
      }
    }
  }
  // Symbols by address: chunk k holds the bytes [first + k kChunk, + kChunk)
  // with first 16-byte aligned, and a lane's symbols in it are those at
  // mine + 8 j.  Chunks go from the stream's last to its first.
  const uintptr_t first = a & ~uintptr_t(15);
  const int64_t nchunks = n > 0 ? int64_t((b - first + kChunk - 1) / kChunk) : 0;
  const int mine = int((a + lane) & 7);
  uint8_t* const buf = bytes[threadIdx.x];
  rans_enc_lane E = {kRansLower, kTop, n >= 0 ? slot_end(base, n, lane) : nullptr};
  uint8_t* const end = E.p;
  const bool kept = n <= kChunk;   // a lane's bytes all fit its buffer
  constexpr int kGranules = kChunk / 16 / kLanes;
  uint4 next[kGranules];
  auto load_chunk = [&](int64_t k) {
    const uintptr_t lo = first + k * kChunk;
    if (lo >= a && lo + kChunk <= b) {
#pragma unroll
      for (int q = 0; q < kGranules; q++) next[q] = __ldg(reinterpret_cast<const uint4*>(lo) + lane + kLanes * q);
    } else {
#pragma unroll
      for (int q = 0; q < kGranules; q++) next[q] = load_granule(lo + 16 * (lane + kLanes * q), a, b);
    }
  };
  if (nchunks) load_chunk(nchunks - 1);
  // (the same form for the whole warp, so that its streams run together)
  const bool one_byte = __all_sync(0xffffffffu, frequent);
  const int64_t rounds = __reduce_max_sync(0xffffffffu, unsigned(min(nchunks, int64_t(0x7fffffff))));
  const uint8_t* row = stage[g];
  const uint4* P = par[g];
  for (int64_t r = 0; r < rounds; r++) {
    const int64_t k = nchunks - 1 - r;
    __syncwarp();
    if (k >= 0) {
#pragma unroll
      for (int q = 0; q < kGranules; q++) reinterpret_cast<uint4*>(stage[g])[lane + kLanes * q] = next[q];
    }
    __syncwarp();
    if (k > 0) load_chunk(k - 1);
    if (k >= 0) {
      const uintptr_t lo = first + k * kChunk;
      if (lo >= a && lo + kChunk <= b) {
        if (one_byte) E.put_chunk<1>(row + mine, P, buf);
        else E.put_chunk<2>(row + mine, P, buf);
      } else {
        const int top = b < lo + kChunk ? (int(b - lo) - 1 - mine) >> 3 : kChunk / kLanes - 1;
        for (int j = top; j >= 0; j--) {
          const uintptr_t at = lo + mine + 8 * j;
          if (at < a) break;
          E.put<2>(P[row[mine + 8 * j]], buf);
        }
      }
      if (!kept) E.flush(buf);
    }
  }
  if (n < 0) return;
  if (!kept) E.finish(buf);
  const uint32_t len = kept ? uint32_t(kTop - E.pos) + 4 : uint32_t(end - E.p);
  uint64_t upto = len;   // the lanes' up to and with this one
  for (int o = 1; o < kLanes; o <<= 1) {
    const uint64_t v = __shfl_up_sync(group, upto, o, 8);
    if (lane >= o) upto += v;
  }
  const uint64_t total = __shfl_sync(group, upto, kLanes - 1, 8);
  if (kept) {
    uint8_t* dst = base + kHeader + (upto - len);
    for (int j = 0; j < 4; j++) dst[j] = uint8_t(E.x >> (24 - 8 * j));
    for (int k = E.pos; k < kTop; k++) dst[4 + k - E.pos] = buf[k];
  } else if (n <= OWN) {
    __syncwarp(group);
    uint8_t* dst = base + kHeader;
    for (int l = 0; l < kLanes; l++) {   // (as in rans_pack_kernel)
      const uint32_t m = __shfl_sync(group, len, l, 8);
      move_down<kLanes, 8>(dst, slot_end(base, n, l) - m, m, lane, [group] { __syncwarp(group); });
      dst += m;
    }
  }
  put_u32(base + 28 + 4 * lane, len);
  if (lane == 0) {
    put_u32(base, 2);
    for (int k = 0; k < 3; k++) put_u64(base + 4 + 8 * k, c[k]);
    sizes[s] = kHeader + int64_t(total);
  }
}

// The lanes' bytes, in lane order, from their slots to behind the header.  A
// lane's bytes move down, and never past a slot that has not moved yet (they
// fit their own).
__global__ void __launch_bounds__(kLongThreads)
rans_pack_kernel(const int64_t* __restrict__ offsets, int nstreams, int64_t own, const int64_t* __restrict__ expect,
                 uint8_t* out, const int64_t* __restrict__ out_offsets, const int64_t* __restrict__ sizes) {
  each_long(offsets, nstreams, own, expect, [&](int64_t s, int64_t n) {
    if (sizes[s] < 0) return;
    uint8_t* base = out + out_offsets[s];
    uint8_t* dst = base + kHeader;
    for (int l = 0; l < kLanes; l++) {
      const uint32_t len = get_u32(base + 28 + 4 * l);
      move_down<kLongThreads, 4>(dst, slot_end(base, n, l) - len, len, threadIdx.x, [] { __syncthreads(); });
      dst += len;
    }
  });
}

// ---------------------------------------------------------------------------
// Decoding: one warp, four streams, like the encoder and bound like it by the
// lanes' chains (symbol, state, renormalization).  A lane's stream bytes are
// not on the chain: they come from a ring in shared memory with the next byte
// always in a register; the ring is filled by
// asynchronous copies three blocks ahead, which no register waits for (a
// warp's 32 lanes run low at different symbols, so a load into a register
// would stop the warp at nearly every symbol).  Symbols are staged
// and leave in 16-byte stores.  1,024 streams of 1 M symbols of a solved
// slice: 3.5 ms (about 51 cycles a symbol of a lane, 41 of them in block_one).

constexpr int kBlockSteps = 128;                     // symbols of a lane per block
constexpr int kBlockSyms = kBlockSteps * kLanes;     // and of a stream
constexpr int kRing = 512;                           // a lane's ring of stream bytes,
constexpr int kMirror = 16 * 9;                      // its first ones again after its last (a block's bytes and one more)
constexpr int kRingRow = kRing + kMirror + 16;
static_assert(kMirror > kBlockSteps + 1, "a one-byte block reads on into the mirror");
constexpr int kOutRow = kBlockSyms + 32;             // a stream's staged symbols (the rows 8 banks apart)

// Shifts by any amount (32 and more give 0), as the hardware does them.
__device__ __forceinline__ uint32_t shift_right(uint32_t x, uint32_t n) {
  uint32_t r;
  asm("shr.u32 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(n));
  return r;
}
__device__ __forceinline__ uint32_t shift_left(uint32_t x, uint32_t n) {
  uint32_t r;
  asm("shl.b32 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(n));
  return r;
}

// Frequencies and where symbols 1 and 2 start.
struct rans_dec_table {
  uint32_t f0, f1, f2, c1, c2;
};

// The state after the symbol that x's low bits name, before it is refilled,
// and the symbol: x = f h + slot - cum, as a sum of differences between
// neighbouring symbols so that the constants ride on the multiply-adds.
__device__ __forceinline__ uint32_t next_symbol(const rans_dec_table& F, uint32_t x, uint32_t& v) {
  const uint32_t slot = x & (kRansTotal - 1), h = x >> kRansTotalBits;
  uint32_t d1, d2;
  select_ge(slot, F.c1, (F.f1 - F.f0) * h - F.c1, 0u, d1, 1u, 0u, v);
  select_ge(slot, F.c2, (F.f2 - F.f1) * h - (F.c2 - F.c1), 0u, d2, 2u, v, v);
  return F.f0 * h + slot + d1 + d2;
}

// kBlockSteps symbols of a lane to at[8 j] when no symbol needs more than one
// byte: the next byte is always at hand, and the one after it is on its way.
// Returns how many were taken from `ring`, where the next one lies.
__device__ __forceinline__ int block_one(const rans_dec_table& F, const uint8_t* ring, uint8_t* at, uint32_t& x) {
  uint32_t pos = 0, b = ring[0];
#pragma unroll 8
  for (int j = 0; j < kBlockSteps; j++) {
    const uint32_t c = ring[pos + 1];
    uint32_t v;
    const uint32_t y = next_symbol(F, x, v);
    at[8 * j] = uint8_t(v);
    uint32_t to;
    select_ge(y, kRansLower, y, y * 256 + b, x, pos, pos + 1, to);
    b = select_ge(y, kRansLower, b, c);
    pos = to;
  }
  return int(pos);
}

// The same when a symbol may need two: the next stream bytes are the top
// `bits` bits of hi:lo (zeros below), and nw is the word after them, at byte
// pos of the ring.
struct rans_dec_window {
  uint32_t hi, lo, bits, nw, pos;
  // kHalf symbols
  static constexpr int kHalf = kBlockSteps / 2;
  __device__ __forceinline__ void half(const rans_dec_table& F, const uint8_t* ring, uint8_t* at, uint32_t& x) {
#pragma unroll 4
    for (int j = 0; j < kHalf; j += 2) {
      // At least 32 bits for two symbols.  Refilled without a branch (nearly
      // every time some lane needs a word): a shift by 32 or more gives 0, and
      // the load gives the same word again when nothing was taken.
      uint32_t more, step;
      select_ge(bits, 32, 0u, 32u, more, 0u, 4u, step);
      hi |= shift_right(nw, bits);
      lo |= shift_left(nw, 32 - bits);
      bits += more;
      pos += step;
      nw = __byte_perm(*reinterpret_cast<const uint32_t*>(ring + (pos & (kRing - 1))), 0, 0x0123);
      uint32_t A = hi, taken = 0;
#pragma unroll
      for (int i = 0; i < 2; i++) {
        uint32_t v, nb;
        const uint32_t y = next_symbol(F, x, v);
        at[8 * (j + i)] = uint8_t(v);
        select_ge(y, kRansLower, y, __funnelshift_l(A, y, 8), x, 0u, 8u, nb);
        select_ge(y, kRansLower >> 8, x, __funnelshift_l(A, y, 16), x, nb, 16u, nb);
        A <<= nb;
        taken += nb;
      }
      hi = __funnelshift_lc(lo, hi, taken);
      lo = shift_left(lo, taken);
      bits -= taken;
    }
  }
};

// One lane's part of a stream.  n: its symbols, 0 for a stream that is not decoded.
struct rans_dec_stream {
  uint64_t n;
  rans_freq t;
  const uint8_t *p, *end, *stream_end;   // the lane's bytes, the stream's end
  int64_t status;                        // what the stream's is to be
  bool given;                            // it is to be decoded
};
// Header checks as arithmetic_deserialize / arithmetic_decode (arithmetic.cc:403-495).
__device__ __forceinline__ rans_dec_stream open_stream(const uint8_t* base, int64_t size, int64_t cap, int only_v2,
                                                       int lane) {
  rans_dec_stream D = {};
  // Streams of another version are left to the learned decoder when asked
  // (whose CTAs that give up say nothing: the status stays this one)
  if (only_v2 && size >= 4 && get_u32(base) != 2) {
    D.status = PG_ERR_CUDA;
    return D;
  }
  D.status = PG_ERR_FORMAT;
  if (size < kHeader || get_u32(base) != 2) return D;
  uint64_t c[3], total = 0, start = 0;
  uint32_t mylen = 0;
  for (int k = 0; k < 3; k++) c[k] = get_u64(base + 4 + 8 * k);
  const uint64_t n = c[0] + c[1] + c[2];
  for (int l = 0; l < kLanes; l++) {
    const uint32_t len = get_u32(base + 28 + 4 * l);
    if (l < lane) start += len;
    if (l == lane) mylen = len;
    total += len;
  }
  if (c[0] > n || c[1] > n || c[2] > n || n > ~uint64_t(0) / 0x3fff) return D;
  if (total != uint64_t(size - kHeader)) return D;
  D.status = PG_ERR_CAPACITY;
  if (int64_t(n) > cap) return D;
  D.status = int64_t(n);
  D.given = true;
  D.n = n;
  D.t = make_freq(c);
  D.p = base + kHeader + start;
  D.end = D.p + mylen;
  D.stream_end = base + size;
  return D;
}
__device__ __forceinline__ rans_dec_table decoder_table(const rans_freq& t) {
  return rans_dec_table{t.freq[0], t.freq[1], t.freq[2], t.cum[1], t.cum[2]};
}

// In a batch of more streams than the warps of rans_decode_kernel that are
// resident at once (its rings leave room for 8 an SM), streams of up to
// kPlainSymbols are decoded here, byte by byte and by as many warps as fit: 65,536 of 512
// symbols 74 us (171 there), of 8,192 833 us (1,440), of 16,384 1.96 ms as there.
// The others get this status for now.
constexpr int kRingStreams = 8 * 148 * kWarpStreams;
constexpr int64_t kPlainSymbols = 12288, kLater = INT64_MIN;
__global__ void __launch_bounds__(256)
rans_decode_plain_kernel(const uint8_t* __restrict__ in, const int64_t* __restrict__ in_offsets,
                         const int64_t* __restrict__ in_sizes, int nstreams, uint8_t* __restrict__ symbols,
                         const int64_t* __restrict__ sym_offsets, const int64_t* __restrict__ sym_caps,
                         int64_t* __restrict__ status, int only_v2) {
  const int64_t s = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 3;
  const int lane = threadIdx.x & 7;
  if (s >= nstreams) return;
  const rans_dec_stream D = open_stream(in + in_offsets[s], in_sizes[s], sym_caps[s], only_v2, lane);
  const bool later = D.n > kPlainSymbols;
  if (lane == 0) status[s] = later ? kLater : D.status;
  if (!D.n || later) return;
  const rans_dec_table F = decoder_table(D.t);
  const uint8_t* p = D.p;
  uint32_t x = 0;
  for (int j = 0; j < 4 && p < D.end; j++) x = x << 8 | *p++;
  uint8_t* out = symbols + sym_offsets[s];
  for (int i = lane; i < int(D.n); i += kLanes) {
    uint32_t v;
    x = next_symbol(F, x, v);
    while (x < kRansLower && p < D.end) x = x << 8 | *p++;
    out[i] = uint8_t(v);
  }
}

// Four streams to a warp.  status[s]: number of symbols decoded, or
// PG_ERR_FORMAT / PG_ERR_CAPACITY.  REST: the streams left by
// rans_decode_plain_kernel among the kSpan of the CTA.
constexpr int kSpan = 8;
template<bool REST>
__global__ void __launch_bounds__(32)
rans_decode_kernel(const uint8_t* __restrict__ in, const int64_t* __restrict__ in_offsets,
                   const int64_t* __restrict__ in_sizes, int nstreams, uint8_t* __restrict__ symbols,
                   const int64_t* __restrict__ sym_offsets, const int64_t* __restrict__ sym_caps,
                   int64_t* __restrict__ status, int only_v2) {
  __shared__ __align__(16) uint8_t ring[32][kRingRow];
  __shared__ __align__(16) uint8_t stage[kWarpStreams][kOutRow];
  const int g = threadIdx.x >> 3, lane = threadIdx.x & 7;
  int64_t s = int64_t(blockIdx.x) * (REST ? kSpan : kWarpStreams);
  const int64_t s0 = s;
  unsigned mask = 0;   // streams s0 + bit that are left
  if (REST)
    mask = __ballot_sync(0xffffffffu, threadIdx.x < kSpan && s0 + threadIdx.x < nstreams &&
                                          status[s0 + threadIdx.x] == kLater);
  if (REST && !mask) return;
  do {
    if (REST) {   // the first four of them
      unsigned mine = mask;
      for (int i = 0; i < g; i++) mine &= mine - 1;
      for (int i = 0; i < kWarpStreams; i++) mask &= mask - 1;
      s = mine ? s0 + __ffs(mine) - 1 : nstreams;
    } else {
      s += g;
    }
    rans_dec_stream D = {};
    if (s < nstreams) {
      D = open_stream(in + in_offsets[s], in_sizes[s], sym_caps[s], only_v2, lane);
      if (lane == 0) status[s] = D.status;
    }
    const uint64_t n = D.n;
    const bool live = D.given;
    const uint8_t *p = D.p, *end = D.end, *stream_end = D.stream_end;
    uint32_t x = 0;
    for (int j = 0; j < 4 && p < end; j++) x = (x << 8) | *p++;
    const rans_dec_table F = decoder_table(D.t);
    const bool one_byte =
        __all_sync(0xffffffffu, !n || min(min(F.f0, F.f1), F.f2) >= kOneByteFreq);   // the same for the whole warp
    // The stream's bytes from the 16-byte boundary at or below p: byte k of
    // them goes to byte k % kRing of the ring.  The state has taken the first
    // `taken`; `filled` 16-byte granules have been asked for, and one replaces
    // only words that are used up.
    const uintptr_t src = reinterpret_cast<uintptr_t>(p) & ~uintptr_t(15);
    const int64_t extent = int64_t(reinterpret_cast<uintptr_t>(end) - src);
    uint8_t* myring = ring[threadIdx.x];
    int filled = 0;
    int64_t taken = int64_t(reinterpret_cast<uintptr_t>(p) - src);
    const int granules = int((extent + 15) / 16);   // (a lane has less than 2^32 bytes)
    const int whole = int(min(int64_t(granules), int64_t(reinterpret_cast<uintptr_t>(stream_end) - src) / 16));
    auto top_up = [&]() {
      const int to = min(int((taken + kRing) >> 4), granules);
#pragma unroll 1
      for (; filled < to; filled++) {
        const int o = (16 * filled) & (kRing - 1);
        const uint8_t* from = reinterpret_cast<const uint8_t*>(src) + 16 * int64_t(filled);
        const unsigned at = unsigned(__cvta_generic_to_shared(myring + o));
        if (filled < whole) {
          asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(at), "l"(from) : "memory");
          if (o < kMirror) asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(at + kRing), "l"(from) : "memory");
        } else {
          // the last bytes before the stream's end
          for (int k = 0; from + k < stream_end; k++) {
            myring[o + k] = from[k];
            if (o < kMirror) myring[kRing + o + k] = from[k];
          }
        }
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    rans_dec_window W = {};
    if (n) {
      top_up();
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
      W.pos = uint32_t(taken) & ~3u;
      const uint32_t skip = 8 * (uint32_t(taken) & 3);
      W.hi = __byte_perm(*reinterpret_cast<const uint32_t*>(myring + W.pos), 0, 0x0123) << skip;
      W.bits = 32 - skip;
      W.pos += 4;
      W.nw = __byte_perm(*reinterpret_cast<const uint32_t*>(myring + W.pos), 0, 0x0123);
    }
    // Symbols are staged by output address: row byte v of block k is byte
    // k kBlockSyms + v from the 16-byte boundary at or below the stream's first,
    // so a block's last `shift` symbols lie past kBlockSyms and move to the
    // row's start when the rest has left.
    uint8_t* out = live ? symbols + sym_offsets[s] : nullptr;
    const int shift = int(reinterpret_cast<uintptr_t>(out) & 15);
    uint8_t* out0 = out - shift;
    uint8_t* row = stage[g];
    const int64_t blocks = int64_t((n + kBlockSyms - 1) / kBlockSyms);
    const unsigned long long most = __reduce_max_sync(0xffffffffu, unsigned(min(blocks, int64_t(0x7fffffff))));
    // The fast forms take a block when its lane cannot run out of bytes in it
    // and the state is a coder's (2^23 .. 2^31, so that no symbol needs a third
    // byte).  The stream's end, or damage, takes the careful form from there on.
    const int enough = one_byte ? kBlockSteps : 2 * kBlockSteps;
    bool careful = false;
    for (int64_t k = 0; k < int64_t(most); k++) {
      if (k < blocks) {
        uint8_t* at = row + shift + lane;
        careful = careful || extent - taken < enough || x < kRansLower || x >= (1u << 31) ||
                  uint64_t(k + 1) * kBlockSyms > n;
        if (!careful && one_byte) {
          top_up();
          asm volatile("cp.async.wait_group 2;\n" ::: "memory");
          taken += block_one(F, myring + (int(taken) & (kRing - 1)), at, x);
        } else if (!careful) {
#pragma unroll 1
          for (int i = 0; i < 2; i++) {
            top_up();
            asm volatile("cp.async.wait_group 2;\n" ::: "memory");
            const uint32_t before = W.pos - (W.bits >> 3);
            W.half(F, myring, at + 8 * W.kHalf * i, x);
            taken += W.pos - (W.bits >> 3) - before;
          }
        } else {
          top_up();
          asm volatile("cp.async.wait_group 0;\n" ::: "memory");
          const int steps = int(min(int64_t(kBlockSteps), (int64_t(n) - k * kBlockSyms - lane + kLanes - 1) / kLanes));
          for (int j = 0; j < steps; j++) {
            uint32_t v;
            x = next_symbol(F, x, v);
            at[8 * j] = uint8_t(v);
            while (x < kRansLower && taken < extent) {
              // (a damaged state can take more in a block than the ring holds)
              x = x << 8 | (taken < 16 * int64_t(filled) ? myring[taken & (kRing - 1)]
                                                         : *(reinterpret_cast<const uint8_t*>(src) + taken));
              taken++;
            }
          }
        }
      }
      __syncwarp();
      if (k < blocks) {
        // Row bytes below kBlockSyms are complete (and, after the last block,
        // those up to the stream's end).  The first block of an unaligned
        // stream and the last leave by bytes.
        const int from = k ? 0 : shift;
        const int stop = k == blocks - 1 ? int(shift + int64_t(n) - k * kBlockSyms) : kBlockSyms;
        uint8_t* o = out0 + k * kBlockSyms;
        if (from == 0 && stop == kBlockSyms) {
          uint4 w[kBlockSyms / 16 / kLanes];
#pragma unroll
          for (int i = 0; i < kBlockSyms / 16 / kLanes; i++)
            w[i] = reinterpret_cast<const uint4*>(row)[lane + kLanes * i];
#pragma unroll
          for (int i = 0; i < kBlockSyms / 16 / kLanes; i++) reinterpret_cast<uint4*>(o)[lane + kLanes * i] = w[i];
        } else {
          for (int v = 16 * lane; v < stop; v += 16 * kLanes)
            for (int e = max(v, from); e < min(v + 16, stop); e++) o[e] = row[e];
        }
        __syncwarp(0xffu << (8 * g));
        if (lane == 0) *reinterpret_cast<uint4*>(row) = *reinterpret_cast<const uint4*>(row + kBlockSyms);
      }
      __syncwarp();
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    if (REST) __syncwarp();
  } while (REST && mask);
}

int64_t rans_stream_bound(int64_t n) { return stream_bound(n); }

template<int64_t OWN>
static int launch_rans_encoders(const uint8_t* symbols, const int64_t* offsets, int nstreams, uint8_t* out,
                                const int64_t* out_offsets, int64_t* sizes, const int64_t* expect,
                                cudaStream_t stream) {
  const int ctas = nstreams < kLongCtas ? nstreams : kLongCtas;
  rans_count_kernel<<<ctas, kLongThreads, 0, stream>>>(symbols, offsets, nstreams, OWN, expect, out, out_offsets);
  PG_CUDA(cudaGetLastError());
  rans_encode_kernel<OWN><<<(nstreams + kWarpStreams - 1) / kWarpStreams, 32, 0, stream>>>(
      symbols, offsets, nstreams, out, out_offsets, sizes, expect);
  PG_CUDA(cudaGetLastError());
  rans_pack_kernel<<<ctas, kLongThreads, 0, stream>>>(offsets, nstreams, OWN, expect, out, out_offsets, sizes);
  PG_CUDA(cudaGetLastError());
  return PG_OK;
}

int launch_rans_encode(const uint8_t* symbols, const int64_t* offsets, int nstreams, uint8_t* out,
                       const int64_t* out_offsets, int64_t* sizes, const int64_t* expect, cudaStream_t stream) {
  return (nstreams > 1024 ? launch_rans_encoders<kOwnOfMany> : launch_rans_encoders<kOwnOfFew>)(
      symbols, offsets, nstreams, out, out_offsets, sizes, expect, stream);
}

int launch_rans_decode(const uint8_t* in, const int64_t* in_offsets, const int64_t* in_sizes, int nstreams,
                       uint8_t* symbols, const int64_t* sym_offsets, const int64_t* sym_caps, int64_t* status,
                       int only_v2, cudaStream_t stream) {
  const int rest = nstreams > kRingStreams;
  if (rest) {
    rans_decode_plain_kernel<<<unsigned((int64_t(nstreams) * kLanes + 255) / 256), 256, 0, stream>>>(
        in, in_offsets, in_sizes, nstreams, symbols, sym_offsets, sym_caps, status, only_v2);
    PG_CUDA(cudaGetLastError());
  }
  const int each = rest ? kSpan : kWarpStreams;
  (rest ? rans_decode_kernel<true> : rans_decode_kernel<false>)<<<(nstreams + each - 1) / each, 32, 0, stream>>>(
      in, in_offsets, in_sizes, nstreams, symbols, sym_offsets, sym_caps, status, only_v2);
  PG_CUDA(cudaGetLastError());
  return PG_OK;
}

// Ternary symbols of solved nodes in the on-disk convention
// (shard/shard.cc:448-449 after end/check.cc:154-156, 197-200): for rotation r
// of node k, symbol = black wins + 2 white wins.  Nodes are [we-win,
// we-win-or-tie] for the player to move; `turn` = 1 when white moves.
// A thread writes 16 symbols in one 16-byte store, so a warp's stores are
// contiguous: 1 G symbols in 0.26 ms, 5.1 TB/s (6.1 ms with one thread per 64
// symbols, byte by byte).  An output that is not 16-byte aligned is
// written by bytes.
__device__ __forceinline__ uint32_t spread_nibble(uint32_t x) { return (x & 15) * 0x00204081u & 0x01010101u; }
__global__ void node_symbols_kernel(const uint16_t* __restrict__ nodes, int64_t n, int turn,
                                    uint8_t* __restrict__ symbols) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;  // one thread per 16 symbols
  if (i >= n * 16) return;
  const int64_t k = i >> 4;
  const int w = int(i & 15);
  const uint32_t win = nodes[32 * k + w], lost = ~uint32_t(nodes[32 * k + 16 + w]);
  const uint32_t black = turn ? lost : win, white = turn ? win : lost;
  uint32_t v[4];
#pragma unroll
  for (int q = 0; q < 4; q++) v[q] = spread_nibble(black >> (4 * q)) + 2 * spread_nibble(white >> (4 * q));
  uint8_t* out = symbols + 16 * i;
  if ((reinterpret_cast<uintptr_t>(symbols) & 15) == 0) {
    *reinterpret_cast<uint4*>(out) = make_uint4(v[0], v[1], v[2], v[3]);
  } else {
#pragma unroll
    for (int b = 0; b < 16; b++) out[b] = uint8_t(v[b >> 2] >> (8 * (b & 3)));
  }
}

// The inverse: nodes of the side to move from their symbols (one thread per
// 64 symbols, read as four 16-byte words).
__global__ void symbols_nodes_kernel(const uint8_t* __restrict__ symbols, int64_t n, int turn,
                                     uint64_t* __restrict__ nodes) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n * 4) return;
  const int64_t k = i >> 2;
  const int w = int(i & 3);
  const uint4* in = reinterpret_cast<const uint4*>(symbols + 64 * i);
  uint64_t black = 0, white = 0;
#pragma unroll
  for (int v = 0; v < 4; v++) {
    const uint4 q = in[v];
    const uint32_t part[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int p = 0; p < 4; p++)
#pragma unroll
      for (int b = 0; b < 4; b++) {
        const uint32_t sym = part[p] >> (8 * b) & 0xff;
        const int bit = 16 * v + 4 * p + b;
        black |= uint64_t(sym == 1) << bit;
        white |= uint64_t(sym == 2) << bit;
      }
  }
  nodes[8 * k + w] = turn ? white : black;
  nodes[8 * k + 4 + w] = ~(turn ? black : white);
}

// Copy stream s (in + in_offsets[s], sizes[s] bytes) to out + out_offsets[s]:
// one CTA per stream, 16-byte words where both ends allow it.
__global__ void pack_streams_kernel(const uint8_t* __restrict__ in, const int64_t* __restrict__ in_offsets,
                                    const int64_t* __restrict__ sizes, uint8_t* __restrict__ out,
                                    const int64_t* __restrict__ out_offsets) {
  const int s = blockIdx.x;
  const uint8_t* src = in + in_offsets[s];
  uint8_t* dst = out + out_offsets[s];
  const int64_t n = sizes[s];
  if (((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0) {
    const int64_t w = n >> 4;
    for (int64_t i = threadIdx.x; i < w; i += blockDim.x)
      reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(src)[i];
    for (int64_t i = 16 * w + threadIdx.x; i < n; i += blockDim.x) dst[i] = src[i];
  } else {
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) dst[i] = src[i];
  }
}

}  // namespace pg

using namespace pg;

extern "C" int pg_symbols_nodes(const uint8_t* symbols, int64_t n, int turn, uint64_t* nodes, void* stream) {
  if (n < 0 || (n && (!symbols || !nodes))) return fail(PG_ERR_ARG, "bad node count");
  if (reinterpret_cast<uintptr_t>(symbols) & 15) return fail(PG_ERR_ARG, "symbols must be 16-byte aligned");
  if (!n) return PG_OK;
  const int64_t threads = 4 * n;
  symbols_nodes_kernel<<<unsigned((threads + 255) / 256), 256, 0, (cudaStream_t)stream>>>(symbols, n, turn & 1, nodes);
  PG_CUDA(cudaGetLastError());
  return PG_OK;
}

extern "C" int pg_pack_streams(const uint8_t* in, const int64_t* in_offsets, const int64_t* sizes, int n, uint8_t* out,
                               const int64_t* out_offsets, void* stream) {
  if (n < 0 || (n && (!in || !in_offsets || !sizes || !out || !out_offsets))) return fail(PG_ERR_ARG, "bad pack arguments");
  for (int s0 = 0; s0 < n; s0 += 65535) {
    const int k = n - s0 < 65535 ? n - s0 : 65535;
    pack_streams_kernel<<<k, 256, 0, (cudaStream_t)stream>>>(in, in_offsets + s0, sizes + s0, out, out_offsets + s0);
    PG_CUDA(cudaGetLastError());
  }
  return PG_OK;
}

extern "C" int64_t pg_rans_bound(int64_t n) { return n < 0 ? PG_ERR_ARG : stream_bound(n); }

extern "C" int pg_rans_encode_batch(const uint8_t* symbols, const int64_t* offsets, int nstreams, uint8_t* out,
                                    const int64_t* out_offsets, int64_t* sizes, void* stream) {
  if (nstreams < 0) return fail(PG_ERR_ARG, "bad stream count");
  if (!nstreams) return PG_OK;
  return launch_rans_encode(symbols, offsets, nstreams, out, out_offsets, sizes, nullptr, (cudaStream_t)stream);
}

extern "C" int pg_rans_decode_batch(const uint8_t* in, const int64_t* in_offsets, const int64_t* in_sizes,
                                    int nstreams, uint8_t* symbols, const int64_t* sym_offsets,
                                    const int64_t* sym_caps, int64_t* status, void* stream) {
  if (nstreams < 0) return fail(PG_ERR_ARG, "bad stream count");
  if (!nstreams) return PG_OK;
  return launch_rans_decode(in, in_offsets, in_sizes, nstreams, symbols, sym_offsets, sym_caps, status, 0,
                            (cudaStream_t)stream);
}

extern "C" int pg_node_symbols(const uint64_t* nodes, int64_t n, int turn, uint8_t* symbols, void* stream) {
  if (n < 0) return fail(PG_ERR_ARG, "bad node count");
  if (!n) return PG_OK;
  const int64_t threads = 16 * n;
  node_symbols_kernel<<<unsigned((threads + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      reinterpret_cast<const uint16_t*>(nodes), n, turn & 1, symbols);
  PG_CUDA(cudaGetLastError());
  return PG_OK;
}
