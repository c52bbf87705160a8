// Store coder: how the sweep keeps finished slices compressed in HBM.  No
// reference counterpart (the reference compresses blocks in memory with
// snappy, pentago/end/fast_compress.cc); this is an internal format that
// never leaves the device, so only its round trip is specified.
//
// A block of solved nodes is coded as the ternary symbols black wins + 2
// white wins of its 256 rotations per node (the on-disk convention), with
// static rANS (14-bit frequencies, byte renormalization at 2^23) whose
// frequencies depend on a context of five already-coded symbols: the same
// node one step back along each of the four rotation axes (3 where the
// coordinate is 0) and the same rotation of the previous node of the lane.
// One frequency table (1024 contexts x 3) serves a whole batch of blocks.
// A block's 32 lanes (one warp) each take a contiguous run of its nodes, so
// every context symbol is on the lane that codes the symbol and the lanes
// decode in parallel.  Stream layout: 32 lane lengths (u32), then the lanes'
// bytes; a block that some lane cannot code within its nodes' raw size is
// stored raw instead (first length ~0, then the 64-byte nodes), so a stream
// never needs more than its raw size plus 128 + 32 x 64 bytes.
#include "../../include/pentago_b200.h"
#include "coder.cuh"
#include "runtime.h"
#include <cstdint>

namespace pg {
namespace {

constexpr int kCtx = 1024;
constexpr int kLanesS = 32;   // lanes per block: one warp
constexpr uint32_t kTotBits = 14, kTot = 1u << kTotBits, kLow = 1u << 23;
constexpr int kHead = 4 * kLanesS;
// Threads of a CTA of the coder kernels: one CTA fills an SM, so that the
// tables of a batch are in shared memory once per SM.
constexpr int kThreads = 1024;
// A batch's frequency table counts the contexts of at most this many of its
// blocks, spread evenly over it (about 2 G symbols for full blocks).
constexpr int kTableBlocks = 2048;

// Nodes per lane of a block of n nodes.
__host__ __device__ inline int lane_nodes(int n) { return (n + kLanesS - 1) / kLanesS; }
__host__ __device__ inline int64_t lane_cap(int n) { return int64_t(lane_nodes(n)) * 64 + 64; }
__host__ __device__ inline int64_t store_bound(int n) { return kHead + kLanesS * lane_cap(n); }

// Bit i of the low half to bit 2 i, bit i of the high half to bit 2 i + 1,
// and back.
__device__ __forceinline__ uint32_t shuffle16(uint32_t x) {
  x = __byte_perm(x, 0, 0x3120);
  uint32_t t = (x ^ (x >> 4)) & 0x00f000f0u;
  x ^= t ^ (t << 4);
  t = (x ^ (x >> 2)) & 0x0c0c0c0cu;
  x ^= t ^ (t << 2);
  t = (x ^ (x >> 1)) & 0x22222222u;
  return x ^ t ^ (t << 1);
}
__device__ __forceinline__ uint32_t unshuffle16(uint32_t x) {
  uint32_t t = (x ^ (x >> 1)) & 0x22222222u;
  x ^= t ^ (t << 1);
  t = (x ^ (x >> 2)) & 0x0c0c0c0cu;
  x ^= t ^ (t << 2);
  t = (x ^ (x >> 4)) & 0x00f000f0u;
  x ^= t ^ (t << 4);
  return __byte_perm(x, 0, 0x3120);
}

// Symbols of one node packed 2 bits each (16 per word, rotation r at bits
// 2 (r & 15) of word r >> 4): black bit + 2 white bit, for the side-to-move
// form [win, win or tie] of the sweep.  A node's words live kThreads words
// apart in shared memory: the coder threads keep theirs in columns, so that a
// warp whose threads read the same word index reads 32 different banks.
__device__ __forceinline__ void pack_node(const uint64_t* node, bool wide, int turn, uint32_t* sym) {
#pragma unroll
  for (int h = 0; h < 2; h++) {
    uint32_t win[4], nl[4];   // words 4 h .. 4 h + 3 of the two supers
    if (wide) {
      const uint4 a = reinterpret_cast<const uint4*>(node)[h], b = reinterpret_cast<const uint4*>(node)[2 + h];
      win[0] = a.x; win[1] = a.y; win[2] = a.z; win[3] = a.w;
      nl[0] = b.x; nl[1] = b.y; nl[2] = b.z; nl[3] = b.w;
    } else {
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const uint64_t a = node[2 * h + i], b = node[4 + 2 * h + i];
        win[2 * i] = uint32_t(a); win[2 * i + 1] = uint32_t(a >> 32);
        nl[2 * i] = uint32_t(b); nl[2 * i + 1] = uint32_t(b >> 32);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t black = turn ? ~nl[i] : win[i], white = turn ? win[i] : ~nl[i];
      sym[kThreads * (8 * h + 2 * i)] = shuffle16(__byte_perm(black, white, 0x5410));
      sym[kThreads * (8 * h + 2 * i + 1)] = shuffle16(__byte_perm(black, white, 0x7632));
    }
  }
}
// And back to the node.
__device__ __forceinline__ void unpack_node(const uint32_t* sym, int turn, bool wide, uint64_t* node) {
#pragma unroll
  for (int h = 0; h < 2; h++) {
    uint32_t win[4], nl[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t lo = unshuffle16(sym[kThreads * (8 * h + 2 * i)]);
      const uint32_t hi = unshuffle16(sym[kThreads * (8 * h + 2 * i + 1)]);
      const uint32_t black = __byte_perm(lo, hi, 0x5410), white = __byte_perm(lo, hi, 0x7632);
      win[i] = turn ? white : black;
      nl[i] = ~(turn ? black : white);
    }
    if (wide) {
      reinterpret_cast<uint4*>(node)[h] = make_uint4(win[0], win[1], win[2], win[3]);
      reinterpret_cast<uint4*>(node)[2 + h] = make_uint4(nl[0], nl[1], nl[2], nl[3]);
    } else {
#pragma unroll
      for (int i = 0; i < 2; i++) {
        node[2 * h + i] = uint64_t(win[2 * i + 1]) << 32 | win[2 * i];
        node[4 + 2 * h + i] = uint64_t(nl[2 * i + 1]) << 32 | nl[2 * i];
      }
    }
  }
}

// The contexts of a word's 16 rotations (r = 16 w + i) come from five words.
// Axis 0's neighbour r - 1 and axis 1's r - 4 are symbols i - 1 and i - 4 of
// the same word (none where i % 4 == 0, resp. i < 4); axis 2's r - 16 and
// axis 3's r - 64 are words w - 1 and w - 4 (none where w % 4 == 0, resp.
// w < 4); the previous node's symbol is its word w.  A missing neighbour
// reads as 3.
constexpr uint32_t kNoAxis0 = 0x03030303u, kNoAxis1 = 0x000000ffu;

// 2-bit fields of two words side by side, hi field above lo field, in
// nibbles: of the even symbols, of the odd ones.
constexpr uint32_t kEven = 0x33333333u;
__device__ __forceinline__ uint32_t even_pairs(uint32_t hi, uint32_t lo) { return (hi & kEven) << 2 | (lo & kEven); }
__device__ __forceinline__ uint32_t odd_pairs(uint32_t hi, uint32_t lo) { return (hi & ~kEven) | (lo >> 2 & kEven); }

// Context and symbol of all 16 rotations of a word, 16 (4 c + symbol) each:
// rotation i's at half i >> 2 & 1 of at[i >> 3][i & 3].  (c = a0 a1 a2 a3
// ap, two bits each, a0 highest.)
struct word_index {
  uint32_t at[2][4];
  __device__ __forceinline__ word_index(uint32_t x, uint32_t a2, uint32_t a3, uint32_t ap) {
    const uint32_t a0 = x << 2 | kNoAxis0, a1 = x << 8 | kNoAxis1;
    const uint32_t hi[2] = {even_pairs(a0, a1), odd_pairs(a0, a1)};
    const uint32_t mid[2] = {even_pairs(a2, a3), odd_pairs(a2, a3)};
    const uint32_t low[2] = {even_pairs(ap, x), odd_pairs(ap, x)};
#pragma unroll
    for (int o = 0; o < 2; o++) {
      // nibbles 0, 2, 4, 6 (rotations 4 j + o), then 1, 3, 5, 7 (4 j + 2 + o)
      const uint32_t b0 = (hi[o] << 4 & 0xf0f0f0f0u) | (mid[o] & 0x0f0f0f0fu), l0 = low[o] << 4 & 0xf0f0f0f0u;
      const uint32_t b1 = (hi[o] & 0xf0f0f0f0u) | (mid[o] >> 4 & 0x0f0f0f0fu), l1 = low[o] & 0xf0f0f0f0u;
      at[0][o] = __byte_perm(l0, b0, 0x5140);
      at[1][o] = __byte_perm(l0, b0, 0x7362);
      at[0][2 + o] = __byte_perm(l1, b1, 0x5140);
      at[1][2 + o] = __byte_perm(l1, b1, 0x7362);
    }
  }
  __device__ __forceinline__ uint32_t operator()(int i) const {
    const uint32_t t = at[i >> 3][i & 3];
    return i & 4 ? t >> 16 : t & 0xffff;
  }
};

// Context counts over every stride-th block of a batch: a thread takes 16
// rotations of a node (it packs the four words their contexts come from for
// itself).  Bound by the shared-memory counters: most symbols of a solved
// slice fall on a few of them, and a warp's additions to one address go one
// after another, so there are kCopies of each counter, used by different
// lanes.  2,000 blocks: 1.3 ms (4.9 with one copy, a thread per rotation and two
// barriers a node).
constexpr int kCopies = 8;
constexpr size_t kHistSmem = sizeof(unsigned) * 4 * kCtx * kCopies;
__global__ void __launch_bounds__(kThreads)
store_hist_kernel(const uint64_t* __restrict__ nodes, const int64_t* __restrict__ first,
                  const int32_t* __restrict__ count, int nblocks, int stride, int turn, unsigned* __restrict__ hist) {
  extern __shared__ __align__(16) unsigned char smem[];
  unsigned* h = reinterpret_cast<unsigned*>(smem);   // [4 c + symbol][copy]
  for (int i = threadIdx.x; i < 4 * kCtx * kCopies; i += kThreads) h[i] = 0;
  __syncthreads();
  unsigned* mine = h + threadIdx.x % kCopies;
  for (int64_t b = int64_t(blockIdx.x) * stride; b < nblocks; b += int64_t(gridDim.x) * stride) {
    const int n = count[b], m = lane_nodes(n);
    const uint16_t* base = reinterpret_cast<const uint16_t*>(nodes + 8 * first[b]);
    for (int64_t t = threadIdx.x; t < 16 * int64_t(n); t += kThreads) {
      const int k = int(t >> 4), w = int(t & 15);
      const uint16_t* node = base + 32 * int64_t(k);
      auto word = [&](const uint16_t* p) {
        const uint32_t win = p[0], lost = uint16_t(~p[16]);
        return shuffle16(turn ? lost | win << 16 : win | lost << 16);
      };
      const word_index at(word(node + w), w & 3 ? word(node + w - 1) : ~0u, w >= 4 ? word(node + w - 4) : ~0u,
                          k % m ? word(node - 32 + w) : ~0u);
#pragma unroll
      for (int i = 0; i < 16; i++) atomicAdd(mine + (at(i) >> 4) * kCopies, 1u);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 4 * kCtx; i += kThreads) {
    unsigned s = 0;
    for (int c = 0; c < kCopies; c++) s += h[i * kCopies + c];
    if (s && (i & 3) < 3) atomicAdd(hist + 3 * (i >> 2) + (i & 3), s);
  }
}

// Frequencies per context from its counts: proportional, at least 1, the
// rounding left on the largest (uniform when the context never occurs).
__global__ void store_table_kernel(const unsigned* __restrict__ hist, uint16_t* __restrict__ freq) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= kCtx) return;
  const uint64_t n[3] = {hist[3 * c], hist[3 * c + 1], hist[3 * c + 2]};
  const uint64_t sum = n[0] + n[1] + n[2];
  uint32_t f[3];
  if (!sum) {
    f[0] = kTot - 2 * (kTot / 3);
    f[1] = f[2] = kTot / 3;
  } else {
    for (int i = 0; i < 3; i++) {
      f[i] = uint32_t(n[i] * kTot / sum);
      if (!f[i]) f[i] = 1;
    }
    const int big = f[1] > f[0] ? (f[2] > f[1] ? 2 : 1) : (f[2] > f[0] ? 2 : 0);
    f[big] = uint32_t(int32_t(f[big]) + int32_t(kTot) - int32_t(f[0] + f[1] + f[2]));
  }
  for (int i = 0; i < 3; i++) freq[3 * c + i] = uint16_t(f[i]);
}

// ---------------------------------------------------------------------------
// Encode: one warp per block; lane l codes its run of nodes backward, each
// node's rotations from 255 to 0, into its own slot, then the lanes are packed
// behind the header.
//
// Bound by instructions (the batch keeps every warp slot of an SM busy), so a
// symbol costs as few as possible: a word's 16 table offsets come from eleven
// word operations on packed fields, everything the coder needs of a context
// and symbol is one 16-byte shared load (64 KB of tables, once per SM: hence
// one CTA of 1,024 threads), a renormalization is selects, and its bytes
// gather in a register and leave as whole words.  17.6 M nodes (6,000 blocks)
// of a solved slice: 6.6 ms (30 instructions a symbol, 20 of
// them on the ALU pipe).

// {xmax, rcp, bias, shift | cmpl << 5} of context c and symbol v at
// 4 c + v: the encoder divides the state by the frequency f with a
// reciprocal multiply, as in F. Giesen's ryg_rans (after Alverson, "Integer
// division using reciprocals", 1991): with 2^(sh-1) < f <= 2^sh, rcp =
// ceil(2^(sh+31) / f) gives state / f = umulhi(state, rcp) >> (sh - 1) for
// every state below 2^31 (renormalization keeps it below 2^17 f <= 2^31), and
// the new state is state + bias + (state / f) (2^14 - f).  f = 1 takes rcp =
// 2^32 - 1, shift 0 and a bias of 2^14 - 1 more, which yields the same.
__device__ __forceinline__ void encoder_table(const uint16_t* __restrict__ freq, uint4* E) {
  for (int i = threadIdx.x; i < 4 * kCtx; i += kThreads) {
    const int c = i >> 2, v = min(i & 3, 2);
    const uint32_t f = freq[3 * c + v];
    const uint32_t cum = v == 0 ? 0u : v == 1 ? freq[3 * c] : uint32_t(freq[3 * c]) + freq[3 * c + 1];
    uint32_t sh = 0;
    while (f > (1u << sh)) sh++;
    const uint32_t rcp = f < 2 ? ~0u : uint32_t(((uint64_t(1) << (sh + 31)) + f - 1) / f);
    E[i] = make_uint4(f << 17, rcp, cum + (f < 2 ? kTot - 1 : 0u), (f < 2 ? 0u : sh - 1) | (kTot - f) << 5);
  }
}

// The next block of a warp, -1 when there is none: warps draw them from a
// counter, the large ones first (a batch's ragged blocks are a quarter or a
// sixteenth of its full ones; with a fixed share of the batch a third of the
// warps and a quarter of the SMs' time stayed idle).
constexpr int kLarge = 2048;   // nodes
__device__ __forceinline__ int next_block(int* next, const int32_t* __restrict__ count, int nblocks) {
  // (a small batch is spread over the CTAs, not taken by the first of them)
  if (int(threadIdx.x / 32) * int(gridDim.x) >= nblocks) return -1;
  for (;;) {
    int j = 0;
    if (threadIdx.x % 32 == 0) j = atomicAdd(next, 1);
    j = __shfl_sync(0xffffffffu, j, 0);
    if (j >= 2 * nblocks) return -1;
    const int b = j < nblocks ? j : j - nblocks;
    if ((count[b] >= kLarge) == (j < nblocks)) return b;
  }
}

// Shared memory of the encoder: the table, then the threads' current and
// previous node.
constexpr size_t kEncSmem = sizeof(uint4) * 4 * kCtx + sizeof(uint32_t) * 32 * kThreads;

__global__ void __launch_bounds__(kThreads)
store_encode_kernel(const uint64_t* __restrict__ nodes, const int64_t* __restrict__ first,
                    const int32_t* __restrict__ count, int nblocks, int turn, const uint16_t* __restrict__ freq,
                    uint8_t* __restrict__ out, const int64_t* __restrict__ out_offsets, int64_t* __restrict__ sizes,
                    int* __restrict__ next) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint4* E = reinterpret_cast<uint4*>(smem);
  uint32_t* buf = reinterpret_cast<uint32_t*>(smem + sizeof(uint4) * 4 * kCtx) + threadIdx.x;
  encoder_table(freq, E);
  __syncthreads();
  const int lane = threadIdx.x % 32;
  const bool wide = (reinterpret_cast<uintptr_t>(nodes) & 15) == 0;
  for (int b; (b = next_block(next, count, nblocks)) >= 0;) {
    const int n = count[b], m = lane_nodes(n);
    const int k0 = lane * m, k1 = min(n, k0 + m);
    const uint64_t* base = nodes + 8 * first[b];
    uint8_t* sbase = out + out_offsets[b];
    const int cap = int(lane_cap(n));
    uint8_t* slot = sbase + kHead + int64_t(lane) * cap;
    const bool words = (reinterpret_cast<uintptr_t>(sbase) & 3) == 0;
    // The state; the bytes not yet stored (the top `bits` bits of hi:lo, the
    // oldest byte lowest); the stored ones are slot[off .. cap), as far as
    // they fit.
    uint32_t x = kLow, hi = 0, lo = 0, bits = 0;
    int off = cap;
    auto put = [&](const uint4 P) {
      uint32_t y, nb;
      const uint32_t x8 = x >> 8;
      select_ge(x, P.x, x8, x, y, 8u, 0u, nb);
      select_ge(x8, P.x, x >> 16, y, y, 16u, nb, nb);
      lo = __funnelshift_r(lo, hi, nb);
      hi = __funnelshift_r(hi, x, nb);
      bits += nb;
      const uint32_t q = __funnelshift_r(__umulhi(y, P.y), 0u, P.w);   // a shift by P.w mod 32
      x = y + P.z + q * (P.w >> 5);
    };
    auto flush = [&]() {
      if (bits >= 32) {
        const uint32_t w = __byte_perm(__funnelshift_rc(lo, hi, 64 - bits), 0, 0x0123);
        off -= 4;
        bits -= 32;
        if (off >= 0) {
          if (words) {
            *reinterpret_cast<uint32_t*>(slot + off) = w;
          } else {
            for (int j = 0; j < 4; j++) slot[off + j] = uint8_t(w >> (8 * j));
          }
        }
      }
    };
    uint32_t* cur = buf;
    uint32_t* prev = buf + 16 * kThreads;
    if (k1 > k0) pack_node(base + 8 * int64_t(k1 - 1), wide, turn, cur);
    for (int k = k1 - 1; k >= k0; k--) {
      const bool has_prev = k > k0;
      if (has_prev) pack_node(base + 8 * int64_t(k - 1), wide, turn, prev);
#pragma unroll 1
      for (int w = 15; w >= 0; w--) {
        const word_index at(cur[kThreads * w], w & 3 ? cur[kThreads * (w - 1)] : ~0u,
                            w >= 4 ? cur[kThreads * (w - 4)] : ~0u, has_prev ? prev[kThreads * w] : ~0u);
#pragma unroll
        for (int i = 15; i > 0; i -= 2) {
          put(*reinterpret_cast<const uint4*>(smem + at(i)));
          put(*reinterpret_cast<const uint4*>(smem + at(i - 1)));
          flush();
        }
      }
      uint32_t* t = cur; cur = prev; prev = t;
    }
    // A lane that passes its nodes' raw size (its slot, with the final state)
    // makes the block raw.
    if (__any_sync(0xffffffffu, off - int(bits >> 3) < 4)) {
      __syncwarp();
      const int64_t nw = 8 * int64_t(n);
      uint8_t* raw = sbase + kHead;
      if ((reinterpret_cast<uintptr_t>(raw) & 7) == 0) {
        for (int64_t i = lane; i < nw; i += kLanesS) reinterpret_cast<uint64_t*>(raw)[i] = base[i];
      } else {
        for (int64_t i = lane; i < nw; i += kLanesS)
          for (int j = 0; j < 8; j++) raw[8 * i + j] = uint8_t(base[i] >> (8 * j));
      }
      for (int j = lane; j < kHead; j += 32) sbase[j] = j < 4 ? 0xff : 0;
      if (lane == 0) sizes[b] = kHead + 8 * nw;
      continue;
    }
    for (; bits; bits -= 8) slot[--off] = uint8_t((uint64_t(hi) << 32 | lo) >> (64 - bits));
    for (int j = 0; j < 4; j++) slot[--off] = uint8_t(x >> (8 * j));
    const uint32_t len = uint32_t(cap - off);
    // Destination of this lane's bytes behind the header: the lengths of the
    // lanes before it (an exclusive warp scan), and the stream's total.
    uint32_t before = len;
#pragma unroll
    for (int o = 1; o < kLanesS; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, before, o);
      if (lane >= o) before += v;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, before, kLanesS - 1);
    before -= len;
    __syncwarp();
    // The lanes' bytes move down, one lane after another.  A lane's
    // destination never passes its own source nor a later lane's (each lane's
    // bytes fit its slot).
    for (int l = 0; l < kLanesS; l++) {
      const uint32_t len_l = __shfl_sync(0xffffffffu, len, l);
      const uint32_t dst_l = __shfl_sync(0xffffffffu, before, l);
      move_down<32, 8>(sbase + kHead + dst_l, sbase + kHead + int64_t(l + 1) * cap - len_l, len_l, lane,
                       [] { __syncwarp(); });
    }
    for (int j = 0; j < 4; j++) sbase[4 * lane + j] = uint8_t(len >> (8 * j));
    if (lane == 0) sizes[b] = kHead + int64_t(total);
  }
}

// ---------------------------------------------------------------------------
// Decode: lane l decodes its nodes forward into shared memory, one node at a
// time, and writes each finished node (64 bytes) to its place.  status[b] =
// nodes decoded, or PG_ERR_FORMAT for a stream that does not end exactly
// where its lengths say with the initial state.
//
// Bound by instructions like the encoder.  A context's two boundaries between
// its symbols are one word of a table, a symbol's frequency and start another; the part of its index that earlier
// words give is made for 16 symbols at once.  The next 32 stream bits are
// picked from a ring in shared memory before every two symbols (which take at
// most that many); the ring's words lie in the thread's column and come by
// asynchronous copies, eight symbols ahead.  17.6 M nodes: 6.6 ms
// (36 instructions a symbol, 22 on the ALU pipe).

constexpr int kRing = 16;   // words of a lane's ring; row kRing repeats row 0
constexpr int kDecTable = 5 * kCtx;   // words of the tables
constexpr size_t kDecSmem = sizeof(uint32_t) * (kDecTable + (32 + kRing + 1) * kThreads);

// Of the context with fields a0, a1, a2, a3, ap, at index c = a2 a3 ap a1 a0:
// D[c] = c1 | c2 << 16 (where symbols 1 and 2 start), and frequency | start
// << 16 of its symbol v at D[kCtx + 4 c + v].
__device__ __forceinline__ void decoder_table(const uint16_t* __restrict__ freq, uint32_t* D) {
  for (int c = threadIdx.x; c < kCtx; c += kThreads) {
    const int at = (c & 63) << 4 | (c >> 6 & 3) << 2 | c >> 8;
    const uint32_t f0 = freq[3 * c], f1 = freq[3 * c + 1], f2 = freq[3 * c + 2];
    D[at] = f0 | (f0 + f1) << 16;
    D[kCtx + 4 * at] = f0;
    D[kCtx + 4 * at + 1] = f1 | f0 << 16;
    D[kCtx + 4 * at + 2] = f2 | (f0 + f1) << 16;
    D[kCtx + 4 * at + 3] = 0;
  }
}

// The symbol that x's low bits name in the context at byte 4 c of D, times
// four, and the state after it, before it is refilled.
__device__ __forceinline__ uint32_t next_symbol(const unsigned char* D, uint32_t c4, uint32_t x, uint32_t& v4) {
  const uint32_t starts = *reinterpret_cast<const uint32_t*>(D + c4);
  const uint32_t slot = x & (kTot - 1);
  v4 = select_ge(slot, starts >> 16, 8u, select_ge(slot, starts & 0xffff, 4u, 0u));
  const uint32_t e = *reinterpret_cast<const uint32_t*>(D + 4 * kCtx + 4 * c4 + v4);
  return (e & 0xffff) * (x >> kTotBits) + (slot - (e >> 16));
}

// A lane's stream bytes from the word boundary at or below its first, in its
// column of the ring: word w at row w % kRing.
struct lane_ring {
  const uint8_t* src;    // word 0
  unsigned column;       // the lane's column of the ring (shared address)
  int asked, words;      // words asked for; words that hold the lane's bytes
  int whole;             // words that lie inside the stream: nothing is read past its end
  // Four more words when there is room for them above bit `pos`.
  __device__ __forceinline__ void top_up(uint32_t pos) {
    if (asked < words && asked - int(pos >> 5) <= kRing - 4) {
      const uint8_t* from = src + 4 * int64_t(asked);
      const unsigned to = column + (asked & (kRing - 1)) * (4 * kThreads);
      if (asked + 4 <= whole) {
#pragma unroll
        for (int i = 0; i < 4; i++) copy(to + 4 * kThreads * i, from + 4 * i);
        if ((asked & (kRing - 1)) == 0) copy(to + 4 * kThreads * kRing, from);
      } else {
        tail(to, from);
      }
      asked += 4;
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  static __device__ __forceinline__ void copy(unsigned to, const uint8_t* from) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(to), "l"(from) : "memory");
  }
  // The stream's last words, up to three bytes of them outside it
  const uint8_t* stop;
  __device__ __noinline__ void tail(unsigned to, const uint8_t* from) const {
    for (int i = 0; i < 4; i++) {
      uint32_t w = 0;
      for (int k = 0; k < 4; k++)
        if (from + 4 * i + k < stop) w |= uint32_t(from[4 * i + k]) << (8 * k);
      asm volatile("st.shared.u32 [%0], %1;\n" ::"r"(to + 4 * kThreads * i), "r"(w) : "memory");
      if (i == 0 && (asked & (kRing - 1)) == 0)
        asm volatile("st.shared.u32 [%0], %1;\n" ::"r"(to + 4 * kThreads * kRing), "r"(w) : "memory");
    }
  }
  // The 32 bits from bit pos on
  __device__ __forceinline__ uint32_t peek(uint32_t pos) const {
    // word pos / 32 at its row: (pos & 32 (kRing - 1)) / 32 rows of 4 kThreads bytes
    const unsigned at = column + (pos & (32 * (kRing - 1))) * (4 * kThreads / 32);
    uint32_t a, b;
    asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(a) : "r"(at) : "memory");
    asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(b) : "r"(at + 4 * kThreads) : "memory");
    return __funnelshift_l(__byte_perm(b, 0, 0x0123), __byte_perm(a, 0, 0x0123), pos);
  }
};

// A lane's nodes byte by byte, for streams whose states no coder left
// (damaged, or not this coder's): any number of bytes per symbol, none past
// the lane's end.  Returns whether the lane ends as it should.
__device__ bool decode_careful(const unsigned char* D, const uint8_t* p, const uint8_t* end, int k0, int k1, int turn, bool wide,
                               uint32_t* cur, uint32_t* prev, uint64_t* out) {
  uint32_t x = 0;
  for (int j = 0; j < 4 && p < end; j++) x = (x << 8) | *p++;
  for (int k = k0; k < k1; k++) {
    for (int w = 0; w < 16; w++) {
      const uint32_t a2 = w & 3 ? cur[kThreads * (w - 1)] : ~0u, a3 = w >= 4 ? cur[kThreads * (w - 4)] : ~0u;
      const uint32_t ap = k > k0 ? prev[kThreads * w] : ~0u;
      uint32_t s = 0;   // the word's symbols decoded so far
      for (int i = 0; i < 16; i++) {
        const uint32_t a0 = s << 2 | kNoAxis0, a1 = s << 8 | kNoAxis1;
        const uint32_t c = (a2 >> (2 * i) & 3) << 8 | (a3 >> (2 * i) & 3) << 6 | (ap >> (2 * i) & 3) << 4 |
                           (a1 >> (2 * i) & 3) << 2 | (a0 >> (2 * i) & 3);
        uint32_t v4;
        x = next_symbol(D, 4 * c, x, v4);
        while (x < kLow && p < end) x = (x << 8) | *p++;
        s |= v4 >> 2 << (2 * i);
      }
      cur[kThreads * w] = s;
    }
    unpack_node(cur, turn, wide, out + 8 * int64_t(k));
    uint32_t* t = cur; cur = prev; prev = t;
  }
  return p == end && x == kLow;
}

__global__ void __launch_bounds__(kThreads)
store_decode_kernel(const uint8_t* __restrict__ in, const int64_t* __restrict__ in_offsets,
                    const int64_t* __restrict__ in_sizes, const int32_t* __restrict__ count,
                    const int64_t* __restrict__ dst, int nblocks, int turn, const uint16_t* __restrict__ freq,
                    uint64_t* __restrict__ nodes, int64_t* __restrict__ status, int* __restrict__ next) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint32_t* D = reinterpret_cast<uint32_t*>(smem);
  uint32_t* buf = D + kDecTable + threadIdx.x;
  decoder_table(freq, D);
  __syncthreads();
  const int lane = threadIdx.x % 32;
  const bool wide = (reinterpret_cast<uintptr_t>(nodes) & 15) == 0;
  for (int b; (b = next_block(next, count, nblocks)) >= 0;) {
    const int n = count[b], m = lane_nodes(n);
    const int k0 = lane * m, k1 = min(n, k0 + m);
    const uint8_t* sbase = in + in_offsets[b];
    const int64_t size = in_sizes[b];
    uint64_t* o = nodes + 8 * dst[b];
    if (size >= kHead && (sbase[0] & sbase[1] & sbase[2] & sbase[3]) == 0xff) {
      // a block stored raw
      const int64_t words = 8 * int64_t(n);
      const int ok = size == kHead + 8 * words;
      const uint8_t* src = sbase + kHead;
      if (ok && !(reinterpret_cast<uintptr_t>(src) & 7)) {
        for (int64_t i = lane; i < words; i += kLanesS) o[i] = reinterpret_cast<const uint64_t*>(src)[i];
      } else if (ok) {
        for (int64_t i = lane; i < words; i += kLanesS) {
          uint64_t v = 0;
          for (int j = 0; j < 8; j++) v |= uint64_t(src[8 * i + j]) << (8 * j);
          o[i] = v;
        }
      }
      if (lane == 0) status[b] = ok ? n : PG_ERR_FORMAT;
      continue;
    }
    // this lane's length, the lengths before it (exclusive scan) and the sum
    uint32_t len = 0;
    if (size >= kHead)
      for (int j = 0; j < 4; j++) len |= uint32_t(sbase[4 * lane + j]) << (8 * j);
    uint64_t incl = len;
#pragma unroll
    for (int q = 1; q < kLanesS; q <<= 1) {
      const uint64_t u = __shfl_up_sync(0xffffffffu, incl, q);
      if (lane >= q) incl += u;
    }
    if (size < kHead || __shfl_sync(0xffffffffu, incl, kLanesS - 1) != uint64_t(size - kHead)) {
      if (lane == 0) status[b] = PG_ERR_FORMAT;
      continue;
    }
    const uint8_t* p = sbase + kHead + (incl - len);
    uint32_t* cur = buf;
    uint32_t* prev = buf + 16 * kThreads;
    uint32_t x = 0;
    for (int j = 0; j < int(min(len, 4u)); j++) x = (x << 8) | p[j];
    // A coder leaves every lane a state of 2^23 .. 2^31, and the bit counts
    // below are 32-bit: anything else is decoded with care.
    if (__any_sync(0xffffffffu, x < kLow || len < 4 || len > (1u << 28))) {
      const bool ok = decode_careful(smem, p, p + len, k0, k1, turn, wide, cur, prev, o);
      const bool all = __all_sync(0xffffffffu, ok);
      if (lane == 0) status[b] = all ? n : PG_ERR_FORMAT;
      continue;
    }
    const uint32_t skip = uint32_t(reinterpret_cast<uintptr_t>(p) & 3);
    lane_ring R = {p - skip, unsigned(__cvta_generic_to_shared(buf + 32 * kThreads)), 0, int((skip + len + 3) / 4),
                   int(min(int64_t(1) << 30, (sbase + size - (p - skip)) / 4)), sbase + size};
    uint32_t pos = 8 * (skip + 4);   // the next bit of the lane
#pragma unroll
    for (int i = 0; i < kRing / 4; i++) R.top_up(pos);
    for (int k = k0; k < k1; k++) {
      const bool has_prev = k > k0;
#pragma unroll 1
      for (int w = 0; w < 16; w++) {
        const uint32_t a2 = w & 3 ? cur[kThreads * (w - 1)] : ~0u, a3 = w >= 4 ? cur[kThreads * (w - 4)] : ~0u;
        const uint32_t ap = has_prev ? prev[kThreads * w] : ~0u;
        // a2 a3 ap of rotations 4 j + c in byte j of known[c]
        const uint32_t e = even_pairs(a2, a3), d = odd_pairs(a2, a3);
        const uint32_t known[4] = {(e << 2 & 0x3c3c3c3cu) | (ap & 0x03030303u),
                                   (d << 2 & 0x3c3c3c3cu) | (ap >> 2 & 0x03030303u),
                                   (e >> 2 & 0x3c3c3c3cu) | (ap >> 4 & 0x03030303u),
                                   (d >> 2 & 0x3c3c3c3cu) | (ap >> 6 & 0x03030303u)};
        uint32_t v[16], s = 0;
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
          if (i % 8 == 0) {
            R.top_up(pos);
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
          }
          uint32_t A = R.peek(pos);
#pragma unroll
          for (int j = i; j < i + 2; j++) {
            // 4 c = 64 (a2 a3 ap) + 16 a1 + 4 a0, with 4 times the symbols kept in v
            const uint32_t c4 = __byte_perm(known[j & 3], 0, 0x4440 + (j >> 2)) * 64 + (j >= 4 ? v[j >= 4 ? j - 4 : 0] : 12) * 4 +
                                (j & 3 ? v[j & 3 ? j - 1 : 0] : 12);
            const uint32_t y = next_symbol(smem, c4, x, v[j]);
            const uint32_t nb = select_ge(y, kLow >> 8, select_ge(y, kLow, 0u, 8u), 16u);
            x = __funnelshift_l(A, y, nb);
            A = A << nb;
            pos += nb;
            s += j ? v[j] << (j ? 2 * j - 2 : 0) : v[j] >> 2;
          }
        }
        cur[kThreads * w] = s;
      }
      unpack_node(cur, turn, wide, o + 8 * int64_t(k));
      uint32_t* t = cur; cur = prev; prev = t;
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    const bool bad = __any_sync(0xffffffffu, pos != 8 * (skip + len) || x != kLow);
    if (lane == 0) status[b] = bad ? PG_ERR_FORMAT : n;
  }
}

// CTAs of the coder kernels: one per SM, no more than there are blocks.
int coder_grid(int nblocks) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return nblocks < sms ? nblocks : sms;
}

int coder_smem() {
  return cudaFuncSetAttribute(store_hist_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kHistSmem)) ==
                     cudaSuccess &&
                 cudaFuncSetAttribute(store_encode_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kEncSmem)) ==
                     cudaSuccess &&
                 cudaFuncSetAttribute(store_decode_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kDecSmem)) ==
                     cudaSuccess
             ? PG_OK
             : PG_ERR_CUDA;
}
int prepare_coder() {
  const int rc = per_device_once((const void*)&coder_smem, coder_smem);
  return rc ? fail(rc, "cudaFuncSetAttribute failed") : PG_OK;
}

// A zeroed counter for next_block.
int block_counter(stream_scratch& scratch, int** next) {
  PG_CUDA(scratch.alloc(next, sizeof(int)));
  PG_CUDA(cudaMemsetAsync(*next, 0, sizeof(int), scratch.stream));
  return PG_OK;
}

}  // namespace
}  // namespace pg

using namespace pg;

extern "C" int64_t pg_store_bound(int64_t nodes) {
  if (nodes < 0 || nodes > 8 * 8 * 8 * 8 * 64) return fail(PG_ERR_ARG, "bad node count");
  return store_bound(int(nodes));
}

extern "C" int pg_store_table(const uint64_t* nodes, const int64_t* first, const int32_t* count, int nblocks, int turn,
                              uint16_t* table, void* stream_) {
  if (nblocks < 0 || !table || (nblocks && (!nodes || !first || !count))) return fail(PG_ERR_ARG, "bad store arguments");
  cudaStream_t stream = (cudaStream_t)stream_;
  stream_scratch scratch(stream);
  unsigned* hist = nullptr;
  PG_CUDA(scratch.alloc(&hist, sizeof(unsigned) * kCtx * 3));
  PG_CUDA(cudaMemsetAsync(hist, 0, sizeof(unsigned) * kCtx * 3, stream));
  if (nblocks) {
    const int stride = (nblocks + kTableBlocks - 1) / kTableBlocks;
    if (int rc = prepare_coder()) return rc;
    store_hist_kernel<<<coder_grid((nblocks + stride - 1) / stride), kThreads, kHistSmem, stream>>>(
        nodes, first, count, nblocks, stride, turn & 1, hist);
    PG_CUDA(cudaGetLastError());
  }
  store_table_kernel<<<kCtx / 256, 256, 0, stream>>>(hist, table);
  PG_CUDA(cudaGetLastError());
  return PG_OK;
}

extern "C" int pg_store_encode(const uint64_t* nodes, const int64_t* first, const int32_t* count, int nblocks, int turn,
                               const uint16_t* table, uint8_t* out, const int64_t* out_offsets, int64_t* sizes,
                               void* stream) {
  if (nblocks < 0 || (nblocks && (!nodes || !first || !count || !table || !out || !out_offsets || !sizes)))
    return fail(PG_ERR_ARG, "bad store arguments");
  if (!nblocks) return PG_OK;
  if (int rc = prepare_coder()) return rc;
  stream_scratch scratch((cudaStream_t)stream);
  int* next = nullptr;
  if (int rc = block_counter(scratch, &next)) return rc;
  store_encode_kernel<<<coder_grid(nblocks), kThreads, kEncSmem, (cudaStream_t)stream>>>(
      nodes, first, count, nblocks, turn & 1, table, out, out_offsets, sizes, next);
  PG_CUDA(cudaGetLastError());
  return PG_OK;
}

extern "C" int pg_store_decode(const uint8_t* in, const int64_t* in_offsets, const int64_t* in_sizes,
                               const int32_t* count, const int64_t* dst, int nblocks, int turn, const uint16_t* table,
                               uint64_t* nodes, int64_t* status, void* stream) {
  if (nblocks < 0 || (nblocks && (!in || !in_offsets || !in_sizes || !count || !dst || !table || !nodes || !status)))
    return fail(PG_ERR_ARG, "bad store arguments");
  if (!nblocks) return PG_OK;
  if (int rc = prepare_coder()) return rc;
  stream_scratch scratch((cudaStream_t)stream);
  int* next = nullptr;
  if (int rc = block_counter(scratch, &next)) return rc;
  store_decode_kernel<<<coder_grid(nblocks), kThreads, kDecSmem, (cudaStream_t)stream>>>(
      in, in_offsets, in_sizes, count, dst, nblocks, turn & 1, table, nodes, status, next);
  PG_CUDA(cudaGetLastError());
  return PG_OK;
}
