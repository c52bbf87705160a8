// The midsolve solve of one board, shared by the batch kernel (mid.cu) and
// the server kernel (serve.cu).  See mid.cu for the algorithm.
#pragma once
#include "superscore.cuh"
#include "tables.h"
#include "runtime.h"
#include "../../include/pentago_b200.h"
#include <cstring>
#include <string>

namespace pg {

// Tables the midsolve code reads: combinations[n][k] for n, k <= 18 (0 for k > n;
// mid/subsets.h:17-21), the 32 five-in-a-row masks, and the win factors.  The
// combinations are looked up with indexes that differ from thread to thread,
// so on the device they are in shared memory, not in constant memory.
using mid_choose = uint16_t[20];
struct mid_tables {
  const mid_choose* choose;
  const uint64_t* winpat;
  const uint32_t* wf;
};

PG_HD int choose_t(const mid_choose* C, int n, int k) { return C[n][k]; }

struct mid_grab { int ny, lo, size; };

struct mid_job_t {
  uint64_t side[2];
  uint32_t ply;
  int32_t spots;
  uint8_t empty[18];
  uint8_t pad[6];
  int32_t sets1p_off[20], wins1_off[20], cs1ps_off[20];
  mid_grab spaces[20];
  uint64_t* sets1p;       // global scratch
  uint4* wins1;           // 2 per entry: after, before
  uint16_t* cs1ps;
  uint4* workspace;       // global workspace, or null when it lives in shared memory
  pg_mid_values_t* out;
  int32_t ws_size;        // workspace entries, for bounds checks
  int32_t pad2;
};

static_assert(sizeof(mid_job_t) % 16 == 0, "mid_job_t is copied in 16-byte words");

// make_set0_info (mid/internal.h:174-259) of one s0 row, in a tile of rows in
// shared memory: the side's wins, then for the q-th free spot and the i-th of
// s1p's stones standing on it a word (C(spot, i + 1) << 16) + offset0[i][q] at
// q k1 + i, whose sum over the stones is s1 << 16 | s0p (the offsets are
// signed, both sums lie in 0..65535), then per free spot where the child's
// row starts in the level below, child_s0s[q] in_ny.  A tile is no larger than
// a chunk's rows need: what shared memory leaves of the SM's 228 KB is L1, which
// holds the gathers in flight (18 stones: 7.0 ms with three CTAs of 64 KB per
// SM, 6.0 with four of 24 KB).
constexpr int kTileBytes = 24 << 10;
PG_HD int row_bytes(int k1, int free_spots) {
  return int(sizeof(uint4)) + ((4 * free_spots * (k1 + 1) + 15) & ~15);
}

// ---------------------------------------------------------------------------
// Subset ranking (mid/subsets.h:34-105)
// ---------------------------------------------------------------------------

// The index-th k-subset of [0,n) in large-entry-major order, as a mask: from
// the top, an element is in it when the rank left covers the subsets without
// it (at k = 0 the rank is 0 and covers none).
PG_HD uint32_t unrank(const mid_choose* C, int n, int k, int index) {
  uint32_t set = 0;
  for (int j = n - 1; j >= 0; j--) {
    const int c = choose_t(C, j, k), yes = index >= c;
    index -= yes ? c : 0;
    set |= uint32_t(yes) << j;
    k -= yes;
  }
  return set;
}

PG_HD uint64_t set_side(const uint8_t* empty, int spots, uint32_t set) {
  uint64_t s = 0;
  for (int i = 0; i < spots; i++) s |= uint64_t(set >> i & 1) << empty[i];
  return s;
}

PG_HD int popc32(uint32_t x) {
#ifdef __CUDA_ARCH__
  return __popc(x);
#else
  return __builtin_popcount(x);
#endif
}

// ---------------------------------------------------------------------------
// Wins of one side: super_wins split by parity (halfsuper_wins, generated by
// pentago/base/precompute.cc:330-505; here computed from the full super).
// ---------------------------------------------------------------------------

PG_HD half4 h_wins(const uint32_t* wf, uint64_t side, int parity) {
  return s_split(s_super_wins(wf, side), parity);
}

PG_HD bool won(const uint64_t* pats, uint64_t side) {
  for (int i = 0; i < 32; i++)
    if ((side & pats[i]) == pats[i]) return true;
  return false;
}

// ---------------------------------------------------------------------------
// The per-board CTA kernel
// ---------------------------------------------------------------------------

constexpr int kMidThreads = 256;
// Items of a chunk, about, when a board's groups take several each: an
// 18-stone board takes 9.0 ms with chunks of 16,384, 7.0 with 4,096, 8.0 with
// 1,024 (the smaller ones share more of the level below in L2, until building
// their rows costs more than that saves).
constexpr int kChunkItems = 3072;
constexpr int kSmemWorkspaceMax = 8400;  // bottleneck(10), in halfsupers

struct level_t {
  int n, k0, k1, spots, parity;
  uint64_t root0, root1;
  int nsets0, nsets1p, nsets1;
};

PG_HD level_t make_level(const mid_job_t& J, const mid_tables& MT, int n) {
  level_t L;
  L.n = n;
  L.k0 = n >> 1;
  L.k1 = n - L.k0;
  L.spots = J.spots;
  L.parity = int((n + J.ply) & 1);
  L.root0 = J.side[(J.spots + n) & 1];
  L.root1 = J.side[(J.spots + n + 1) & 1];
  L.nsets0 = choose_t(MT.choose, J.spots, L.k0);
  L.nsets1p = choose_t(MT.choose, J.spots - L.k0, L.k1);
  L.nsets1 = choose_t(MT.choose, J.spots, L.k1);
  return L;
}

// x = k n + i with 0 <= i < n, with m = floor((2^32 - 1) / n): the high
// product gives k exactly or one short.
PG_HD void split_index(uint32_t x, uint32_t n, uint32_t m, int& k, int& i) {
#ifdef __CUDA_ARCH__
  uint32_t q = __umulhi(x, m);
#else
  uint32_t q = uint32_t((uint64_t(x) * m) >> 32);
#endif
  uint32_t r = x - q * n;
  if (r >= n) { r -= n; q++; }
  k = int(q);
  i = int(r);
}

// What the rows and items of a level need, worked out once.
struct level_src {
  const uint64_t* sets1p;
  const uint16_t* cs1ps;
  const uint4* wins1;
  const uint4* in;
  uint4* out;
  int in_ny, out_ny;
  unsigned in_size, out_size;   // entries in and out may touch
  uint4* results;               // of levels 0 and 1
  int turn_aggressive;
};

// Part i of row s0's data: for i < k1 the words of s1p's i-th stone, for
// i = k1 the children's rows and the side's wins.  (No branch on the subset:
// the threads of a warp have different ones.)
PG_HD void row_part(const mid_job_t& J, const mid_tables& MT, const level_t& L, int in_ny, int s0, int i, uint4* row) {
  const int k0 = L.k0, k1 = L.k1, free_spots = J.spots - k0;
  const uint32_t taken = unrank(MT.choose, J.spots, k0, s0);
  uint32_t* words = reinterpret_cast<uint32_t*>(row + 1);
  if (i < k1) {
    // make_offset0: minus C(v - i - 1, a) for every stone a at v above the spot (and above i)
    int offset = i ? 0 : s0;
#ifdef __CUDA_ARCH__
#pragma unroll 5
#endif
    for (int spot = J.spots - 1; spot >= 0; spot--) {
      const int stone = taken >> spot & 1, below = popc32(taken & ((1u << spot) - 1));   // set0's stones below the spot
      const uint32_t word = (uint32_t(choose_t(MT.choose, spot, i + 1)) << 16) + uint32_t(offset);
      if (!stone) words[(spot - below) * k1 + i] = word;
      offset -= stone && spot > i ? choose_t(MT.choose, spot > i ? spot - i - 1 : 0, below) : 0;
    }
  } else {
    // make_child_s0s: the rank of the subset with the spot added, whose stones
    // above it count one place higher
    uint32_t* child = words + free_spots * k1;
    int rank = s0;
#ifdef __CUDA_ARCH__
#pragma unroll 5
#endif
    for (int spot = J.spots - 1; spot >= 0; spot--) {
      const int stone = taken >> spot & 1, below = popc32(taken & ((1u << spot) - 1));
      const int low = choose_t(MT.choose, spot, below + 1), high = choose_t(MT.choose, spot, below + 2);
      if (!stone) child[spot - below] = uint32_t((rank + low) * in_ny);
      rank += stone ? high - low : 0;
    }
    // A side's stones at level n are those of the other side at level n - 1
    // (the roots alternate, and k0(n) = k1(n - 1)), so its wins are already in
    // that level's wins1, in the parity stored second.
    *row = L.n ? J.wins1[2 * (J.wins1_off[L.n - 1] + s0) + 1] : h_to(h_wins(MT.wf, L.root0, L.parity));
  }
}

// inner (mid/internal.h:358-408) of item (row, s1p), K1 stones in s1p.
// Returns false (and writes nothing) if an index would leave the workspace.
template<int K1>
PG_HD bool inner(const level_t& L, const level_src& S, const uint4* row, int s1p, uint64_t set1p) {
  const int n = L.n, spots = L.spots, free_spots = spots - L.k0;
  const uint32_t* words = reinterpret_cast<const uint32_t*>(row + 1);
  uint32_t at = 0;
#pragma unroll
  for (int i = 0; i < K1; i++) at += words[int(set1p >> (5 * i) & 0x1f) * K1 + i];
  const int s1 = int(at >> 16), s0p = int(at & 0xffff);
  const unsigned o = unsigned(s1) * unsigned(S.out_ny) + unsigned(s0p);
  if (o >= S.out_size || s1 >= L.nsets1 || (n <= 1 && n + s1p >= 19)) return false;
  const uint4* w1 = S.wins1 + 2 * s1;
  const half4 after = h_from(w1[0]), before = h_from(w1[1]);
  // The children: a move to each free spot that is not s1p's.
  half4 us = (spots == n && !S.turn_aggressive) ? h_not(h_zero()) : h_zero();
  const uint32_t* child = words + free_spots * K1;
  const uint16_t* cs = S.cs1ps + s1p;
  uint32_t open = ~uint32_t(set1p >> 45) & ((1u << free_spots) - 1);
  unsigned worst = 0;
#ifdef __CUDA_ARCH__
  open = __brev(open);
#pragma unroll 4
#endif
  for (int m = spots - n; m > 0; m--) {
#ifdef __CUDA_ARCH__
    const unsigned i = unsigned(__clz(open));
    open ^= 0x80000000u >> i;
#else
    const unsigned i = unsigned(ctz32(open));
    open &= open - 1;
#endif
    const unsigned idx = child[i] + cs[i * unsigned(L.nsets1p)];
    worst = worst > idx ? worst : idx;
    us = h_or(us, h_from(S.in[idx < S.in_size ? idx : S.in_size - 1]));
  }
  if (spots > n && worst >= S.in_size) return false;
  const half4 wins0 = h_from(*row);
  const half4 inplay = h_not(h_or(wins0, after));
  const half4 mask = S.turn_aggressive ? h_not(after) : h_not(h_zero());
  us = h_or(h_and(inplay, us), h_and(wins0, mask));
  if (n <= 1) S.results[n + s1p] = h_to(us);
  S.out[o] = h_to(h_or(h_rmax(h_not(us)), before));
  return true;
}

// Items [a, b) of a tile (item 0 is the tile's first), by the group's threads.
template<int K1>
PG_HD bool tile_items(const level_t& L, const level_src& S, const char* tile, int stride, int a, int b, int tid, int nt) {
  bool ok = true;
  const int ns = L.nsets1p, row_step = nt / ns, s1p_step = nt - row_step * ns;
  int row = (a + tid) / ns, s1p = a + tid - row * ns;
  uint64_t next = a + tid < b ? S.sets1p[s1p] : 0;
  for (int it = a + tid; it < b; it += nt) {
    const uint64_t set1p = next;
    const int row_now = row, s1p_now = s1p;
    row += row_step;
    s1p += s1p_step;
    if (s1p >= ns) { s1p -= ns; row++; }
    next = S.sets1p[s1p];   // (some s1p of the level, also after the last item)
    ok &= inner<K1>(L, S, reinterpret_cast<const uint4*>(tile + row_now * stride), s1p_now, set1p);
  }
  return ok;
}

// high_board_t helpers for the traversal (high/board.cc)

// A quadrant side's 9 bits as base-3 digits, three at a time.
PG_HD uint32_t pack9(uint32_t v) {
  const uint64_t three = 0x0d0c0a0904030100ull;
  return (uint32_t(three >> (8 * (v & 7))) & 0xff) + 27 * (uint32_t(three >> (8 * (v >> 3 & 7))) & 0xff) +
         729 * (uint32_t(three >> (8 * (v >> 6 & 7))) & 0xff);
}
PG_HD uint64_t board_of(uint64_t s0, uint64_t s1) {
  uint64_t board = 0;
  for (int q = 0; q < 4; q++) {
    const uint32_t a = uint32_t(s0 >> (16 * q)) & 0x1ff, b = uint32_t(s1 >> (16 * q)) & 0x1ff;
    board |= uint64_t(pack9(a) + 2 * pack9(b)) << (16 * q);
  }
  return board;
}

// A quadrant side rotated one step (d = 1 left, -1 right).
PG_HD uint32_t rotate9(uint32_t v, int d) {
  uint32_t r = 0;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
  for (int i = 0; i < 9; i++) r |= (v >> i & 1) << (4 - d * (3 * (i % 3) - i / 3 - 2));
  return r;
}
// The board with quadrant q of both sides rotated, from the board as it is.
PG_HD uint64_t rotated_board(uint64_t board, const uint64_t* side, int q, int d) {
  const uint32_t a = uint32_t(side[0] >> (16 * q)) & 0x1ff, b = uint32_t(side[1] >> (16 * q)) & 0x1ff;
  return (board & ~(uint64_t(0xffff) << (16 * q))) |
         uint64_t(pack9(rotate9(a, d)) + 2 * pack9(rotate9(b, d))) << (16 * q);
}

// done_and_value (high/board.cc:20-29)
PG_HD bool done_value(const mid_tables& MT, const uint64_t* side, uint32_t ply, int* value) {
  const bool bw = won(MT.winpat, side[0]), ww = won(MT.winpat, side[1]);
  const int turn = int(ply >> 1 & 1);
  if (bw || ww) { *value = (bw && ww) ? 0 : (bw == !turn ? 1 : -1); return true; }
  if (ply == 72) { *value = 0; return true; }
  return false;
}

PG_HD int hbit(const uint4& h, int i) {
  const uint32_t w = i < 32 ? h.x : i < 64 ? h.y : i < 96 ? h.z : h.w;
  return int(w >> (i & 31) & 1);
}

PG_HD void append(pg_mid_values_t* out, uint64_t raw, int v) {
  const int k = out->size++;
  if (k < 163) { out->entries[k].raw = raw; out->entries[k].value = v; out->entries[k].pad = 0; }
}

// midsolve_traverse (midengine.cc:127-158), iteratively; supers[i] = (win, notlose)
PG_HD void traverse(const mid_job_t& J, const mid_tables& MT, const uint4* supers, pg_mid_values_t* out) {
  out->size = 0;
  out->pad = 0;
  uint64_t side[2] = {J.side[0], J.side[1]};
  const uint32_t ply = J.ply;
  auto middle_children = [&](const uint64_t* sd, uint32_t p, const uint4* r) {
    int best = -1;
    const uint64_t board = board_of(sd[0], sd[1]);
    for (int s = 0; s < 8; s++) {
      const int q = s >> 1, d = (s & 1) ? -1 : 1;
      const int idx = ((d & 3) << (2 * q)) >> 1;
      const int v = hbit(r[0], idx) + hbit(r[1], idx) - 1;
      append(out, rotated_board(board, sd, q, d) | uint64_t((p + 1) & 1) << 63, v);
      best = best > -v ? best : -v;
    }
    return best;
  };
  int value;
  if (done_value(MT, side, ply, &value)) {
  } else if (!(ply & 1)) {
    value = -1;
    const uint64_t empty = 0x01ff01ff01ff01ffull ^ side[0] ^ side[1];
    int s = 0;
    for (int bit = 0; bit < 64; bit++) {
      if (!(empty >> bit & 1)) continue;
      s++;
      uint64_t cs[2] = {side[0], side[1]};
      cs[(ply >> 1) & 1] |= uint64_t(1) << bit;
      const uint32_t cply = ply + 1;
      int cv;
      if (!done_value(MT, cs, cply, &cv)) cv = middle_children(cs, cply, supers + 2 * s);
      append(out, board_of(cs[0], cs[1]) | uint64_t(1) << 63, cv);
      value = value > cv ? value : cv;
    }
  } else {
    value = middle_children(side, ply, supers);
  }
  append(out, board_of(side[0], side[1]) | uint64_t(ply & 1) << 63, value);
}

#ifdef __CUDA_ARCH__
// traverse on the device, by one warp or several (each works the layout out
// for itself, and they share the records): lane p holds the p-th five-in-a-row
// mask, so whether a side has won is a vote, and the cells that would complete
// a five are one reduction; lane s holds the root's s-th child, whose records
// start 9 places on per child before it, 8 fewer for each that is done.
__device__ __forceinline__ void put_record(pg_mid_values_t* out, int k, uint64_t raw, int v) {
  if (k < 163) { out->entries[k].raw = raw; out->entries[k].value = v; out->entries[k].pad = 0; }
}
// The value of rotation s (quadrant s >> 1, left or right) from its parent's results.
__device__ __forceinline__ int rotation_value(const uint4& r0, const uint4& r1, int s) {
  const int idx = (((s & 1) ? 3 : 1) << (s & 6)) >> 1;
  return hbit(r0, idx) + hbit(r1, idx) - 1;
}
__device__ __forceinline__ uint64_t rotation_board(const uint64_t* side, int s) {
  return rotated_board(board_of(side[0], side[1]), side, s >> 1, (s & 1) ? -1 : 1);
}
// raw: both passes' n <= 1 results, interleaved as (win, notlose) of entry i
// = raw[i == 0], raw[i != 0] at i (midengine.cc:119-124).
__device__ void traverse_warps(const uint64_t* root, uint32_t ply, const uint64_t* winpat, const uint4 (*raw)[19],
                               pg_mid_values_t* out, int warp, int warps, int lane) {
  const unsigned full = 0xffffffffu;
  const uint64_t side[2] = {root[0], root[1]};
  const int turn = int(ply >> 1 & 1);
  const uint64_t pattern = winpat[lane];
  const bool bw = __any_sync(full, (side[0] & pattern) == pattern), ww = __any_sync(full, (side[1] & pattern) == pattern);
  int value, total = 0;
  if (bw || ww || ply == 72) {   // done_value
    value = bw == ww ? 0 : bw == !turn ? 1 : -1;
  } else if (!(ply & 1)) {
    // The children: a stone of the side to move on each empty cell (at most 18)
    const uint64_t empty = 0x01ff01ff01ff01ffull ^ side[0] ^ side[1], missing = pattern & ~side[turn];
    const bool one = (missing & (missing - 1)) == 0;
    const uint64_t fives = uint64_t(__reduce_or_sync(full, one ? uint32_t(missing >> 32) : 0u)) << 32 |
                           __reduce_or_sync(full, one ? uint32_t(missing) : 0u);
    const int nempty = __popcll(empty);
    uint64_t e = empty;
    for (int i = 0; i < lane; i++) e &= e - 1;
    const uint64_t stone = e & (~e + 1);   // (0 beyond the last child)
    const bool wins = (stone & fives) != 0;
    const unsigned won = __ballot_sync(full, wins);
    total = 9 * nempty - 8 * __popc(won);
    int cv = -1;
    if (wins) cv = 1;
    else if (lane < nempty) {
      const uint4 r0 = raw[0][lane + 1], r1 = raw[1][lane + 1];
#pragma unroll
      for (int s = 0; s < 8; s++) cv = max(cv, -rotation_value(r0, r1, s));
    }
    value = __reduce_max_sync(full, cv);
    for (int c0 = 4 * warp; c0 < nempty; c0 += 4 * warps) {   // four children's rotations at once
      const int c = c0 + (lane >> 3), s = lane & 7;
      const uint64_t cstone = __shfl_sync(full, stone, c & 31);
      const int ccv = __shfl_sync(full, cv, c & 31);
      if (c >= nempty) continue;
      uint64_t cs[2] = {side[0], side[1]};
      cs[turn] |= cstone;
      const int at = 9 * c - 8 * __popc(won & ((1u << c) - 1));
      const bool done = won >> c & 1;
      if (!done) put_record(out, at + s, rotation_board(cs, s), rotation_value(raw[0][c + 1], raw[1][c + 1], s));
      if (s == 0) put_record(out, at + (done ? 0 : 8), board_of(cs[0], cs[1]) | uint64_t(1) << 63, ccv);
    }
  } else {
    // lanes 0..7: the root's 8 rotation children
    const int v = rotation_value(raw[1][0], raw[0][0], lane & 7);
    if (warp == 0 && lane < 8) put_record(out, lane, rotation_board(side, lane), v);
    value = __reduce_max_sync(full, -v);
    total = 8;
  }
  if (warp == 0 && lane == 0) {
    put_record(out, total, board_of(side[0], side[1]) | uint64_t(ply & 1) << 63, value);
    out->size = total + 1;
    out->pad = 0;
  }
}
#endif

// The whole solve of one board by ncta groups of nt cooperating threads
// (thread tid of group cta).  `barrier` synchronizes one group, `gbarrier`
// all groups (with one group it is the same barrier).  Inside a level the
// (s0, s1p) items are split into contiguous chunks dealt out to the groups in
// turn, and each group builds the rows of its own chunks; a level's output is
// read by the next level only after the all-group barrier.  Run with one group
// of one thread and no-op barriers it is the same computation done sequentially
// (used by the CPU self-test).  `raw` and `fault` are shared by the groups;
// `tile` has room for tile_bytes of s0 rows.
//
// Bound by the instructions of a level's items and, on small boards, by the
// chain of levels, so what an item needs is laid out beforehand: the stones of
// its s1p (5 bits each, and as a mask above them) in one word, the two sums
// over them in one table word per stone, the children's columns side by side
// for neighbouring s1p, and a row's table built by one thread per entry.  A
// board of 18 stones on all SMs: 5.8 ms (12.0 with the indexes worked out from
// each item's subsets); 64 boards of 26 stones, a CTA each: 0.25 ms with what the
// call costs (0.51).
template<class Barrier, class GridBarrier>
PG_HD void mid_board_body(const mid_job_t& J, const mid_tables& MT, char* tile, uint4* ws,
                          uint4 (*raw)[19], int* fault, int tid, int nt, int cta, int ncta, Barrier barrier,
                          GridBarrier gbarrier, uint4* dump = nullptr, int tile_bytes = kTileBytes) {
  const int spots = J.spots;
  const int gtid = cta * nt + tid, gnt = ncta * nt;
  // Per-level tables, the same for both passes (midengine.cc:57-76, :101-107),
  // over all levels at once: entry x of a table belongs to the level whose
  // offsets enclose it.
  auto level_of = [&](const int32_t* off, int x) {
    int n = 0;
    while (x >= off[n + 1]) n++;
    return n;
  };
  for (int x = gtid; x < J.wins1_off[spots + 1]; x += gnt) {
    const int n = level_of(J.wins1_off, x), k1 = n - (n >> 1);
    const int parity = int((n + J.ply) & 1);
    const uint64_t root1 = J.side[(spots + n + 1) & 1];
    const uint64_t side1 = root1 | set_side(J.empty, spots, unrank(MT.choose, spots, k1, x - J.wins1_off[n]));
    const super8 w = s_super_wins(MT.wf, side1);
    J.wins1[2 * x] = h_to(s_split(w, parity));
    J.wins1[2 * x + 1] = h_to(s_split(w, !parity));
  }
  for (int x = gtid; x < J.sets1p_off[spots + 1]; x += gnt) {
    const int n = level_of(J.sets1p_off, x), k0 = n >> 1, k1 = n - k0;
    const uint32_t mask = unrank(MT.choose, spots - k0, k1, x - J.sets1p_off[n]);
    uint64_t set = uint64_t(mask) << 45;   // above at most 9 stones of 5 bits
    uint32_t left = mask;
    for (int a = 0; a < k1; a++, left &= left - 1) set |= uint64_t(ctz32(left)) << (5 * a);
    J.sets1p[x] = set;
  }
  gbarrier();
  for (int x = gtid; x < J.cs1ps_off[spots + 1]; x += gnt) {  // make_cs1ps (mid/internal.h:135-150)
    const int n = level_of(J.cs1ps_off, x), k0 = n >> 1, k1 = n - k0;
    const int ns1p = choose_t(MT.choose, spots - k0, k1);
    const int idx = x - J.cs1ps_off[n], j = idx / ns1p, s1p = idx - j * ns1p;   // [spot][s1p]
    const uint64_t set = J.sets1p[J.sets1p_off[n] + s1p];
    int c = s1p;
    for (int a = 0; a < k1; a++) {
      const int v = int(set >> (5 * a) & 0x1f);
      if (j < v) c -= choose_t(MT.choose, v - 1, a);
    }
    J.cs1ps[x] = uint16_t(c);
  }
  gbarrier();

  for (int aggressive = 0; aggressive < 2; aggressive++) {
    for (int n = spots; n >= 0; n--) {
      const level_t L = make_level(J, MT, n);
      const mid_grab gi = J.spaces[n + 1], go = J.spaces[n];
      const level_src S = {J.sets1p + J.sets1p_off[n], J.cs1ps + J.cs1ps_off[n], J.wins1 + 2 * J.wins1_off[n],
                           ws + gi.lo, ws + go.lo, gi.ny, go.ny, unsigned(J.ws_size - gi.lo),
                           unsigned(J.ws_size - go.lo), raw[aggressive], aggressive ^ (n & 1)};
      const int stride = row_bytes(L.k1, spots - L.k0), most = tile_bytes / stride;
      const uint32_t m_parts = 0xffffffffu / uint32_t(L.k1 + 1);
      // A group's share: one chunk of the level's items, or several apart from
      // each other, so that the groups work side by side on neighbouring rows
      // and share the rows below them in the cache.
      const int64_t total = int64_t(L.nsets0) * L.nsets1p;
      const int chunks = ncta == 1 ? 1 : ncta * int(total / (int64_t(ncta) * kChunkItems) + 1);
      for (int chunk = cta; chunk < chunks; chunk += ncta) {
        const int64_t i0 = total * chunk / chunks, i1 = total * (chunk + 1) / chunks;
        const int r0 = int(i0 / L.nsets1p), r1 = i1 > i0 ? int((i1 - 1) / L.nsets1p) + 1 : r0;
        for (int base = r0; base < r1; base += most) {
          const int rows = r1 - base < most ? r1 - base : most;
          if (base > r0 || chunk > cta) barrier();
          for (int e = tid; e < rows * (L.k1 + 1); e += nt) {
            int r, i;
            split_index(uint32_t(e), uint32_t(L.k1 + 1), m_parts, r, i);
            row_part(J, MT, L, gi.ny, base + r, i, reinterpret_cast<uint4*>(tile + r * stride));
          }
          barrier();
          const int64_t first = int64_t(base) * L.nsets1p, last = first + int64_t(rows) * L.nsets1p;
          const int a = int((i0 > first ? i0 : first) - first), b = int((i1 < last ? i1 : last) - first);
          bool ok = true;
          switch (L.k1) {
#define PG_CASE(K) case K: ok = tile_items<K>(L, S, tile, stride, a, b, tid, nt); break;
            PG_CASE(0) PG_CASE(1) PG_CASE(2) PG_CASE(3) PG_CASE(4) PG_CASE(5) PG_CASE(6) PG_CASE(7) PG_CASE(8) PG_CASE(9)
#undef PG_CASE
          }
          if (!ok) *fault = 1;
        }
      }
      gbarrier();
    }
  }

  // Interleave (midengine.cc:119-124) and traverse; a failed bounds check
  // marks the record with size -1 instead.
  if (gtid == 0 && *fault) { J.out->size = -1; J.out->pad = 0; }
#ifdef __CUDA_ARCH__
  // the first warp traverses (nt >= 32 on the device)
  if (gtid < 32 && !*fault) traverse_warps(J.side, J.ply, MT.winpat, raw, J.out, 0, 1, gtid);
#else
  if (gtid == 0 && !*fault) {
    uint4 supers[2 * 19];
    for (int i = 0; i < 19; i++)
      for (int j = 0; j < 2; j++) supers[2 * i + j] = raw[j ^ (i == 0)][i];
    if (dump)
      for (int i = 0; i < 38; i++) dump[i] = supers[i];
    traverse(J, MT, supers, J.out);
  }
#endif
}


// Per translation unit: each .cu file that launches the body uploads these.
static __constant__ uint16_t c_choose[19][20];
static __constant__ uint64_t c_winpat[32];
// The combinations' copy in a CTA's shared memory (mid_choose rows).
struct mid_choose_smem { mid_choose row[19]; };
static __device__ __forceinline__ void load_choose(mid_choose_smem& S) {
  for (int i = threadIdx.x; i < 19 * 20; i += blockDim.x) (&S.row[0][0])[i] = (&c_choose[0][0])[i];
}

struct sync_threads { __device__ void operator()() const { __syncthreads(); } };

// Barrier over the CTAs that solve one board together.  They are co-resident
// (a cooperative launch, or workers of the persistent server); the wait is bounded, and a timeout marks the board
// as failed and turns every later barrier of that board into a no-op, so the
// kernel always finishes.
constexpr unsigned kBarrierPolls = 1u << 28;  // about 20 s of 64 ns sleeps

struct board_barrier {
  unsigned* count;  // arrivals in the current generation
  unsigned* gen;    // generation number
  int ncta;
  int* fault;
  unsigned polls = kBarrierPolls;  // wait limit
  __device__ void operator()() const {
    __syncthreads();
    if (threadIdx.x == 0) {
      volatile unsigned* vg = gen;
      volatile int* vf = fault;
      const unsigned g = *vg;
      __threadfence();
      if (atomicAdd(count, 1u) == unsigned(ncta) - 1) {
        atomicExch(count, 0u);
        __threadfence();
        atomicAdd(gen, 1u);
      } else {
        for (unsigned i = 0; *vg == g && !*vf; i++) {
          if (i > polls) { atomicExch(fault, 1); break; }
          __nanosleep(64);
        }
      }
      __threadfence();
    }
    __syncthreads();
  }
};


// ---------------------------------------------------------------------------
// Host helpers (mid.cu)
// ---------------------------------------------------------------------------

struct board_plan {
  mid_job_t job;
  size_t sets1p, wins1, cs1ps, workspace;  // element counts
};

int bottleneck(int spots);
int hchoose(int n, int k);
bool plan_board(uint64_t raw, board_plan& P, std::string& err);
// Device scratch the board needs, and pointing the job's tables into it.  The
// workspace is in global scratch when it does not fit shared memory, or
// always with global_ws.
size_t scratch_bytes_of(const board_plan& P, bool global_ws = false);
void carve_scratch(board_plan& P, char* base, bool global_ws = false);

// Upload this translation unit's constant tables (once per device).
static int mid_upload_constants() {
  uint16_t ch[19][20];
  for (int n = 0; n <= 18; n++)
    for (int k = 0; k < 20; k++) ch[n][k] = uint16_t(hchoose(n, k));
  const tables_t& T = tables();
  if (cudaMemcpyToSymbol(c_choose, ch, sizeof ch) != cudaSuccess ||
      cudaMemcpyToSymbol(c_winpat, T.winpat, sizeof T.winpat) != cudaSuccess)
    return PG_ERR_CUDA;
  return PG_OK;
}
static int mid_prepare_device() { return per_device_once((const void*)&c_choose, mid_upload_constants); }

}  // namespace pg
