// The midsolve passes of a board with up to 10 empty spots, over index tables.
//
// Where an item of a level reads and writes depends only on how many spots are
// empty, not on the board: which entries of the level below its children are,
// where it goes, and whose wins it takes.  With up to 10 empty spots that is
// 17,303 items at most, so these indexes are listed once per device, like the
// library's other lookup tables, and a pass is left with the work that depends
// on the board.  The tables list, per level, a word per item and a 16-bit
// entry per item and child, child by child (so that a warp's loads are runs).
#pragma once
#include "mid_body.cuh"
#include <vector>

namespace pg {

constexpr int kSmallSpots = 10;

struct small_job {
  uint64_t side[2];
  uint32_t ply;
  int32_t spots;
  uint8_t empty[kSmallSpots + 6];
  pg_mid_values_t* out;
};

struct small_table {
  int32_t spots;
  int32_t nwins;            // entries of the wins table: (level, s1) as in mid_job_t::wins1_off
  int32_t items[12];        // per level n: items,
  int32_t rec[12], child[12];  //   where their words and children start,
  int32_t lo[12];           //   where the level lies in the workspace,
  int32_t wins[12];         //   and its first wins entry
  const uint32_t* recs;     // o | s0 << 13 | s1 << 21: the entry written, and the two sides' subsets
  const uint16_t* children;
  const uint16_t* subsets;  // per wins entry: the subset of the empty spots | level << 10
};

// Half h of wins entry x (0: the level's parity, 1: the other) lies at
// 2 x + h; after them, the wins of level 0's side 0.  put(i, v) stores word i.
template<class Put>
PG_HD void small_wins(const small_job& J, const uint32_t* wf, const small_table& T, int tid, int nt, Put put) {
  for (int x = tid; x <= T.nwins; x += nt) {
    const bool last = x == T.nwins;
    const uint32_t e = last ? 0u : ldg(T.subsets + x);
    const int n = int(e >> 10), parity = int((n + J.ply) & 1);
    const uint64_t side = J.side[(T.spots + n + !last) & 1] | set_side(J.empty, T.spots, e & 1023);
    const super8 w = s_super_wins(wf, side);
    put(2 * x, h_to(s_split(w, parity)));
    if (!last) put(2 * x + 1, h_to(s_split(w, !parity)));
  }
}

// An item's word and its C children's entries.
template<int C> struct small_item {
  uint32_t rec;
  uint32_t child[C ? C : 1];
  PG_HD void load(const small_table& T, int n, int it) {
    if (it >= T.items[n]) return;
    rec = ldg(T.recs + T.rec[n] + it);
    const uint16_t* c = T.children + T.child[n] + it;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int i = 0; i < C; i++) child[i] = ldg(c + i * T.items[n]);
  }
};

// Levels n = spots - C down to 0 of one pass (inner, mid/internal.h:358-408);
// `next` is the thread's first item of level n, and a level's next item is
// loaded while the current one is computed, across the barrier too.
template<int C, class Barrier>
PG_HD void small_levels(const small_table& T, int aggressive, uint4* ws, const uint4* wins, uint4* results,
                        small_item<C> next, int tid, int nt, Barrier barrier) {
  const int n = T.spots - C, items = T.items[n];
  const uint4* in = ws + (C ? T.lo[n + 1] : 0);
  uint4* out = ws + T.lo[n];
  const uint4* w1 = wins + 2 * T.wins[n];
  const uint4* w0 = n ? wins + 2 * T.wins[n - 1] + 1 : wins + 2 * T.nwins;
  const int turn_aggressive = aggressive ^ (n & 1);
  const uint32_t first = C == 0 && !turn_aggressive ? ~0u : 0u, keep = turn_aggressive ? ~0u : 0u;
  for (int it = tid; it < items; it += nt) {
    const small_item<C> now = next;
    next.load(T, n, it + nt);
    half4 us = half4{{first, first, first, first}};
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int i = 0; i < C; i++) us = h_or(us, h_from(in[now.child[i]]));
    const unsigned s0 = now.rec >> 13 & 255, s1 = now.rec >> 21;
    const half4 wins0 = h_from(w0[2 * s0]), after = h_from(w1[2 * s1]), before = h_from(w1[2 * s1 + 1]);
    half4 lost;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int k = 0; k < 4; k++) {
      us.w[k] = (us.w[k] & ~(wins0.w[k] | after.w[k])) | (wins0.w[k] & ~(after.w[k] & keep));
      lost.w[k] = ~us.w[k];
    }
    if (n <= 1) results[n + it] = h_to(us);
    out[now.rec & 8191] = h_to(h_or(h_rmax(lost), before));
  }
  if constexpr (C < kSmallSpots) {
    if (n == 0) return;
    small_item<C + 1> after;
    after.load(T, n - 1, tid);
    barrier();
    small_levels<C + 1>(T, aggressive, ws, wins, results, after, tid, nt, barrier);
  }
}

// One pass over a workspace of bottleneck(spots) entries; the wins table must
// be complete.  results: entries 0 .. spots.
template<class Barrier>
PG_HD void small_pass(const small_table& T, int aggressive, uint4* ws, const uint4* wins, uint4* results, int tid,
                      int nt, Barrier barrier) {
  small_item<0> first;
  first.load(T, T.spots, tid);
  small_levels<0>(T, aggressive, ws, wins, results, first, tid, nt, barrier);
}

// The tables of every count of empty spots up to kSmallSpots, on the host.
struct small_tables_host {
  small_table table[kSmallSpots + 1];
  std::vector<uint32_t> recs;
  std::vector<uint16_t> children, subsets;
  size_t rec0[kSmallSpots + 1], child0[kSmallSpots + 1], subset0[kSmallSpots + 1];   // where each count's start
};
const small_tables_host& small_tables();

}  // namespace pg
