// Learned-model rANS for solved blocks (stream format version 3) and the
// kernels that train its network.  The model and the exact arithmetic of the
// coding path are specified in learned.cuh.
//
// Coder layout: 32 lanes per stream; lane l codes the run of nodes l R ..
// l R + R - 1 (R = ceil(n / 32)), node l R + k in round k, its own rANS
// state walking the steps (round, rotation) in order.  The encoder runs the
// steps backward; at each step the lanes that renormalize append one 16-bit
// word each, in lane order, to the stream's shared word array, so the decoder
// (running forward) finds the words of its step as the last unread ones.
//
// Training: the forward pass and the backward pass of the softmax cross
// entropy with the bf16-rounded weights run on the tensor cores, 16 samples
// (stream, node, rotation) to a warp; partial sums per CTA are added in a
// fixed order, and an Adam step updates the fp32 master parameters.
#include "learned.cuh"
#include "lines.h"
#include "runtime.h"
#include "tables.h"
#include "../../include/pentago_b200.h"
#include <algorithm>
#include <vector>

namespace pg {

// Format-2 coder (rans.cu); the decoder can be restricted to version-2 streams.
int64_t rans_stream_bound(int64_t n);
int launch_rans_encode(const uint8_t* symbols, const int64_t* offsets, int nstreams, uint8_t* out,
                       const int64_t* out_offsets, int64_t* sizes, const int64_t* expect, cudaStream_t stream);
int launch_rans_decode(const uint8_t* in, const int64_t* in_offsets, const int64_t* in_sizes, int nstreams,
                       uint8_t* symbols, const int64_t* sym_offsets, const int64_t* sym_caps, int64_t* status,
                       int only_v2, cudaStream_t stream);

constexpr int kLmWarps = 4;
constexpr int kLmThreads = 32 * kLmWarps;
constexpr int kLmCtxRows = kLmIn - kLmRot;   // W1 rows 72..123: the rotation, neighbour and previous-node features

// Tables of the frequency check kernel in shared memory, transposed: one row
// of 64 bf16 (8 chunks of 16 bytes) per output unit, w1t row k with
// W1[72 + 8 c .. 72 + 8 c + 7][k] in chunk c (c < 7), w2t row j with
// W2[8 c .. 8 c + 7][j], chunk c at c ^ (row & 7).
struct lm_tables {
  uint4 w1t[kLmHidden][8];
  uint4 w2t[kLmHidden][8];
  float b1[kLmHidden], b2[kLmHidden];
  float w3[kLmHidden][4];        // [j][c]
  float b3[4];
};

__device__ __forceinline__ int swz(int row, int chunk) { return chunk ^ (row & 7); }

__device__ void lm_build_tables(lm_tables& S, const uint16_t* __restrict__ P, int tid, int nt) {
  auto w = [&](int i) { return bf16_value(P[i]); };
  for (int i = tid; i < kLmHidden * 8; i += nt) {
    const int j = i >> 3, c = i & 7;
    uint32_t v[4], u[4];
    for (int e = 0; e < 4; e++) {
      const int f = 8 * c + 2 * e;   // feature rows 72 + f, 72 + f + 1 (zero past the 48)
      u[e] = f < kLmCtxRows ? uint32_t(P[kLmW1 + (kLmRot + f) * kLmHidden + j]) |
                                  uint32_t(P[kLmW1 + (kLmRot + f + 1) * kLmHidden + j]) << 16
                            : 0u;
      v[e] = uint32_t(P[kLmW2 + (8 * c + 2 * e) * kLmHidden + j]) |
             uint32_t(P[kLmW2 + (8 * c + 2 * e + 1) * kLmHidden + j]) << 16;
    }
    S.w1t[j][swz(j, c)] = make_uint4(u[0], u[1], u[2], u[3]);
    S.w2t[j][swz(j, c)] = make_uint4(v[0], v[1], v[2], v[3]);
  }
  for (int i = tid; i < kLmHidden; i += nt) {
    S.b1[i] = w(kLmB1 + i);
    S.b2[i] = w(kLmB2 + i);
    for (int c = 0; c < 3; c++) S.w3[i][c] = w(kLmW3 + i * kLmOut + c);
    S.w3[i][3] = 0.f;
  }
  if (tid < 3) S.b3[tid] = w(kLmB3 + tid);
  if (tid == 3) S.b3[3] = 0.f;
}

// Element k of row t of a transposed table (bf16 -> float).
__device__ __forceinline__ float lm_tab(const uint4 (*tab)[8], int row, int k) {
  const uint4 ch = tab[row][swz(row, k >> 3)];
  const uint32_t pr = (k & 7) < 2 ? ch.x : (k & 7) < 4 ? ch.y : (k & 7) < 6 ? ch.z : ch.w;
  return f_bits(k & 1 ? pr & 0xffff0000u : pr << 16);
}

// node[k] = b1[k] + stone rows, ascending (registers of one thread); the
// stone rows are read from the model (bf16, global memory: a lane reads them
// once per node).
__device__ __forceinline__ void lm_node_sum(const float* b1, const uint16_t* __restrict__ P, const uint8_t* feats,
                                            int nf, float* node) {
#pragma unroll
  for (int k = 0; k < kLmHidden; k++) node[k] = b1[k];
  for (int i = 0; i < nf; i++) {
    const uint4* row = reinterpret_cast<const uint4*>(P + kLmW1 + feats[i] * kLmHidden);
#pragma unroll
    for (int c = 0; c < 8; c++) {
      const uint4 v = ldg(row + c);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int e = 0; e < 4; e++) {
        node[8 * c + 2 * e] = f_add(node[8 * c + 2 * e], f_bits(w[e] << 16));
        node[8 * c + 2 * e + 1] = f_add(node[8 * c + 2 * e + 1], f_bits(w[e] & 0xffff0000u));
      }
    }
  }
}

// The 4 rotation, 8 neighbour and 1 previous-node features of symbol r
// (indices into W1 rows 72..123): 4 q + i_q, then 16 + 4 n + v_n with
// u[q] = v_2q + 4 v_2q+1, then 48 + the previous node's symbol (3: none).
__device__ __forceinline__ void lm_ctx_features(int r, const int* u, int prev, int* f) {
#pragma unroll
  for (int q = 0; q < 4; q++) {
    f[q] = 4 * q + ((r >> (2 * q)) & 3);
    f[4 + 2 * q] = 16 + 8 * q + (u[q] & 3);
    f[5 + 2 * q] = 20 + 8 * q + (u[q] >> 2);
  }
  f[12] = kLmPrev - kLmRot + prev;
}

// Logits of one symbol, one thread (the frequency check kernel): S1 and C by
// fp32 chains, exact on a model whose grid columns are on their grids, and layer 3 in the order of
// learned.cuh.
__device__ __forceinline__ void lm_logits(const lm_tables& S, const float* node, int r, const int* u, int prev,
                                          float* z) {
  int f[13];
  lm_ctx_features(r, u, prev, f);
  float hq[kLmHidden];
  for (int k = 0; k < kLmHidden; k++) {
    float s1 = 0.f;
    for (int i = 0; i < 13; i++) s1 = f_add(s1, lm_tab(S.w1t, k, f[i]));
    hq[k] = lm_act_q(f_add(node[k], s1));
  }
  float part[4][3];
#pragma unroll
  for (int t = 0; t < 4; t++) part[t][0] = part[t][1] = part[t][2] = 0.f;
  for (int j = 0; j < kLmHidden; j++) {
    float c = 0.f;
    for (int k = 0; k < kLmHidden; k++) c = f_fma(lm_tab(S.w2t, j, k), hq[k], c);
    const float h = relu(f_fma(c, kLmActInv, S.b2[j]));
    const int t = (j >> 1) & 3;
    for (int cc = 0; cc < 3; cc++) part[t][cc] = f_fma(S.w3[j][cc], h, part[t][cc]);
  }
  for (int cc = 0; cc < 3; cc++)
    z[cc] = f_add(S.b3[cc], f_add(f_add(part[0][cc], part[1][cc]), f_add(part[2][cc], part[3][cc])));
}

// Tensor-core pieces (mma.sync m16n8k16, bf16 inputs, fp32 accumulation).
__device__ __forceinline__ void ldsm_x4(uint32_t* r, const void* p) {
  const unsigned a = unsigned(__cvta_generic_to_shared(p));
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void mma_bf16(float* d, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
               "{%8, %9}, {%0, %1, %2, %3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// ---------------------------------------------------------------------------
// Coding: logits on the tensor cores (tcgen05, tensor memory)

// Tables and operands of a coding CTA, from a base of 1,024 bytes.  The
// operands of the products are K-major rows of 64 bf16 in the 128-byte swizzle (chunk c of row j at
// c ^ (j & 7)): w1t row k holds W1[72 ..][k] / 16, w2t row i holds W2[..][j] of
// the unit j that accumulator column i is, lm_unit(i); operand[t] the 128
// rows of tile t.
struct lm_coder {
  uint4 w1t[kLmHidden][8];
  uint4 w2t[kLmHidden][8];
  uint4 operand[2][128][8];
  float b1[kLmHidden];
  uint64_t mbar[2];
  uint32_t tmem;
  uint32_t pad[3];
};

// Accumulator columns are ordered so that columns 2 i and 2 i + 1 belong to the
// chains P_t and P_t+1 (t even) of layer 3: one packed operation serves both.
__host__ __device__ __forceinline__ int lm_unit(int column) { return (column & ~7) + 2 * (column & 3) + (column >> 2 & 1); }

// What all threads read at the same place, as a kernel parameter (read from
// shared memory, by 32 lanes at once, layer 3's weights took as long as its
// arithmetic): layer 3 and the biases beside it, per pair of accumulator
// columns, and where each step finds its symbols' neighbours.
struct lm_const {
  struct alignas(16) { float b2[2], w3[3][2]; } at[kLmHidden / 2];
  uint32_t near[128][4];   // per neighbour of symbol st 16 bits: its word in the row | lm_symbol16's rotation << 8
  float b3[4];
};
static lm_const lm_consts(const uint8_t* model) {
  auto w = [&](int i) {
    const uint8_t* p = model + kLmModelHeader + 2 * i;
    return bf16_value(uint16_t(p[0] | p[1] << 8));
  };
  lm_const O = {};
  for (int i = 0; i < kLmHidden; i++) {
    O.at[i >> 1].b2[i & 1] = w(kLmB2 + lm_unit(i));
    for (int c = 0; c < 3; c++) O.at[i >> 1].w3[c][i & 1] = w(kLmW3 + lm_unit(i) * kLmOut + c);
  }
  for (int st = 0; st < 128; st++)
    for (int n = 0; n < 8; n++) {
      const int a = lm_neighbour(st, n);
      O.near[st][n >> 1] |= uint32_t((a >> 4) | ((2 * a - 4) & 31) << 8) << (16 * (n & 1));
    }
  for (int c = 0; c < 3; c++) O.b3[c] = w(kLmB3 + c);
  return O;
}

__device__ void lm_build_coder(lm_coder& S, const uint16_t* __restrict__ P, int tid, int nt) {
  auto w = [&](int i) { return bf16_value(P[i]); };
  for (int i = tid; i < kLmHidden * 8; i += nt) {
    const int j = i >> 3, c = i & 7, unit = lm_unit(j);
    uint32_t v[4], u[4];
    for (int e = 0; e < 4; e++) {
      const int f = 8 * c + 2 * e;   // feature rows 72 + f, 72 + f + 1 (zero past the 52)
      u[e] = v[e] = 0;
      for (int h = 0; h < 2; h++) {
        // the sixteenth of a bf16 is one, except below 2^-122, where nothing is left of it in an activation
        if (f + h < kLmCtxRows)
          u[e] |= uint32_t(bf16_round(f_mul(w(kLmW1 + (kLmRot + f + h) * kLmHidden + j), kLmActInv))) << (16 * h);
        v[e] |= uint32_t(P[kLmW2 + (f + h) * kLmHidden + unit]) << (16 * h);
      }
    }
    S.w1t[j][swz(j, c)] = make_uint4(u[0], u[1], u[2], u[3]);
    S.w2t[j][swz(j, c)] = make_uint4(v[0], v[1], v[2], v[3]);
  }
  for (int i = tid; i < kLmHidden; i += nt) S.b1[i] = w(kLmB1 + i);
  // (read by the tensor cores)
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Tensor memory of a CTA, by column: the accumulators of its two tiles of 128
// rows; a warp reads its 32 lanes.
constexpr uint32_t kLmTmemCols = 128;
// Instruction descriptor: fp32 accumulators, bf16 A and B, both K-major, N = 64, M = 128.
constexpr uint32_t kLmIdesc = 1u << 4 | 1u << 7 | 1u << 10 | (kLmHidden / 8) << 17 | (128 / 16) << 24;

// Shared-memory descriptor of an operand: 128-byte swizzle, groups of 8 rows 1,024 bytes apart.
__device__ __forceinline__ uint64_t lm_desc(const void* rows) {
  const uint64_t a = __cvta_generic_to_shared(rows);
  return (a >> 4) | uint64_t(1) << 16 | uint64_t(1024 >> 4) << 32 | uint64_t(1) << 46 | uint64_t(2) << 61;
}
// Tile t's accumulators = operand x table (K = 64, in steps of 16), then an
// arrival on its barrier: one thread of warp t (a product takes its thread
// some 300 cycles to issue).
__device__ __forceinline__ void lm_product(lm_coder& S, const void* table) {
  const int t = int(threadIdx.x >> 5);
  if (t >= 2 || (threadIdx.x & 31)) return;
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint64_t a = lm_desc(S.operand[t]), b = lm_desc(table);
#pragma unroll
  for (int k = 0; k < 4; k++) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %4, 0;\n"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                 :: "r"(S.tmem + kLmHidden * t), "l"(a + 2 * k), "l"(b + 2 * k), "r"(kLmIdesc),
                    "r"(uint32_t(k > 0)) : "memory");
  }
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
               :: "r"(unsigned(__cvta_generic_to_shared(&S.mbar[t]))) : "memory");
}
// Waits for a tile's product; false if it has not come after a bounded number of polls.
__device__ __forceinline__ bool lm_product_wait(lm_coder& S, int t, uint32_t phase) {
  const unsigned bar = unsigned(__cvta_generic_to_shared(&S.mbar[t]));
  uint32_t done = 0;
  for (int poll = 0; poll < (1 << 20) && !done; poll++)
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.b32 %0, 1, 0, p;\n}\n"
                 : "=r"(done) : "r"(bar), "r"(phase) : "memory");
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  return done != 0;
}

#define PG_W8(v, b) "=r"(v[b]), "=r"(v[b + 1]), "=r"(v[b + 2]), "=r"(v[b + 3]), "=r"(v[b + 4]), "=r"(v[b + 5]), "=r"(v[b + 6]), "=r"(v[b + 7])
// 32 columns of the thread's row, or 16 each of two places (the wait belongs to
// the load: nothing may use the registers before it).
__device__ __forceinline__ void tmem_ld32(uint32_t* v, uint32_t at) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
               "%14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
               "tcgen05.wait::ld.sync.aligned;\n"
               : PG_W8(v, 0), PG_W8(v, 8), PG_W8(v, 16), PG_W8(v, 24) : "r"(at) : "memory");
}
__device__ __forceinline__ void tmem_ld16x2(uint32_t* v, uint32_t* w, uint32_t at, uint32_t bt) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
               "%14, %15}, [%32];\n"
               "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, "
               "%28, %29, %30, %31}, [%33];\n"
               "tcgen05.wait::ld.sync.aligned;\n"
               : PG_W8(v, 0), PG_W8(v, 8), PG_W8(w, 0), PG_W8(w, 8) : "r"(at), "r"(bt) : "memory");
}
#undef PG_W8

// Two fp32 operations, each rounded as usual, in one instruction.
__device__ __forceinline__ uint64_t f2(float a, float b) { return uint64_t(f_raw(b)) << 32 | f_raw(a); }
__device__ __forceinline__ float f2_lo(uint64_t v) { return f_bits(uint32_t(v)); }
__device__ __forceinline__ float f2_hi(uint64_t v) { return f_bits(uint32_t(v >> 32)); }
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float f_add_sat(float a, float b) {   // to [0, 1]; 0 for NaN
  float d;
  asm("add.rn.sat.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ uint32_t shl_clamped(uint32_t v, uint32_t by) {   // 0 from 32 on
  uint32_t d;
  asm("shl.b32 %0, %1, %2;" : "=r"(d) : "r"(v), "r"(by));
  return d;
}
// bf16 1.0 at element v16 / 16 of four: two words of the A operand.
__device__ __forceinline__ void onehot4(uint32_t* op, uint32_t v16) {
  op[0] = shl_clamped(0x3f80u, v16);
  op[1] = shl_clamped(0x3f80u, v16 - 32u);
}

// lm_act_q of two sums, as a bf16 pair.  a, b are the node's sums and s, t
// layer 1's products, all a sixteenth of theirs (exact), so that one
// saturated addition is the sum held to [0, 1], a 256th of the activation,
// with the cut at 256: adding 2^23 rounds it to an integer, and what then is
// 256 becomes 255.
__device__ __forceinline__ uint32_t lm_act_q2(float a, float s, float b, float t) {
  constexpr float two23 = 8388608.f;
  const uint64_t y = f2(f_add_sat(a, s), f_add_sat(b, t));
  const uint64_t q = f2_add(f2_fma(y, f2(256.f, 256.f), f2(two23, two23)), f2(-two23, -two23));
  uint32_t d;
  asm("min.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(__byte_perm(uint32_t(q), uint32_t(q >> 32), 0x7632)), "r"(0x437f437fu));
  return d;
}

// The coding kernels give a stream a warp: lane l has the node of the stream's
// lane l, whose two symbols of a step (neither is the other's neighbour) are
// row m of the CTA's two tiles, 128 rows of four streams.  All warps of a CTA
// take their steps together; nodes have 128 steps, so the streams of a CTA
// begin their nodes together, and a warp without a stream keeps step
// without coding.
//
// Dynamic shared memory: the tables and operands, then per warp two buffers
// of its nodes' symbols (the nodes being coded and the ones before them; 2
// bits a symbol, 3: not coded yet, 17 words a lane so that lanes reading the
// same rotation use different banks) and, for the decoder, a window of the
// stream's next words.
//
// Bound by the instructions of a step, 1,700 a warp, and their chain: 7,500
// cycles for three warps a scheduler, of which the operands take 900, the
// products 700 each, activations 900, layer 3 1,300, the frequencies 1,000 and the
// states 700.  2,048 blocks of a solved slice: 75 ms each way; 166 with mma.sync
// (256 products a step and stream), 87 with two warps per stream, one tile
// and the operands in tensor memory (6 streams an SM instead of 12).
constexpr int kLmCodeThreads = 128;
constexpr int kLmRowWords = 17;
constexpr int kLmWordWin = 512;   // the decoder's window of upcoming stream words
constexpr size_t kLmStreamSmem = size_t(2) * 32 * 4 * kLmRowWords + 2 * kLmWordWin;
constexpr size_t kLmCodeSmem = 1024 + sizeof(lm_coder) + 4 * kLmStreamSmem;   // (from a multiple of 1,024)
constexpr int kLmCodeCtas = 3;
static_assert(sizeof(lm_coder) % 16 == 0 && kLmStreamSmem % 16 == 0, "coding rows stay aligned");
static_assert(kLmCodeCtas * kLmTmemCols <= 512, "tensor memory of an SM");

struct lm_warp {   // a thread's place, and its warp's buffers
  int lane;
  uint32_t* row[2];
  uint16_t* win;
  __device__ __forceinline__ void fill(uint32_t* to) const {
    for (int w = 0; w < 16; w++) to[w] = 0xffffffffu;
  }
  // A node's 256 symbols between global memory and its row; true if one is above 2.
  __device__ __forceinline__ bool in(uint32_t* to, const uint8_t* g) const {
    bool bad = false;
    const bool aligned = (reinterpret_cast<uintptr_t>(g) & 3) == 0;
#pragma unroll 2
    for (int w = 0; w < 16; w++) {
      uint32_t word = 0;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const uint8_t* from = g + 16 * w + 4 * k;
        const uint32_t v = aligned ? *reinterpret_cast<const uint32_t*>(from)
                                   : from[0] | from[1] << 8 | from[2] << 16 | uint32_t(from[3]) << 24;
        bad |= (v & 0xfcfcfcfcu) != 0 || (v & v >> 1 & 0x01010101u) != 0;   // a byte above 2
        word |= ((v & 3) | (v >> 6 & 0xc) | (v >> 12 & 0x30) | (v >> 18 & 0xc0)) << (8 * k);
      }
      to[w] = word;
    }
    return bad;
  }
  __device__ __forceinline__ void out(const uint32_t* from, uint8_t* g) const {
    const bool aligned = (reinterpret_cast<uintptr_t>(g) & 3) == 0;
#pragma unroll 2
    for (int w = 0; w < 16; w++) {
      const uint32_t word = from[w];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const uint32_t b = word >> (8 * k), v = (b & 3) | (b & 0xc) << 6 | (b & 0x30) << 12 | (b & 0xc0) << 18;
        uint8_t* at = g + 16 * w + 4 * k;
        if (aligned) *reinterpret_cast<uint32_t*>(at) = v;
        else
          for (int e = 0; e < 4; e++) at[e] = uint8_t(v >> (8 * e));
      }
    }
  }
};

// The next stream of a launch, largest first (streams are handed to warps one
// at a time through a counter, in the order the host sorted them), or -1.
__device__ __forceinline__ int lm_next_stream(int* next, const int32_t* order, int nstreams, int lane) {
  int k = 0;
  if (lane == 0) k = atomicAdd(next, 1);
  k = __shfl_sync(0xffffffffu, k, 0);
  return k < nstreams ? order[k] : -1;
}

__device__ __forceinline__ uint32_t lm_symbol16(uint32_t word, uint32_t rotation) {   // 16 v, given v's word
  return __funnelshift_r(word, word, rotation) & 48u;
}

// lm_freqs of two rows' logits at once, operation by operation.
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t f2_both(float v) { return f2(v, v); }
__device__ __forceinline__ void lm_freqs2(const uint64_t* z, lm_freq_t* F) {
  auto top = [](float a, float b, float c) {   // (a NaN is passed over unless it comes first)
    a = b > a ? b : a;
    return c > a ? c : a;
  };
  const uint64_t m = f2(top(f2_lo(z[0]), f2_lo(z[1]), f2_lo(z[2])), top(f2_hi(z[0]), f2_hi(z[1]), f2_hi(z[2])));
  uint64_t e[3];
#pragma unroll
  for (int c = 0; c < 3; c++) {   // lm_exp2
    const uint64_t d = f2_mul(f2_fma(m, f2_both(-1.f), z[c]), f2_both(1.44269504f));
    uint64_t u;
    asm("add.rm.f32x2 %0, %1, %2;" : "=l"(u) : "l"(d), "l"(f2_both(12582912.f)));
    const uint64_t t = f2_fma(f2_add(u, f2_both(-12582912.f)), f2_both(-1.f), d);
    uint64_t p = f2_both(1.5252734e-05f);
    p = f2_fma(p, t, f2_both(1.5403530e-04f));
    p = f2_fma(p, t, f2_both(1.3333558e-03f));
    p = f2_fma(p, t, f2_both(9.6181291e-03f));
    p = f2_fma(p, t, f2_both(5.5504109e-02f));
    p = f2_fma(p, t, f2_both(2.4022651e-01f));
    p = f2_fma(p, t, f2_both(6.9314718e-01f));
    p = f2_fma(p, t, f2_both(1.0f));
    p = f2_mul(p, f2(f_bits((uint32_t(u) << 23) + 0x3f800000u), f_bits((uint32_t(u >> 32) << 23) + 0x3f800000u)));
    e[c] = f2(f2_lo(d) >= -24.f ? f2_lo(p) : 0.f, f2_hi(d) >= -24.f ? f2_hi(p) : 0.f);
  }
  const uint64_t s = f2_add(f2_add(e[0], e[1]), e[2]);
#pragma unroll
  for (int row = 0; row < 2; row++) {
    auto half = [&](uint64_t v) { return row ? f2_hi(v) : f2_lo(v); };
    uint32_t f[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const float a = half(e[c]), q = f_mul(f_div(a > 0.f ? a : 1.f, half(s)), float(kLmProbTotal - 3));
      f[c] = 1 + (a > 0.f ? lm_trunc(q) : 0u);
    }
    const uint32_t rest = kLmProbTotal - (f[0] + f[1] + f[2]);
    const bool one = f[1] > f[0], two = f[2] > (one ? f[1] : f[0]);
    f[0] += one || two ? 0 : rest;
    f[1] += one && !two ? rest : 0;
    f[2] += two ? rest : 0;
    F[row].f[0] = f[0];
    F[row].f[1] = f[1];
    F[row].f[2] = f[2];
    F[row].cum[0] = 0;
    F[row].cum[1] = f[0];
    F[row].cum[2] = f[0] + f[1];
  }
}

// Row m of both tiles' operands for step st: the one-hot features of symbols st
// and st + 128 (rotation, neighbours, the previous node's symbol, zeros), a
// chunk of two features after the other.
__device__ __forceinline__ void lm_operands(lm_coder& S, const lm_const& O, const uint32_t* row, const uint32_t* prev, int st, int m) {
  // (all loads before the first store, which the compiler may not move them past)
  uint32_t sym[2][10];
#pragma unroll
  for (int c = 0; c < 4; c++) {
    // (a symbol 128 on is 8 words on, in the same place)
    const uint32_t near = O.near[st][c], a = near & 15, b = near >> 16 & 15;
#pragma unroll
    for (int t = 0; t < 2; t++) {
      sym[t][2 * c] = lm_symbol16(row[a ^ 8 * t], near >> 8);
      sym[t][2 * c + 1] = lm_symbol16(row[b ^ 8 * t], near >> 24);
    }
  }
#pragma unroll
  for (int t = 0; t < 2; t++) {
    sym[t][8] = lm_symbol16(prev[(st >> 4) + 8 * t], 2 * st - 4);
    sym[t][9] = 64;   // (none)
  }
#pragma unroll
  for (int t = 0; t < 2; t++) {
    auto put = [&](int c, uint32_t a16, uint32_t b16) {
      uint32_t op[4];
      onehot4(op, a16);
      onehot4(op + 2, b16);
      S.operand[t][m][swz(m, c)] = make_uint4(op[0], op[1], op[2], op[3]);
    };
    const int r = st + 128 * t;
    put(0, uint32_t(r & 3) << 4, uint32_t(r >> 2 & 3) << 4);
    put(1, uint32_t(r >> 4 & 3) << 4, uint32_t(r >> 6 & 3) << 4);
#pragma unroll
    for (int c = 0; c < 5; c++) put(2 + c, sym[t][2 * c], sym[t][2 * c + 1]);
    S.operand[t][m][swz(m, 7)] = make_uint4(0, 0, 0, 0);
  }
}

// Frequencies of the two symbols of step st of the thread's node.  row has the
// node's symbols, prev the previous node's; node: the node's sums / 16.  The
// CTA's 128 threads are the rows of the products and come here together.
// ok: the thread has seen all its products so far; false is returned to all of
// them if one of them has not (the caller looks at ok after its last step).
// phase is the parity of the latest products; with `drill` the wait for the
// second is taken to have run out.
__device__ __forceinline__ bool lm_step_freqs(lm_coder& S, const lm_const& O, const uint32_t* row, const uint32_t* prev,
                                              int st, const float* node, uint32_t& phase, bool& ok, lm_freq_t* F,
                                              bool drill) {
  const int m = threadIdx.x;
  const uint32_t tm = S.tmem + (uint32_t(m) >> 5 << 21);   // the warp's lanes
  lm_operands(S, O, row, prev, st, m);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (__syncthreads_or(!ok)) return false;
  phase ^= 1;
  lm_product(S, S.w1t);
#pragma unroll
  for (int t = 0; t < 2; t++) {
    ok &= lm_product_wait(S, t, phase);
#pragma unroll
    for (int h = 0; h < kLmHidden; h += 32) {
      uint32_t acc[32], op[16];
      tmem_ld32(acc, tm + kLmHidden * t + h);
#pragma unroll
      for (int i = 0; i < 16; i++)
        op[i] = lm_act_q2(node[h + 2 * i], f_bits(acc[2 * i]), node[h + 2 * i + 1], f_bits(acc[2 * i + 1]));
#pragma unroll
      for (int c = 0; c < 4; c++)
        S.operand[t][m][swz(m, h / 8 + c)] = make_uint4(op[4 * c], op[4 * c + 1], op[4 * c + 2], op[4 * c + 3]);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\nfence.proxy.async.shared::cta;" ::: "memory");
  if (__syncthreads_or(!ok)) return false;
  phase ^= 1;
  lm_product(S, S.w2t);
  ok &= lm_product_wait(S, 0, phase) && !drill;
  ok &= lm_product_wait(S, 1, phase);
  // Layer 3 of both rows at once, each constant used twice: P_0 and P_1, P_2 and P_3
  uint64_t part[2][2][3] = {};
#pragma unroll
  for (int h = 0; h < kLmHidden; h += 16) {
    uint32_t acc[2][16];
    tmem_ld16x2(acc[0], acc[1], tm + h, tm + kLmHidden + h);
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const auto& o = O.at[h / 2 + i];
#pragma unroll
      for (int t = 0; t < 2; t++) {
        const uint64_t a =
            f2_fma(uint64_t(acc[t][2 * i + 1]) << 32 | acc[t][2 * i], f2(kLmActInv, kLmActInv), f2(o.b2[0], o.b2[1]));
        const uint64_t v = f2(relu(f2_lo(a)), relu(f2_hi(a)));
#pragma unroll
        for (int c = 0; c < 3; c++) part[t][i & 1][c] = f2_fma(f2(o.w3[c][0], o.w3[c][1]), v, part[t][i & 1][c]);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  uint64_t z[3];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    auto chains = [&](int i) {   // of both rows, each the sum of its two
      const uint64_t a = part[0][i][c], b = part[1][i][c];
      return f2_add(f2(f2_lo(a), f2_lo(b)), f2(f2_hi(a), f2_hi(b)));
    };
    z[c] = f2_add(f2(O.b3[c], O.b3[c]), f2_add(chains(0), chains(1)));
  }
  lm_freqs2(z, F);
  return true;
}

// Neighbour context of symbol r from the node's symbols (those of earlier
// steps; later ones read as 3), packed as 4 bits per quadrant.
__device__ __forceinline__ uint32_t lm_context_packed(const uint8_t* sym, int r) {
  uint32_t p = 0;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int a = lm_neighbour(r, 2 * q), b = lm_neighbour(r, 2 * q + 1);
    const int va = lm_before(a, r) ? (sym[a] & 3) : 3, vb = lm_before(b, r) ? (sym[b] & 3) : 3;
    p |= uint32_t(va + 4 * vb) << (4 * q);
  }
  return p;
}
__device__ __forceinline__ void lm_context_clamped(const uint8_t* sym, int r, int* u) {
  const uint32_t p = lm_context_packed(sym, r);
#pragma unroll
  for (int q = 0; q < 4; q++) u[q] = int(p >> (4 * q)) & 15;
}

__device__ __forceinline__ int lm_load_node(const lm_block_t& B, int64_t i, const dev_tables_t& T, uint8_t* feats) {
  uint16_t qid[4];
  lm_node_quadrants(B, i, T.rmin_flat, qid);
  return lm_node_features(qid, T.unpack, feats);
}

__device__ __forceinline__ void put16(uint8_t* p, uint16_t v) { p[0] = uint8_t(v); p[1] = uint8_t(v >> 8); }
__device__ __forceinline__ uint16_t get16(const uint8_t* p) { return uint16_t(p[0] | p[1] << 8); }
__device__ __forceinline__ void put32(uint8_t* p, uint32_t v) { for (int i = 0; i < 4; i++) p[i] = uint8_t(v >> (8 * i)); }
__device__ __forceinline__ uint32_t get32(const uint8_t* p) {
  return uint32_t(p[0]) | uint32_t(p[1]) << 8 | uint32_t(p[2]) << 16 | uint32_t(p[3]) << 24;
}

// Tables, tensor memory and barriers of a coding CTA; and giving them back.
__device__ lm_coder& lm_coder_begin(unsigned char* raw, const uint16_t* __restrict__ P, lm_warp& W) {
  unsigned char* base = raw + ((1024 - (__cvta_generic_to_shared(raw) & 1023)) & 1023);
  lm_coder& S = *reinterpret_cast<lm_coder*>(base);
  const int warp = threadIdx.x >> 5;
  W.lane = threadIdx.x & 31;
  unsigned char* mine = base + sizeof(lm_coder) + kLmStreamSmem * warp;
  for (int b = 0; b < 2; b++) W.row[b] = reinterpret_cast<uint32_t*>(mine) + (32 * b + W.lane) * kLmRowWords;
  W.win = reinterpret_cast<uint16_t*>(mine + 2 * 32 * 4 * kLmRowWords);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(unsigned(__cvta_generic_to_shared(&S.tmem))), "r"(kLmTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (threadIdx.x == 0) {
    for (int t = 0; t < 2; t++)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(unsigned(__cvta_generic_to_shared(&S.mbar[t]))) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  lm_build_coder(S, P, threadIdx.x, blockDim.x);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  return S;
}
// `whole`: every product has been seen.  Those that have not are given as long
// again, so that tensor memory is not freed under them.
__device__ void lm_coder_end(lm_coder& S, bool whole, uint32_t phase) {
  if (!whole)
    for (int t = 0; t < 2; t++) lm_product_wait(S, t, phase);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (threadIdx.x < 32)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(S.tmem), "r"(kLmTmemCols) : "memory");
}

// The sums of the thread's node (b1 + stone rows ascending), / 16.
__device__ __forceinline__ void lm_coder_node(const lm_coder& S, const uint16_t* __restrict__ P, const lm_block_t& B,
                                              int64_t i, bool active, const dev_tables_t& T, float* node) {
  uint8_t feats[36];
  const int nf = active ? lm_load_node(B, i, T, feats) : 0;
  lm_node_sum(S.b1, P, feats, nf, node);
#pragma unroll
  for (int k = 0; k < kLmHidden; k++) node[k] = f_mul(node[k], kLmActInv);
}

// Append one 16-bit word per renormalizing lane, in lane order, as long as
// there is room (encoder); inv is 1 / f, rounded.
__device__ __forceinline__ void lm_put_state(uint32_t& x, uint32_t f, float inv, uint32_t cum, bool active, uint8_t* words,
                                             uint32_t room, uint32_t& len, unsigned below) {
  const bool emit = active && x >= (f << 17);
  const unsigned mask = __ballot_sync(0xffffffffu, emit);
  if (emit) {
    const uint32_t at = len + __popc(mask & below);
    if (at < room) put16(words + 2 * size_t(at), uint16_t(x));
    x >>= 16;
  }
  len += __popc(mask);
  // x / f < 2^17: an estimate by the reciprocal is off by less than 2^-4, so
  // its integer part by one at most
  uint32_t q = __float2uint_rz(f_mul(__uint2float_rz(x), inv));
  int r = int(x - q * f);
  q += r < 0 ? ~0u : r >= int(f) ? 1u : 0u;
  r += r < 0 ? int(f) : r >= int(f) ? -int(f) : 0;
  if (active) x = (q << kLmProbBits) + uint32_t(r) + cum;
}

// Decode one symbol per active lane and take this step's words (decoder);
// f0 and f1 are the frequencies of symbols 0 and 1.  Words [wlo, wlo +
// kLmWordWin) are also in win.
__device__ __forceinline__ int lm_get_symbol(uint32_t& x, uint32_t f0, uint32_t f1, bool active, const uint8_t* words,
                                             const uint16_t* win, int64_t wlo, int64_t& ptr, unsigned above,
                                             int& bad) {
  int v = 0;
  if (active) {
    const uint32_t slot = x & (kLmProbTotal - 1), f01 = f0 + f1;
    v = slot < f0 ? 0 : slot < f01 ? 1 : 2;
    const uint32_t cum = v == 0 ? 0 : v == 1 ? f0 : f01, f = v == 0 ? f0 : v == 1 ? f1 : kLmProbTotal - f01;
    x = f * (x >> kLmProbBits) + slot - cum;
  }
  const bool need = active && x < kLmLower;
  const unsigned mask = __ballot_sync(0xffffffffu, need);
  const int64_t at = ptr - 1 - __popc(mask & above);
  if (need) {
    if (at >= wlo) x = (x << 16) | win[at - wlo];
    else if (at >= 0) x = (x << 16) | get16(words + 2 * at);
    else bad = 1;
  }
  ptr -= __popc(mask);
  return v;
}

// sizes[s] = stream bytes, or PG_ERR_ARG for a symbol above 2 or a symbol
// count that does not match; what it was before (PG_ERR_CUDA) if the stream's
// CTA, or all of them, gave up on a product.
// kDrill: the wait for a stream's last product is taken to have run out, to see
// what then becomes of the streams.
template<bool kDrill>
__global__ void __launch_bounds__(kLmCodeThreads, kLmCodeCtas)
lm_encode_kernel(const uint16_t* __restrict__ P, uint64_t hash, const lm_block_t* __restrict__ blocks, int nstreams,
                 const int32_t* __restrict__ order, int* __restrict__ next, const uint8_t* __restrict__ symbols,
                 const int64_t* __restrict__ offsets, uint8_t* __restrict__ out,
                 const int64_t* __restrict__ out_offsets, const int64_t* __restrict__ caps,
                 const int64_t* __restrict__ alt_sizes, int64_t* __restrict__ sizes, const dev_tables_t T,
                 const __grid_constant__ lm_const O) {
  extern __shared__ __align__(16) unsigned char lm_smem_raw[];
  lm_warp W;
  lm_coder& S = lm_coder_begin(lm_smem_raw, P, W);
  const unsigned below = (1u << W.lane) - 1;
  int s = -1, cur = 0;
  bool more = true, ok = true, whole = true;
  uint32_t phase = 1;
  int64_t n = 0, R = 0, round = -1;   // R: the run of nodes of each lane
  const uint8_t* sym0 = nullptr;
  uint8_t *base = nullptr, *words = nullptr;
  uint32_t x = kLmLower, len = 0, room = 0;
  int bad = 0;
  lm_block_t B = {};
  while (whole) {
    while (more && round < 0) {
      if (s >= 0) {   // the stream is done
        put32(base + 20 + 4 * W.lane, x);
        bad = __any_sync(0xffffffffu, bad);
        if (W.lane == 0) {
          put32(base, kLmVersion);
          put32(base + 4, uint32_t(hash));
          put32(base + 8, uint32_t(hash >> 32));
          put32(base + 12, uint32_t(n));
          put32(base + 16, len);
          sizes[s] = bad ? PG_ERR_ARG : kLmStreamHeader + 2 * int64_t(len);
        }
      }
      s = lm_next_stream(next, order, nstreams, W.lane);
      more = s >= 0;
      if (!more) break;
      B = blocks[s];
      n = B.nodes;
      if (offsets[s + 1] - offsets[s] != 256 * n) {
        if (W.lane == 0) sizes[s] = PG_ERR_ARG;
        s = -1;
        continue;
      }
      sym0 = symbols + offsets[s];
      base = out + out_offsets[s];
      words = base + kLmStreamHeader;
      const int64_t end = caps[s] - (alt_sizes[s] > 0 ? alt_sizes[s] : 0) - kLmStreamHeader;   // (bytes)
      room = end > 0 ? uint32_t(end / 2) : 0u;
      x = kLmLower;
      len = 0;
      bad = 0;
      R = (n + 31) / 32;
      round = R - 1;
      const int64_t i = R * W.lane + round;
      if (i < n) bad |= W.in(W.row[cur], sym0 + 256 * i);
    }
    if (!__syncthreads_or(more)) break;
    const int64_t i = R * W.lane + round;
    const bool active = more && i < n;
    float node[kLmHidden];
    lm_coder_node(S, P, B, i, active, T, node);
    uint32_t* row = W.row[cur];
    const uint32_t* prev = W.row[cur ^ 1];
    if (more) {
      if (round == 0) W.fill(W.row[cur ^ 1]);
      else if (i - 1 < n) bad |= W.in(W.row[cur ^ 1], sym0 + 256 * (i - 1));
    }
    for (int st = 127; st >= 0; st--) {
      lm_freq_t F[2];
      whole = lm_step_freqs(S, O, row, prev, st, node, phase, ok, F, kDrill && st == 0 && round == 0);
      if (!whole) break;
      // the decoder takes s then s + 128, so the encoder puts s + 128 first
      uint32_t f[2], cum[2];
      float inv[2];
#pragma unroll
      for (int t = 0; t < 2; t++) {
        uint32_t& word = row[(st >> 4) + 8 * t];
        const int v = int(word >> (2 * (st & 15)) & 3);
        word |= 3u << (2 * (st & 15));   // to the earlier steps' symbols, one that is not coded yet
        f[t] = v == 1 ? F[t].f[1] : v == 2 ? F[t].f[2] : F[t].f[0];
        cum[t] = v == 1 ? F[t].cum[1] : v == 2 ? F[t].cum[2] : 0u;
        inv[t] = __frcp_rn(float(f[t]));
      }
      lm_put_state(x, f[1], inv[1], cum[1], active, words, room, len, below);
      lm_put_state(x, f[0], inv[0], cum[0], active, words, room, len, below);
    }
    if (__syncthreads_or(!ok)) whole = false;   // (the last step's products among them)
    cur ^= 1;
    round--;
  }
  lm_coder_end(S, whole, phase);
}

// status[s] = symbols decoded, or PG_ERR_FORMAT / PG_ERR_CAPACITY; what it was
// before (PG_ERR_CUDA) as in the encoder, and kDrill likewise.  Version-2
// streams are left to the format-2 decoder (and streams too short to carry a
// version, which it rejects).
template<bool kDrill>
__global__ void __launch_bounds__(kLmCodeThreads, kLmCodeCtas)
lm_decode_kernel(const uint16_t* __restrict__ P, uint64_t hash, const lm_block_t* __restrict__ blocks, int nstreams,
                 const int32_t* __restrict__ order, int* __restrict__ next, const uint8_t* __restrict__ in,
                 const int64_t* __restrict__ in_offsets,
                 const int64_t* __restrict__ in_sizes, uint8_t* __restrict__ symbols,
                 const int64_t* __restrict__ sym_offsets, const int64_t* __restrict__ sym_caps,
                 int64_t* __restrict__ status, const dev_tables_t T, const __grid_constant__ lm_const O) {
  extern __shared__ __align__(16) unsigned char lm_smem_raw[];
  lm_warp W;
  lm_coder& S = lm_coder_begin(lm_smem_raw, P, W);
  const bool first = W.lane == 0;
  const unsigned above = W.lane == 31 ? 0u : ~0u << (W.lane + 1);
  int s = -1, cur = 0;
  bool more = true, ok = true, whole = true;
  uint32_t phase = 1;
  int64_t n = 0, R = 0, round = 0;   // R: the run of nodes of each lane
  const uint8_t* words = nullptr;
  uint8_t* out0 = nullptr;
  uint32_t x = kLmLower;
  int64_t ptr = 0;   // words [0, ptr) are unread
  int bad = 0;
  lm_block_t B = {};
  while (whole) {
    while (more && round == R) {
      if (s >= 0) {
        // A well-formed stream ends with every word read and every lane back
        // at the encoder's initial state.
        bad |= x != kLmLower;
        bad = __any_sync(0xffffffffu, bad);
        if (first) status[s] = (bad || ptr != 0) ? PG_ERR_FORMAT : 256 * n;
      }
      s = lm_next_stream(next, order, nstreams, W.lane);
      more = s >= 0;
      if (!more) break;
      const int now = s;
      s = -1;   // (until the stream is known to be one to decode)
      const uint8_t* base = in + in_offsets[now];
      const int64_t size = in_sizes[now];
      if (size < 4) continue;
      const uint32_t version = get32(base);
      if (version == 2) continue;
      B = blocks[now];
      n = B.nodes;
      const uint64_t h = size >= kLmStreamHeader ? uint64_t(get32(base + 4)) | uint64_t(get32(base + 8)) << 32 : 0;
      const uint32_t len = size >= kLmStreamHeader ? get32(base + 16) : 0;
      if (version != kLmVersion || size < kLmStreamHeader || h != hash || get32(base + 12) != uint64_t(n) ||
          int64_t(len) * 2 + kLmStreamHeader != size) {
        if (first) status[now] = PG_ERR_FORMAT;
        continue;
      }
      if (sym_caps[now] < 256 * n) {
        if (first) status[now] = PG_ERR_CAPACITY;
        continue;
      }
      s = now;
      words = base + kLmStreamHeader;
      out0 = symbols + sym_offsets[s];
      x = get32(base + 20 + 4 * W.lane);
      ptr = len;
      bad = 0;
      R = (n + 31) / 32;
      round = 0;
      W.fill(W.row[cur ^ 1]);
    }
    if (!__syncthreads_or(more)) break;
    const int64_t i = R * W.lane + round;
    const bool active = more && i < n;
    float node[kLmHidden];
    lm_coder_node(S, P, B, i, active, T, node);
    uint32_t* row = W.row[cur];
    W.fill(row);
    const uint32_t* prev = W.row[cur ^ 1];   // the previous node of the run is the row of the last round
    // the round's words are the last unread ones: stage up to kLmWordWin of them
    const int64_t wlo = ptr > kLmWordWin ? ptr - kLmWordWin : 0;
    if (more) {
      __syncwarp();
#pragma unroll 4
      for (int64_t w = wlo + W.lane; w < ptr; w += 32) W.win[w - wlo] = get16(words + 2 * w);
      __syncwarp();
    }
    for (int st = 0; st < 128; st++) {
      lm_freq_t F[2];
      whole = lm_step_freqs(S, O, row, prev, st, node, phase, ok, F, kDrill && st == 127 && round == R - 1);
      if (!whole) break;
#pragma unroll
      for (int t = 0; t < 2; t++) {   // (the row's symbols are 3 until they are coded)
        const int v = lm_get_symbol(x, F[t].f[0], F[t].f[1], active, words, W.win, wlo, ptr, above, bad);
        row[(st >> 4) + 8 * t] ^= uint32_t(v ^ 3) << (2 * (st & 15));
      }
    }
    if (__syncthreads_or(!ok)) whole = false;   // (the last step's products among them)
    if (active && whole) W.out(row, out0 + 256 * i);
    cur ^= 1;
    round++;
  }
  lm_coder_end(S, whole, phase);
}

// Frequencies of given samples (for checking the coding path against the CPU).
__global__ void __launch_bounds__(kLmThreads)
lm_freqs_kernel(const uint16_t* __restrict__ P, const lm_block_t* __restrict__ blocks, int nstreams,
                const uint8_t* __restrict__ symbols, const int64_t* __restrict__ offsets,
                const int64_t* __restrict__ samples, int64_t n, uint32_t* __restrict__ freqs, const dev_tables_t T) {
  extern __shared__ __align__(16) unsigned char lm_smem_raw[];
  lm_tables& S = *reinterpret_cast<lm_tables*>(lm_smem_raw);
  lm_build_tables(S, P, threadIdx.x, blockDim.x);
  __syncthreads();
  for (int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; t < n; t += int64_t(gridDim.x) * blockDim.x) {
    const int64_t smp = samples[t];
    const int64_t s = smp >> 24, i = (smp >> 8) & 0xffff;
    const int r = int(smp & 255);
    uint32_t* f = freqs + 3 * t;
    if (s < 0 || s >= nstreams || i >= blocks[s].nodes) { f[0] = f[1] = f[2] = 0; continue; }
    uint8_t feats[36];
    const int nf = lm_load_node(blocks[s], i, T, feats);
    float node[kLmHidden];
    lm_node_sum(S.b1, P, feats, nf, node);
    int u[4];
    const uint8_t* sym = symbols + offsets[s] + 256 * i;
    lm_context_clamped(sym, r, u);
    const int64_t R = (blocks[s].nodes + 31) / 32;   // lanes' runs: the previous node is i - 1 inside a run
    const int prev = i % R ? (sym[r - 256] & 3) : 3;
    float z[3];
    lm_logits(S, node, r, u, prev, z);
    const lm_freq_t F = lm_freqs(z);
    f[0] = F.f[0];
    f[1] = F.f[1];
    f[2] = F.f[2];
  }
}

// The encoder keeps the smaller of the learned and format-2 streams.  The
// format-2 stream is coded first, into its slot, and moved to the slot's end;
// the learned one is coded from the front and drops the words that would reach
// into it (it is then the larger one).
__device__ __forceinline__ void lm_move(uint8_t* to, const uint8_t* from, int64_t n) {   // one CTA; may overlap
  const bool up = to > from;
  for (int64_t done = 0; done < n; done += blockDim.x) {
    const int64_t k = up ? n - 1 - done - threadIdx.x : done + threadIdx.x;
    const bool mine = k >= 0 && k < n;
    const uint8_t v = mine ? from[k] : 0;
    __syncthreads();
    if (mine) to[k] = v;
    __syncthreads();
  }
}
__global__ void lm_aside_kernel(uint8_t* __restrict__ out, const int64_t* __restrict__ out_offsets,
                                const int64_t* __restrict__ caps, const int64_t* __restrict__ alt_sizes,
                                int64_t* __restrict__ sizes) {
  const int64_t b = alt_sizes[blockIdx.x];
  if (threadIdx.x == 0) sizes[blockIdx.x] = PG_ERR_CUDA;   // until the learned coder has been there
  uint8_t* slot = out + out_offsets[blockIdx.x];
  if (b > 0) lm_move(slot + caps[blockIdx.x] - b, slot, b);
}
__global__ void lm_choose_kernel(uint8_t* __restrict__ out, const int64_t* __restrict__ out_offsets,
                                 const int64_t* __restrict__ caps, int64_t* __restrict__ sizes,
                                 const int64_t* __restrict__ alt_sizes) {
  const int s = blockIdx.x;
  const int64_t a = sizes[s], b = alt_sizes[s];
  if (a < 0 || b < 0 || b >= a) return;
  uint8_t* slot = out + out_offsets[s];
  lm_move(slot, slot + caps[s] - b, b);
  if (threadIdx.x == 0) sizes[s] = b;
}

// ---------------------------------------------------------------------------
// Training

// One CTA takes tiles of 224 samples, a warp 16 of them: the largest tile whose
// features, activations and terms fit shared memory beside the weights, as a tile
// costs its barriers and the products over samples whatever it holds.  A batch
// takes the time of its fullest SM: one tile up to 33,152 samples (40 us),
// two from there on.  Every product runs on the tensor
// cores (mma.sync m16n8k16, bf16 inputs, fp32 accumulation): the one-hot
// features, the coding weights and the activations hq / 16 are exact in bf16,
// and the fp32 gradients dL/da2 and dL/da1 enter as three bf16 terms that add
// up to them exactly, so no product is rounded; the products of a step of 16
// samples are summed by the tensor cores and join the rest by rounded fp32
// additions (add_part).  A warp keeps its 16 samples in registers from layer 1
// to dL/da1; the features, activations and gradient terms also lie in shared
// memory, where the products over samples (dW1, dW2) read them transposed.  The
// error against 64 bits is 0.7e-7 of the gradient's norm; one thread per sample
// and fp32 loops over shared memory take 910 us for a batch of 32,768 and have
// 1.0e-7 to 2.1e-7.
constexpr int kGradWarps = 14;
constexpr int kGradThreads = 32 * kGradWarps;
constexpr int kTile = 16 * kGradWarps;
constexpr int kXRow = 136, kHRow = 72;   // elements of a feature row (128 used) and of a hidden row (64): a row of
                                         // either starts 4 banks after the one before, as ldmatrix wants

struct lm_grad_smem {
  uint16_t w1[128][kHRow];         // [feature][hidden], zero from 124 (kOnes) on
  uint16_t w2[kLmHidden][kHRow];   // [hidden][output]
  uint16_t x[kTile][kXRow];        // one-hot features, and 1 at kOnes
  uint16_t h[kTile][kHRow];        // hq / 16
  uint16_t d[3][kTile][kHRow];     // the terms of dL/da2, then of dL/da1
  float b1[kLmHidden], b2[kLmHidden], b3[4];
  float w3[kLmHidden][4];
  float gw3[kGradWarps][kLmOut][kLmHidden];   // dW3 of each warp's samples
  float last[kGradWarps][4];       // their db3 and loss
  int8_t y[kTile];                 // symbol, -1 for a sample that does not count
};
static_assert(sizeof(lm_grad_smem) <= 227 * 1024, "one CTA's shared memory");
constexpr int kOnes = kLmIn;   // this row of the product of features and gradients is the gradient of the biases
constexpr uint16_t kBf16One = 0x3f80;

__device__ __forceinline__ float bf16_of(const float* p, int i) { return bf16_value(bf16_round(p[i])); }

__device__ __forceinline__ void ldsm_x4_t(uint32_t* r, const void* p) {
  const unsigned a = unsigned(__cvta_generic_to_shared(p));
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
// The fragments of a 16 x 16 piece at (r0, c0) of a row-major table: as A;
// as A of the transposed table (rows of the product are columns c0 ..); as B
// for two n-tiles, of the table with k along its rows; as B with n along them.
template<int ROW> __device__ __forceinline__ void frag_a(uint32_t* a, const uint16_t (*t)[ROW], int r0, int c0, int lane) {
  ldsm_x4(a, &t[r0 + (lane & 15)][c0 + 8 * (lane >> 4)]);
}
template<int ROW> __device__ __forceinline__ void frag_at(uint32_t* a, const uint16_t (*t)[ROW], int r0, int c0, int lane) {
  ldsm_x4_t(a, &t[r0 + (lane & 7) + 8 * (lane >> 4)][c0 + (lane & 8)]);
}
template<int ROW> __device__ __forceinline__ void frag_bk(uint32_t* b, const uint16_t (*t)[ROW], int r0, int c0, int lane) {
  ldsm_x4_t(b, &t[r0 + (lane & 15)][c0 + 8 * (lane >> 4)]);
}
template<int ROW> __device__ __forceinline__ void frag_bn(uint32_t* b, const uint16_t (*t)[ROW], int r0, int c0, int lane) {
  ldsm_x4(b, &t[r0 + (lane & 7) + 8 * (lane >> 4)][c0 + (lane & 8)]);
}

// v = term 0 + term 1 + term 2, bf16 each, exactly (8 bits of v's 24 each),
// for two values packed per word; |v| < kSplitMost.
constexpr float kSplitMost = 3.38e38f;   // (what is not below may round to an infinity)
__device__ __forceinline__ uint32_t bf16_pair(float v0, float v1) {   // rounded to nearest even; NaN stays NaN
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(v1), "f"(v0));
  return d;
}
__device__ __forceinline__ void split3(float v0, float v1, uint32_t* term) {
#pragma unroll
  for (int s = 0; s < 3; s++) {
    term[s] = bf16_pair(v0, v1);
    v0 = f_add(v0, -f_bits(term[s] << 16));
    v1 = f_add(v1, -f_bits(term[s] & 0xffff0000u));
  }
}
// The same of any values: of a large one the first term is cut, of an infinity or
// NaN it is that and the others 0.
__device__ __forceinline__ float split_first(float v, float& rest) {
  const uint32_t u = f_raw(v) & 0xffff0000u;
  const float first = v == v ? f_bits(u) : f_bits(0x7fff0000u);
  rest = f_finite(v) ? f_add(v, -first) : 0.f;
  return first;
}
__device__ __forceinline__ void split3_any(float v0, float v1, uint32_t* term) {
  float r0, r1;
  const float f0 = split_first(v0, r0), f1 = split_first(v1, r1);
  term[0] = f_raw(f0) >> 16 | (f_raw(f1) & 0xffff0000u);
  uint32_t more[3];
  split3(r0, r1, more);   // (16 bits are left: two terms)
  term[1] = more[0];
  term[2] = more[1];
}
__device__ __forceinline__ float most_of(float m, float v) {   // max(m, |v|), NaN if either is
  float d;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(m), "f"(fabsf(v)));
  return d;
}

// The coding weights in bf16: stone rows and biases rounded, W1's rotation,
// neighbour and previous-node rows and W2 on their column grids, as the
// exported model holds them (lm_grid_params).  Thread (column, quarter) finds
// its quarter's largest magnitude, then moves its rows onto the column's grid.
// Returns (to all threads) whether the stone rows are finite (the others are, on
// their grids); weights that are not are 0 here, and lm_odd_stones has them.
__device__ __forceinline__ bool lm_grad_weights(lm_grad_smem& G, const float* __restrict__ params, int tid) {
  bool finite = true;
  for (int i = tid; i < kLmRot * kLmHidden; i += kGradThreads) {
    const uint16_t w = bf16_round(params[kLmW1 + i]);
    const bool number = f_finite(bf16_value(w));
    finite &= number;
    G.w1[i / kLmHidden][i % kLmHidden] = number ? w : uint16_t(0);
  }
  for (int i = tid; i < (128 - kLmIn) * kLmHidden; i += kGradThreads) G.w1[kLmIn + i / kLmHidden][i % kLmHidden] = 0;
  if (tid < kLmHidden) {
    G.b1[tid] = bf16_of(params, kLmB1 + tid);
    G.b2[tid] = bf16_of(params, kLmB2 + tid);
    for (int c = 0; c < 3; c++) G.w3[tid][c] = bf16_of(params, kLmW3 + tid * kLmOut + c);
    G.w3[tid][3] = 0.f;
  }
  if (tid < 4) G.b3[tid] = tid < 3 ? bf16_of(params, kLmB3 + tid) : 0.f;
  constexpr int kA = kLmCtxRows / 4, kB = kLmHidden / 4;
  static_assert(kA * 4 == kLmCtxRows, "quarters of the context rows");
  const int col = tid & (kLmHidden - 1), part = tid / kLmHidden;
  float (*top)[2 * kLmHidden] = reinterpret_cast<float (*)[2 * kLmHidden]>(&G.d[0][0][0]);   // column maxima
  float a[kA], b[kB];
  if (part < 4) {
    float ma = 0.f, mb = 0.f;
#pragma unroll
    for (int i = 0; i < kA; i++) {
      a[i] = params[kLmW1 + (kLmRot + kA * part + i) * kLmHidden + col];
      ma = fmaxf(ma, fabsf(a[i]));
    }
#pragma unroll
    for (int i = 0; i < kB; i++) {
      b[i] = params[kLmW2 + (kB * part + i) * kLmHidden + col];
      mb = fmaxf(mb, fabsf(b[i]));
    }
    top[part][col] = ma;
    top[part][kLmHidden + col] = mb;
  }
  finite = __syncthreads_and(finite);
  if (part < 4) {
    auto most = [&](int c) { return fmaxf(fmaxf(top[0][c], top[1][c]), fmaxf(top[2][c], top[3][c])); };
    const float ma = most(col), mb = most(kLmHidden + col);
    const int ea = ma > 0.f ? lm_grid_exp(ma) : 0, eb = mb > 0.f ? lm_grid_exp(mb) : 0;
#pragma unroll
    for (int i = 0; i < kA; i++)
      G.w1[kLmRot + kA * part + i][col] = ma > 0.f ? bf16_round(lm_grid_quantize(a[i], ea)) : 0;
#pragma unroll
    for (int i = 0; i < kB; i++) G.w2[kB * part + i][col] = mb > 0.f ? bf16_round(lm_grid_quantize(b[i], eb)) : 0;
  }
  return finite;
}

// Units of the products over samples: 16 x 16 pieces of dW1 (rows 0..127, db1
// in row kOnes) and of dW2 (and, below it, of the last 16 features with
// dL/da2, for db2 in row kOnes), handed to the warps in turn.
constexpr int kUnits1 = 8 * 4, kUnits2 = 5 * 4;
constexpr int kMine1 = (kUnits1 + kGradWarps - 1) / kGradWarps, kMine2 = (kUnits2 + kGradWarps - 1) / kGradWarps;

// A step's products join the sum by rounded additions: the tensor cores'
// own accumulation drops the bits below the sum's last place, which over many
// steps made the gradient's error against 64 bits 3.9e-7 of its norm; so it is
// 0.7e-7 (batches of 5,000 and 32,768), with fp32 loops over the samples
// 1.0e-7 and 2.1e-7.
__device__ __forceinline__ void add_part(float* acc, const float* part) {
#pragma unroll
  for (int i = 0; i < 4; i++) acc[i] = f_add(acc[i], part[i]);
}
// acc += (A^T D) at (r0, c0): A the features or activations of the tile's
// samples, D the sum of the three gradient terms.
template<int ROW>
__device__ __forceinline__ void sample_product(float (*acc)[4], const uint16_t (*A)[ROW],
                                               const uint16_t (*D)[kTile][kHRow], int r0, int c0, int lane) {
#pragma unroll 2
  for (int k = 0; k < kTile; k += 16) {
    uint32_t a[4];
    frag_at(a, A, k, r0, lane);
    float part[2][4] = {};
#pragma unroll
    for (int s = 2; s >= 0; s--) {
      uint32_t b[4];
      frag_bk(b, D[s], k, c0, lane);
      mma_bf16(part[0], a, b[0], b[1]);
      mma_bf16(part[1], a, b[2], b[3]);
    }
    add_part(acc[0], part[0]);
    add_part(acc[1], part[1]);
  }
}

// A product with the features multiplies all of a column by a sample's 0s and
// 1s, and 0 times an infinity is NaN, so what is not finite goes around the
// products: it reaches a sample from its own features, and their rows from it.

// The sums of those stone weights over the samples of the warp's 16 rows, into
// the place of the gradient terms (not in use yet): [row][hidden].
__device__ __noinline__ void lm_odd_stones(lm_grad_smem& G, const float* __restrict__ params, int row0, int lane) {
  float* sums = reinterpret_cast<float*>(&G.d[0][0][0]) + row0 * kLmHidden;
  for (int i = lane; i < 16 * kLmHidden; i += 32) {
    const int row = row0 + i / kLmHidden, k = i % kLmHidden;
    float s = 0.f;
    for (int f = 0; f < kLmRot; f++) {
      const float w = bf16_of(params, kLmW1 + f * kLmHidden + k);
      if (G.x[row][f] && !f_finite(w)) s += w;
    }
    sums[i] = s;
  }
  __syncwarp();
}
// dL/da1 of a sample's hidden unit k to the rows of its features and to the
// bias, in the CTA's partial sums (whichever order they come in, sums of
// infinities and NaN are the same).
__device__ __noinline__ void lm_odd_gradient(const lm_grad_smem& G, float* out, int row, int k, float v) {
  for (int f = 0; f <= kOnes; f++)
    if (G.x[row][f]) atomicAdd(out + (f < kOnes ? kLmW1 + f * kLmHidden + k : kLmB1 + k), v);
}

__global__ void __launch_bounds__(kGradThreads)
lm_grad_kernel(const float* __restrict__ params, const lm_block_t* __restrict__ blocks, int nstreams,
               const uint8_t* __restrict__ symbols, const int64_t* __restrict__ offsets,
               const int64_t* __restrict__ samples, int64_t n, float* __restrict__ partial, const dev_tables_t T) {
  extern __shared__ __align__(16) unsigned char lm_smem_raw[];
  lm_grad_smem& G = *reinterpret_cast<lm_grad_smem*>(lm_smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const bool finite_stones = lm_grad_weights(G, params, tid);
  for (int i = lane; i < kLmOut * kLmHidden; i += 32) (&G.gw3[warp][0][0])[i] = 0.f;
  float g1[kMine1][2][4] = {}, g2[kMine2][2][4] = {};   // this warp's units of dW1 and dW2
  float gb3[3] = {}, gloss = 0.f;                       // this lane's rows
  auto over_quads = [&](float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 8);
    return v + __shfl_xor_sync(0xffffffffu, v, 16);
  };
  float* out = partial + int64_t(blockIdx.x) * (kLmParams + 1);
  bool odd = false;   // out has what is not finite of dW1 and db1
  const int64_t tiles = (n + kTile - 1) / kTile;
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    // Features: thread 2 s sets the stones of sample s, thread 2 s + 1 the rest
    {
      uint4* x = reinterpret_cast<uint4*>(&G.x[0][0]);
      for (int i = tid; i < kTile * kXRow / 8; i += kGradThreads) x[i] = make_uint4(0, 0, 0, 0);
      __syncthreads();
      const int row = tid >> 1;
      const int64_t k = tile * kTile + row;
      int y = -1;
      if (k < n) {
        const int64_t smp = samples[k];
        const int64_t s = smp >> 24, i = (smp >> 8) & 0xffff;
        const int r = int(smp & 255);
        if (s >= 0 && s < nstreams && i < blocks[s].nodes) {
          const uint8_t* sym = symbols + offsets[s] + 256 * i;
          y = sym[r] <= 2 ? sym[r] : -1;
          if (y >= 0 && !(tid & 1)) {
            uint16_t qid[4];
            lm_node_quadrants(blocks[s], i, T.rmin_flat, qid);
#pragma unroll
            for (int q = 0; q < 4; q++)
#pragma unroll
              for (int c = 0; c < 2; c++)
                for (uint32_t m = T.unpack[2 * qid[q] + c]; m; m &= m - 1)
                  G.x[row][18 * q + 2 * (__ffs(m) - 1) + c] = kBf16One;
          } else if (y >= 0) {
            uint32_t v[8];
#pragma unroll
            for (int nb = 0; nb < 8; nb++) {
              const int a = lm_neighbour(r, nb);
              v[nb] = lm_before(a, r) ? sym[a] & 3 : 3;
            }
            const int64_t R = (blocks[s].nodes + 31) / 32;   // the coder's runs of nodes
            const int prev = i % R ? (sym[r - 256] & 3) : 3;
#pragma unroll
            for (int q = 0; q < 4; q++) G.x[row][kLmRot + 4 * q + ((r >> (2 * q)) & 3)] = kBf16One;
#pragma unroll
            for (int nb = 0; nb < 8; nb++) G.x[row][kLmCtx + 4 * nb + v[nb]] = kBf16One;
            G.x[row][kLmPrev + prev] = kBf16One;
          }
        }
      }
      if (tid & 1) {
        G.y[row] = int8_t(y);
        G.x[row][kOnes] = kBf16One;
      }
    }
    __syncthreads();
    // Layer 1: rows 16 warp + g and + 8
    const int row0 = 16 * warp;
    float acc[8][4] = {};
#pragma unroll 2
    for (int kt = 0; kt < 8; kt++) {
      uint32_t a[4];
      frag_a(a, G.x, row0, 16 * kt, lane);
#pragma unroll
      for (int np = 0; np < 4; np++) {
        uint32_t b[4];
        frag_bk(b, G.w1, 16 * kt, 16 * np, lane);
        float part[2][4] = {};
        mma_bf16(part[0], a, b[0], b[1]);
        mma_bf16(part[1], a, b[2], b[3]);
        add_part(acc[2 * np], part[0]);
        add_part(acc[2 * np + 1], part[1]);
      }
    }
    if (!finite_stones) {
      lm_odd_stones(G, params, row0, lane);
      const float* sums = reinterpret_cast<const float*>(&G.d[0][0][0]) + row0 * kLmHidden;
#pragma unroll
      for (int nt = 0; nt < 8; nt++)
#pragma unroll
        for (int i = 0; i < 4; i++) acc[nt][i] += sums[(g + 8 * (i >> 1)) * kLmHidden + 8 * nt + 2 * t + (i & 1)];
      __syncthreads();   // (before the terms are written there)
    }
    // The activations hq / 16, packed as layer 2's A operand
    uint32_t h[4][4];
#pragma unroll
    for (int nt = 0; nt < 8; nt++) {
      const float2 b1 = *reinterpret_cast<const float2*>(&G.b1[8 * nt + 2 * t]);
#pragma unroll
      for (int half = 0; half < 2; half++) {
        const float q0 = f_mul(lm_act_q(f_add(b1.x, acc[nt][2 * half])), kLmActInv);
        const float q1 = f_mul(lm_act_q(f_add(b1.y, acc[nt][2 * half + 1])), kLmActInv);
        const uint32_t w = __byte_perm(f_raw(q0), f_raw(q1), 0x7632);
        h[nt >> 1][2 * (nt & 1) + half] = w;
        *reinterpret_cast<uint32_t*>(&G.h[row0 + g + 8 * half][8 * nt + 2 * t]) = w;
      }
    }
    // Layer 2 (its sums are exact on the grid, so a2 = b2 + sum rounds once)
#pragma unroll
    for (int nt = 0; nt < 8; nt++) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
#pragma unroll
    for (int kt = 0; kt < 4; kt++)
#pragma unroll
      for (int np = 0; np < 4; np++) {
        uint32_t b[4];
        frag_bk(b, G.w2, 16 * kt, 16 * np, lane);
        mma_bf16(acc[2 * np], h[kt], b[0], b[1]);
        mma_bf16(acc[2 * np + 1], h[kt], b[2], b[3]);
      }
    // Layer 3, the loss and dL/dz of the two rows (every lane of a quad holds
    // both); nothing of a row that does not count, whatever the weights are
    float z[2][3] = {};
    const int ys[2] = {G.y[row0 + g], G.y[row0 + g + 8]};
#pragma unroll
    for (int nt = 0; nt < 8; nt++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int j = 8 * nt + 2 * t + e;
        const float4 w3 = *reinterpret_cast<const float4*>(G.w3[j]);
#pragma unroll
        for (int half = 0; half < 2; half++) {
          const float a2 = ys[half] >= 0 ? f_add(G.b2[j], acc[nt][2 * half + e]) : 0.f;
          acc[nt][2 * half + e] = a2;
          const float r = relu(a2);
          z[half][0] = fmaf(w3.x, r, z[half][0]);
          z[half][1] = fmaf(w3.y, r, z[half][1]);
          z[half][2] = fmaf(w3.z, r, z[half][2]);
        }
      }
    float dz[2][3];
#pragma unroll
    for (int half = 0; half < 2; half++) {
#pragma unroll
      for (int c = 0; c < 3; c++) {
        z[half][c] += __shfl_xor_sync(0xffffffffu, z[half][c], 1);
        z[half][c] += __shfl_xor_sync(0xffffffffu, z[half][c], 2);
        z[half][c] += G.b3[c];
      }
      const int y = ys[half];
      const float m = fmaxf(z[half][0], fmaxf(z[half][1], z[half][2]));
      float e[3], es = 0.f;
#pragma unroll
      for (int c = 0; c < 3; c++) { e[c] = expf(z[half][c] - m); es += e[c]; }
      const float zy = y == 0 ? z[half][0] : y == 1 ? z[half][1] : z[half][2];
      if (y >= 0 && t == 0) gloss += (logf(es) - (zy - m)) * 1.44269504f;  // bits
#pragma unroll
      for (int c = 0; c < 3; c++) {
        dz[half][c] = y >= 0 ? e[c] / es - (c == y ? 1.f : 0.f) : 0.f;
        if (t == 0) gb3[c] += dz[half][c];
      }
    }
    // dW3, and dL/da2 in its terms
    auto d2_at = [&](int nt, int half, int e) {
      const float4 w3 = *reinterpret_cast<const float4*>(G.w3[8 * nt + 2 * t + e]);
      return acc[nt][2 * half + e] > 0.f ? w3.x * dz[half][0] + w3.y * dz[half][1] + w3.z * dz[half][2] : 0.f;
    };
    auto put_terms = [&](int nt, int half, const uint32_t* w) {
#pragma unroll
      for (int s = 0; s < 3; s++) *reinterpret_cast<uint32_t*>(&G.d[s][row0 + g + 8 * half][8 * nt + 2 * t]) = w[s];
    };
    float most = 0.f;
#pragma unroll
    for (int nt = 0; nt < 8; nt++) {
#pragma unroll
      for (int e = 0; e < 2; e++) {
        float v[3] = {};
#pragma unroll
        for (int half = 0; half < 2; half++) {
          const float r = relu(acc[nt][2 * half + e]);
#pragma unroll
          for (int c = 0; c < 3; c++) v[c] = fmaf(r, dz[half][c], v[c]);
        }
#pragma unroll
        for (int c = 0; c < 3; c++) {
          v[c] = over_quads(v[c]);
          if (g == 0) G.gw3[warp][c][8 * nt + 2 * t + e] += v[c];
        }
      }
#pragma unroll
      for (int half = 0; half < 2; half++) {
        const float d0 = d2_at(nt, half, 0), d1 = d2_at(nt, half, 1);
        most = most_of(most_of(most, d0), d1);
        uint32_t w[3];
        split3(d0, d1, w);
        put_terms(nt, half, w);
      }
    }
    if (!(most < kSplitMost)) {
#pragma unroll
      for (int nt = 0; nt < 8; nt++)
#pragma unroll
        for (int half = 0; half < 2; half++) {
          uint32_t w[3];
          split3_any(d2_at(nt, half, 0), d2_at(nt, half, 1), w);
          put_terms(nt, half, w);
        }
    }
    __syncwarp();
    // dL/da1 = dL/da2 W2^T where the quantizer passes the gradient straight
    // through: the activation is neither cut by relu nor clamped at the top
#pragma unroll
    for (int nt = 0; nt < 8; nt++) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
#pragma unroll 2
    for (int kt = 0; kt < 4; kt++) {
      uint32_t a[3][4];
#pragma unroll
      for (int s = 0; s < 3; s++) frag_a(a[s], G.d[s], row0, 16 * kt, lane);
#pragma unroll
      for (int np = 0; np < 4; np++) {
        uint32_t b[4];
        frag_bn(b, G.w2, 16 * np, 16 * kt, lane);
        float part[2][4] = {};
#pragma unroll
        for (int s = 2; s >= 0; s--) {
          mma_bf16(part[0], a[s], b[0], b[1]);
          mma_bf16(part[1], a[s], b[2], b[3]);
        }
        add_part(acc[2 * np], part[0]);
        add_part(acc[2 * np + 1], part[1]);
      }
    }
#pragma unroll
    for (int nt = 0; nt < 8; nt++)
#pragma unroll
      for (int e = 0; e < 2; e++)
#pragma unroll
        for (int half = 0; half < 2; half++) {
          const float a = f_bits(e ? h[nt >> 1][2 * (nt & 1) + half] & 0xffff0000u : h[nt >> 1][2 * (nt & 1) + half] << 16);
          float& d = acc[nt][2 * half + e];
          d = a > 0.f && a < kLmActMax * kLmActInv ? d : 0.f;
        }
    __syncthreads();
    // dW2 from every sample's activations and dL/da2
#pragma unroll
    for (int u = 0; u < kMine2; u++) {
      const int unit = warp + kGradWarps * u;
      if (unit < 16) sample_product(g2[u], G.h, G.d, 16 * (unit >> 2), 16 * (unit & 3), lane);
      else if (unit < kUnits2) sample_product(g2[u], G.x, G.d, 112, 16 * (unit & 3), lane);
    }
    most = 0.f;
#pragma unroll
    for (int nt = 0; nt < 8; nt++)
#pragma unroll
      for (int i = 0; i < 4; i++) most = most_of(most, acc[nt][i]);
    // dW1 from their features and dL/da1
    if (!__syncthreads_or(!(most < kSplitMost))) {
#pragma unroll
      for (int nt = 0; nt < 8; nt++)
#pragma unroll
        for (int half = 0; half < 2; half++) {
          uint32_t w[3];
          split3(acc[nt][2 * half], acc[nt][2 * half + 1], w);
          put_terms(nt, half, w);
        }
    } else {
      if (!odd) {
        for (int i = tid; i < kLmW2; i += kGradThreads) __stcg(out + i, 0.f);
        __threadfence();
        __syncthreads();
      }
      odd = true;
#pragma unroll
      for (int nt = 0; nt < 8; nt++)
#pragma unroll
        for (int half = 0; half < 2; half++) {
#pragma unroll
          for (int e = 0; e < 2; e++) {
            float& d = acc[nt][2 * half + e];
            if (f_finite(d)) continue;
            lm_odd_gradient(G, out, row0 + g + 8 * half, 8 * nt + 2 * t + e, d);
            d = 0.f;
          }
          uint32_t w[3];
          split3_any(acc[nt][2 * half], acc[nt][2 * half + 1], w);
          put_terms(nt, half, w);
        }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kMine1; u++) {
      const int unit = warp + kGradWarps * u;
      if (unit < kUnits1) sample_product(g1[u], G.x, G.d, 16 * (unit >> 2), 16 * (unit & 3), lane);
    }
    __syncthreads();
  }
  // Partial sums of this CTA: the units of dW1 and dW2 (with the biases'
  // rows), then the warps' sums, in order.
  // Rows r0 .. of a unit at columns c0 ..: row `last` to out + bias, those
  // before it to out + base
  auto put = [&](const float (*acc)[4], int base, int r0, int c0, int last, int bias) {
#pragma unroll
    for (int nt = 0; nt < 2; nt++)
#pragma unroll
      for (int half = 0; half < 2; half++) {
        const int r = r0 + g + 8 * half, c = c0 + 8 * nt + 2 * t;
        float* o = r < last ? out + base + r * kLmHidden + c : out + bias + c;
        if (r > last) continue;
        const bool add = odd && base == kLmW1;
        o[0] = acc[nt][2 * half] + (add ? __ldcg(o) : 0.f);
        o[1] = acc[nt][2 * half + 1] + (add ? __ldcg(o + 1) : 0.f);
      }
  };
#pragma unroll
  for (int u = 0; u < kMine1; u++) {
    const int unit = warp + kGradWarps * u;
    if (unit < kUnits1) put(g1[u], kLmW1, 16 * (unit >> 2), 16 * (unit & 3), kOnes, kLmB1);
  }
#pragma unroll
  for (int u = 0; u < kMine2; u++) {
    // (the last four units hold rows 112 .. of the features: db2 is row kOnes)
    const int unit = warp + kGradWarps * u;
    if (unit < 16) put(g2[u], kLmW2, 16 * (unit >> 2), 16 * (unit & 3), kLmHidden, kLmB2);
    else if (unit < kUnits2 && g == kOnes - 112 - 8) {
#pragma unroll
      for (int nt = 0; nt < 2; nt++) {
        float* o = out + kLmB2 + 16 * (unit & 3) + 8 * nt + 2 * t;
        o[0] = g2[u][nt][2];
        o[1] = g2[u][nt][3];
      }
    }
  }
#pragma unroll
  for (int c = 0; c < 4; c++) {
    const float v = over_quads(c < 3 ? gb3[c < 3 ? c : 0] : gloss);
    if (lane == 0) G.last[warp][c] = v;
  }
  __syncthreads();
  if (tid < kLmOut * kLmHidden + 4) {
    const int q = tid / kLmHidden, j = tid % kLmHidden;
    float s = 0.f;
    for (int w = 0; w < kGradWarps; w++) s += q < kLmOut ? G.gw3[w][q][j] : G.last[w][j];
    out[q < kLmOut ? kLmW3 + j * kLmOut + q : j < 3 ? kLmB3 + j : kLmParams] = s;
  }
}

// The CTAs' partial sums, added in a fixed order: eight threads to a
// parameter, each an eighth of the CTAs, then the eight: 3.7 us (5.8 with one
// thread to a parameter).
constexpr int kReduceParts = 8;
__global__ void __launch_bounds__(256)
lm_reduce_kernel(const float* __restrict__ partial, int nparts, float* __restrict__ grad, float* __restrict__ loss) {
  constexpr int kCols = 256 / kReduceParts;
  __shared__ float sum[kReduceParts][kCols];
  const int col = threadIdx.x % kCols, part = threadIdx.x / kCols, p = blockIdx.x * kCols + col;
  float s = 0.f;
  if (p <= kLmParams) {
#pragma unroll 8
    for (int c = part; c < nparts; c += kReduceParts) s += partial[int64_t(c) * (kLmParams + 1) + p];
  }
  sum[part][col] = s;
  __syncthreads();
  if (part || p > kLmParams) return;
  for (int q = 1; q < kReduceParts; q++) s += sum[q][col];
  if (p < kLmParams) grad[p] = s;
  else if (loss) *loss = s;
}

__global__ void lm_adam_kernel(float* __restrict__ params, float* __restrict__ m, float* __restrict__ v,
                               const float* __restrict__ grad, float lr, float scale, float c1, float c2) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= kLmParams) return;
  const float g = grad[p] * scale;
  const float mm = 0.9f * m[p] + 0.1f * g;
  const float vv = 0.999f * v[p] + 0.001f * g * g;
  m[p] = mm;
  v[p] = vv;
  params[p] -= lr * (mm / c1) / (sqrtf(vv / c2) + 1e-8f);
}

__device__ __forceinline__ uint64_t splitmix(uint64_t z) {
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

__global__ void lm_samples_kernel(const int64_t* __restrict__ cand, int64_t ncand, uint64_t seed, int64_t step,
                                  int64_t batch, int64_t* __restrict__ out) {
  const int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (k >= batch) return;
  const uint64_t h = splitmix(seed ^ splitmix(uint64_t(step) * 0x100000001b3ull + uint64_t(k)));
  const int64_t c = cand[(h & 0xffffffffffull) % uint64_t(ncand)];
  out[k] = (c << 8) | int64_t(h >> 56);
}

// ---------------------------------------------------------------------------
// Host side

static uint64_t fnv1a(const uint8_t* p, int64_t n) {
  uint64_t h = 0xcbf29ce484222325ull;
  for (int64_t i = 0; i < n; i++) h = (h ^ p[i]) * 0x100000001b3ull;
  return h;
}

static bool check_model(const uint8_t* model, std::string& err) {
  if (!model) { err = "null model"; return false; }
  uint32_t h[3];
  memcpy(h, model, 12);
  if (h[0] != kLmMagic || h[1] != kLmModelVersion || h[2] != uint32_t(kLmParams)) {
    err = "not a version-3 PGLM model";
    return false;
  }
  // W1's rotation and neighbour rows and W2 must lie on their column grids,
  // or the tensor cores' sums would not be exact
  std::vector<float> w(kLmParams), q;
  for (int i = 0; i < kLmParams; i++) {
    const int b = kLmModelHeader + 2 * i;
    w[i] = bf16_value(uint16_t(model[b] | model[b + 1] << 8));
    if (!std::isfinite(w[i])) { err = "non-finite parameter " + std::to_string(i); return false; }
  }
  q = w;
  lm_grid_params(q.data());
  for (int i = 0; i < kLmParams; i++)
    if (q[i] != w[i]) { err = "parameter " + std::to_string(i) + " is not on its grid"; return false; }
  return true;
}

static bool resolve_blocks(const pg_block_ref_t* refs, int n, std::vector<lm_block_t>& out, std::string& err) {
  const auto& T = tables();
  out.resize(n);
  int off[4], size[4];   // of the section's quadrants (blocks of one section come together)
  for (int s = 0; s < n; s++) {
    if (!s || refs[s].section != refs[s - 1].section) {
      const section_t sec = section_t::from_sig(refs[s].section);
      if (!sec.valid() || sec.sum() > 36) { err = "invalid section in block " + std::to_string(s); return false; }
      for (int q = 0; q < 4; q++) {
        const int k = rmin_bucket(sec.c[q][0], sec.c[q][1]);
        off[q] = T.rmin_off[k];
        size[q] = T.rmin_off[k + 1] - T.rmin_off[k];
      }
    }
    lm_block_t& B = out[s];
    B.nodes = 1;
    for (int q = 0; q < 4; q++) {
      const int b = refs[s].block[q];
      if (b < 0 || 8 * b >= size[q]) { err = "block out of range in block " + std::to_string(s); return false; }
      B.qbase[q] = off[q] + 8 * b;
      B.shape[q] = std::min(8, size[q] - 8 * b);
      B.nodes *= B.shape[q];
    }
  }
  return true;
}

struct lm_launch {
  uint16_t* params = nullptr;
  lm_block_t* blocks = nullptr;
  int32_t* order = nullptr;   // streams by node count, largest first (after the blocks)
  int* next = nullptr;        // the coding kernels' stream counter, zeroed (after the order)
  uint64_t hash = 0;
  cudaStream_t stream = nullptr;
  ~lm_launch() {
    if (params) cudaFreeAsync(params, stream);
    if (blocks) cudaFreeAsync(blocks, stream);
  }
};

static int lm_prepare(const uint8_t* model, const pg_block_ref_t* refs, int n, cudaStream_t stream, lm_launch& L,
                      std::vector<lm_block_t>* host_blocks = nullptr) {
  std::string err;
  L.stream = stream;
  if (model) {
    if (!check_model(model, err)) return fail(PG_ERR_FORMAT, err);
    L.hash = fnv1a(model, kLmModelBytes);
    PG_CUDA(cudaMallocAsync(&L.params, 2 * kLmParams, stream));
    PG_CUDA(cudaMemcpyAsync(L.params, model + kLmModelHeader, 2 * kLmParams, cudaMemcpyHostToDevice, stream));
  }
  std::vector<lm_block_t> B;
  if (!resolve_blocks(refs, n, B, err)) return fail(PG_ERR_ARG, err);
  // One buffer: the blocks, and for the coder the processing order and the counter
  const size_t bb = sizeof(lm_block_t) * std::max(n, 1), ob = (sizeof(int32_t) * std::max(n, 1) + 15) & ~size_t(15);
  char* buf = nullptr;
  PG_CUDA(cudaMallocAsync(&buf, bb + ob + 16, stream));
  L.blocks = reinterpret_cast<lm_block_t*>(buf);
  L.order = reinterpret_cast<int32_t*>(buf + bb);
  L.next = reinterpret_cast<int*>(buf + bb + ob);
  PG_CUDA(cudaMemcpyAsync(L.blocks, B.data(), sizeof(lm_block_t) * n, cudaMemcpyHostToDevice, stream));
  if (model) {
    std::vector<int32_t> order(n);
    for (int s = 0; s < n; s++) order[s] = s;
    std::stable_sort(order.begin(), order.end(), [&](int32_t a, int32_t b) { return B[a].nodes > B[b].nodes; });
    PG_CUDA(cudaMemcpyAsync(L.order, order.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice, stream));
    PG_CUDA(cudaMemsetAsync(L.next, 0, sizeof(int), stream));
  }
  if (host_blocks) *host_blocks = std::move(B);
  return PG_OK;
}

template<class K> static int lm_smem_opt_in(K kernel, size_t bytes) {
  PG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes)));
  return PG_OK;
}

// The coding kernels: as many CTAs as are resident at once (the streams are
// handed out dynamically), no more than there are streams for.  kLmCodeCtas
// fit an SM by their launch bounds, shared and tensor memory; the occupancy
// query answers 1 for any kernel that allocates tensor memory.
static int lm_code_grid(int nstreams) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return std::max(1, std::min((nstreams + 3) / 4, kLmCodeCtas * sms));
}

}  // namespace pg

using namespace pg;

extern "C" int64_t pg_learned_model_bytes(void) { return kLmModelBytes; }

extern "C" int64_t pg_rans_learned_bound(int64_t nodes) {
  if (nodes < 0 || nodes > (int64_t(1) << 32)) return PG_ERR_ARG;
  return std::max<int64_t>(kLmStreamHeader + 2 * 256 * nodes, rans_stream_bound(256 * nodes));
}

extern "C" int pg_learned_export(const float* params, uint8_t* model) {
  if (!params || !model) return fail(PG_ERR_ARG, "null argument");
  const uint32_t h[3] = {kLmMagic, kLmModelVersion, uint32_t(kLmParams)};
  memcpy(model, h, 12);
  std::vector<float> p(params, params + kLmParams);
  for (int i = 0; i < kLmParams; i++)
    if (!std::isfinite(p[i])) return fail(PG_ERR_ARG, "non-finite parameter " + std::to_string(i));
  lm_grid_params(p.data());
  for (int i = 0; i < kLmParams; i++) {
    const uint16_t b = bf16_round(p[i]);
    model[kLmModelHeader + 2 * i] = uint8_t(b);
    model[kLmModelHeader + 2 * i + 1] = uint8_t(b >> 8);
  }
  return PG_OK;
}

template<bool kDrill>
static int learned_encode(const uint8_t* model, const pg_block_ref_t* blocks, int nstreams,
                          const uint8_t* symbols, const int64_t* offsets, uint8_t* out, const int64_t* out_offsets,
                          int64_t* sizes, void* stream) {
  if (nstreams < 0 || (nstreams && !blocks)) return fail(PG_ERR_ARG, "bad stream list");
  if (!nstreams) return PG_OK;
  if (!model) return fail(PG_ERR_ARG, "null model");
  const cudaStream_t st = (cudaStream_t)stream;
  const dev_tables_t* T = device_tables();
  if (!T) return PG_ERR_CUDA;
  lm_launch L;
  std::vector<lm_block_t> hb;
  if (int rc = lm_prepare(model, blocks, nstreams, st, L, &hb)) return rc;
  if (int rc = lm_smem_opt_in(lm_encode_kernel<kDrill>, kLmCodeSmem)) return rc;
  // What every slot has room for, and its stream's symbol count; then the sizes of the format-2 streams
  std::vector<int64_t> slots(2 * size_t(nstreams));
  for (int s = 0; s < nstreams; s++) {
    slots[s] = pg_rans_learned_bound(hb[s].nodes);
    slots[size_t(nstreams) + s] = 256 * hb[s].nodes;
  }
  stream_scratch X(st);
  int64_t* caps = nullptr;
  PG_CUDA(X.alloc(&caps, sizeof(int64_t) * 3 * nstreams));
  int64_t* alt_sizes = caps + 2 * size_t(nstreams);
  PG_CUDA(cudaMemcpyAsync(caps, slots.data(), sizeof(int64_t) * 2 * nstreams, cudaMemcpyHostToDevice, st));
  if (int rc = launch_rans_encode(symbols, offsets, nstreams, out, out_offsets, alt_sizes, caps + nstreams, st)) return rc;
  lm_aside_kernel<<<nstreams, 256, 0, st>>>(out, out_offsets, caps, alt_sizes, sizes);
  PG_CUDA(cudaGetLastError());
  lm_encode_kernel<kDrill><<<lm_code_grid(nstreams), kLmCodeThreads, kLmCodeSmem, st>>>(
      L.params, L.hash, L.blocks, nstreams, L.order, L.next, symbols, offsets, out, out_offsets, caps, alt_sizes, sizes, *T,
      lm_consts(model));
  PG_CUDA(cudaGetLastError());
  lm_choose_kernel<<<nstreams, 256, 0, st>>>(out, out_offsets, caps, sizes, alt_sizes);
  PG_CUDA(cudaGetLastError());
  return PG_OK;
}

template<bool kDrill>
static int learned_decode(const uint8_t* model, const pg_block_ref_t* blocks, int nstreams, const uint8_t* in,
                          const int64_t* in_offsets, const int64_t* in_sizes, uint8_t* symbols,
                          const int64_t* sym_offsets, const int64_t* sym_caps, int64_t* status, void* stream) {
  if (nstreams < 0 || (nstreams && !blocks)) return fail(PG_ERR_ARG, "bad stream list");
  if (!nstreams) return PG_OK;
  if (!model) return fail(PG_ERR_ARG, "null model");
  const cudaStream_t st = (cudaStream_t)stream;
  const dev_tables_t* T = device_tables();
  if (!T) return PG_ERR_CUDA;
  lm_launch L;
  if (int rc = lm_prepare(model, blocks, nstreams, st, L)) return rc;
  if (int rc = launch_rans_decode(in, in_offsets, in_sizes, nstreams, symbols, sym_offsets, sym_caps, status, 1, st))
    return rc;
  if (int rc = lm_smem_opt_in(lm_decode_kernel<kDrill>, kLmCodeSmem)) return rc;
  lm_decode_kernel<kDrill><<<lm_code_grid(nstreams), kLmCodeThreads, kLmCodeSmem, st>>>(
      L.params, L.hash, L.blocks, nstreams, L.order, L.next, in, in_offsets, in_sizes, symbols, sym_offsets, sym_caps,
      status, *T, lm_consts(model));
  PG_CUDA(cudaGetLastError());
  return PG_OK;
}

extern "C" int pg_rans_learned_encode(const uint8_t* model, const pg_block_ref_t* blocks, int nstreams,
                                      const uint8_t* symbols, const int64_t* offsets, uint8_t* out,
                                      const int64_t* out_offsets, int64_t* sizes, void* stream) {
  return learned_encode<false>(model, blocks, nstreams, symbols, offsets, out, out_offsets, sizes, stream);
}

extern "C" int pg_rans_learned_decode(const uint8_t* model, const pg_block_ref_t* blocks, int nstreams,
                                      const uint8_t* in, const int64_t* in_offsets, const int64_t* in_sizes,
                                      uint8_t* symbols, const int64_t* sym_offsets, const int64_t* sym_caps,
                                      int64_t* status, void* stream) {
  return learned_decode<false>(model, blocks, nstreams, in, in_offsets, in_sizes, symbols, sym_offsets, sym_caps, status,
                               stream);
}

// The two with the wait for each stream's last product taken to have run out:
// what a CTA that gives up leaves behind.
extern "C" int pg_debug_learned_encode(const uint8_t* model, const pg_block_ref_t* blocks, int nstreams,
                                       const uint8_t* symbols, const int64_t* offsets, uint8_t* out,
                                       const int64_t* out_offsets, int64_t* sizes, void* stream) {
  return learned_encode<true>(model, blocks, nstreams, symbols, offsets, out, out_offsets, sizes, stream);
}

extern "C" int pg_debug_learned_decode(const uint8_t* model, const pg_block_ref_t* blocks, int nstreams,
                                       const uint8_t* in, const int64_t* in_offsets, const int64_t* in_sizes,
                                       uint8_t* symbols, const int64_t* sym_offsets, const int64_t* sym_caps,
                                       int64_t* status, void* stream) {
  return learned_decode<true>(model, blocks, nstreams, in, in_offsets, in_sizes, symbols, sym_offsets, sym_caps, status,
                              stream);
}

extern "C" int pg_learned_freqs(const uint8_t* model, const pg_block_ref_t* blocks, int nstreams,
                                const uint8_t* symbols, const int64_t* offsets, const int64_t* samples, int64_t n,
                                uint32_t* freqs, void* stream) {
  if (nstreams < 0 || n < 0 || (nstreams && !blocks)) return fail(PG_ERR_ARG, "bad arguments");
  if (!n) return PG_OK;
  if (!model) return fail(PG_ERR_ARG, "null model");
  const cudaStream_t st = (cudaStream_t)stream;
  const dev_tables_t* T = device_tables();
  if (!T) return PG_ERR_CUDA;
  lm_launch L;
  if (int rc = lm_prepare(model, blocks, nstreams, st, L)) return rc;
  if (int rc = lm_smem_opt_in(lm_freqs_kernel, sizeof(lm_tables))) return rc;
  const int grid = int(std::min<int64_t>((n + kLmThreads - 1) / kLmThreads, 1024));
  lm_freqs_kernel<<<grid, kLmThreads, sizeof(lm_tables), st>>>(L.params, L.blocks, nstreams, symbols, offsets, samples,
                                                                n, freqs, *T);
  PG_CUDA(cudaGetLastError());
  return PG_OK;
}

extern "C" int pg_learned_samples(const int64_t* candidates, int64_t ncand, uint64_t seed, int64_t step,
                                  int64_t batch, int64_t* samples, void* stream) {
  if (ncand <= 0 || batch < 0 || step < 0) return fail(PG_ERR_ARG, "bad arguments");
  if (!batch) return PG_OK;
  lm_samples_kernel<<<unsigned((batch + 255) / 256), 256, 0, (cudaStream_t)stream>>>(candidates, ncand, seed, step,
                                                                                    batch, samples);
  PG_CUDA(cudaGetLastError());
  return PG_OK;
}

extern "C" int pg_learned_grad(const float* params, const pg_block_ref_t* blocks, int nstreams, const uint8_t* symbols,
                               const int64_t* offsets, const int64_t* samples, int64_t n, float* grad, float* loss,
                               void* stream) {
  if (nstreams < 0 || n < 0 || (nstreams && !blocks) || !params || !grad) return fail(PG_ERR_ARG, "bad arguments");
  const cudaStream_t st = (cudaStream_t)stream;
  const dev_tables_t* T = device_tables();
  if (!T) return PG_ERR_CUDA;
  lm_launch L;
  if (int rc = lm_prepare(nullptr, blocks, nstreams, st, L)) return rc;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int grid = int(std::max<int64_t>(1, std::min<int64_t>((n + kTile - 1) / kTile, sms)));
  stream_scratch X(st);
  float* partial = nullptr;
  PG_CUDA(X.alloc(&partial, sizeof(float) * grid * (kLmParams + 1)));
  if (int rc = lm_smem_opt_in(lm_grad_kernel, sizeof(lm_grad_smem))) return rc;
  lm_grad_kernel<<<grid, kGradThreads, sizeof(lm_grad_smem), st>>>(params, L.blocks, nstreams, symbols, offsets,
                                                                    samples, n, partial, *T);
  PG_CUDA(cudaGetLastError());
  constexpr int kCols = 256 / kReduceParts;
  lm_reduce_kernel<<<(kLmParams + 1 + kCols - 1) / kCols, 256, 0, st>>>(partial, grid, grad, loss);
  PG_CUDA(cudaGetLastError());
  return PG_OK;
}

extern "C" int pg_learned_adam(float* params, float* m, float* v, const float* grad, int64_t step, float lr,
                               float scale, void* stream) {
  if (!params || !m || !v || !grad || step < 1) return fail(PG_ERR_ARG, "bad arguments");
  const float c1 = 1.f - std::pow(0.9f, float(step)), c2 = 1.f - std::pow(0.999f, float(step));
  lm_adam_kernel<<<(kLmParams + 255) / 256, 256, 0, (cudaStream_t)stream>>>(params, m, v, grad, lr, scale, c1, c2);
  PG_CUDA(cudaGetLastError());
  return PG_OK;
}
