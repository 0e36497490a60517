// Shared pieces of the gated delta-rule kernels (64-token chunks).
//
// Recurrence per head (S is d_v x d_k, a_t = done_t ? 0 : alpha_t):
//   S_t = a_t S_{t-1} (I - beta_t k_t k_t^T) + beta_t v_t k_t^T,   o_t = S_t q_t.
// Chunk form used by both kernels (rows t, j inside a chunk; cum_t = sum_{i<=t} log alpha_i):
//   G_tj  = exp(cum_t - cum_j) if no reset in (j, t] else 0           (j <= t)
//   g_t   = G from the chunk start (0 once a reset has been passed)   ("live" rows)
//   gam_j = G_{last,j}                                                  ("keep" rows)
//   L = strict_tril(G o K K^T),  (I + diag(beta) L) U = diag(beta) (V - diag(g) K S_in^T)
//   O = diag(g) Q S_in^T + tril(G o Q K^T) U,   S_out = g_last S_in + (diag(gam) U)^T K.
//
// Layout of the kernels, for heads of D = 64 or 128.  Matrices with tokens on their rows are 64 high and none fills the 128
// TMEM lanes of an M = 128 product, so products are M = 64 and cut into two halves of their N columns, the first in lanes
// 0..15 of each warp's TMEM quarter and the second in lanes 16..31.  All 256 threads then own a quarter of the columns of one
// row: what is summed over features is summed in a thread and by one shuffle, and tiles leave in 16-byte vectors.  (Padded to
// 128, a head of 64 took as long as one of 128; with features on the rows, a 64 x 128 matrix in whole lanes needed 31 shuffles
// a sum and two-byte stores for every tile.)
#pragma once

#include <cuda_bf16.h>

#include "linattn_common.cuh"
#include "mxk_common.cuh"
#include "tma.cuh"
#include "umma.cuh"

namespace mxk {
namespace gdelta {

using namespace umma;
using linattn::row_first_key;
using linattn::row_keep;
using linattn::row_live;

constexpr int kC = 64;
constexpr int kSquareVecs = kC * 8;            // uint4 per 64 x 64 bf16 matrix (8 KiB)
constexpr uint32_t kBlockBytes = kC * 128;     // a 64-column block of "lines" (SW tiles, umma.cuh)
constexpr uint32_t kUpperLanes = 16u << 16;

// State-independent part of a chunk, written by the preparation kernel (gdelta_prep.cu) for both the
// forward and the backward kernel: T' = (I + diag(beta) L)^-1 diag(beta) as bf16, [j/8][t][8] (8 KiB).
constexpr int kAinvVecs = kSquareVecs;
// Launches the preparation kernel over all (batch, head, chunk) items; defined in gdelta_prep.cu.
int launch_prep(const void* k, const float* alpha, const float* beta, const uint8_t* done, void* ainv, int* status,
                int B, int T, int H, int d, cudaStream_t stream);

// Residual the forward call leaves per (sequence, chunk): the state entering the chunk [k/8][v][8], then U [v/8][t][8].
__host__ __device__ constexpr int state_vecs(int d) { return d * d / 8; }
__host__ __device__ constexpr int tile_vecs(int d) { return kC * d / 8; }
__host__ __device__ constexpr int residual_vecs(int d) { return state_vecs(d) + tile_vecs(d); }

// Bit e: key j0 + e is one that token `row` of a chunk sees (no reset in between), up to itself.
__device__ __forceinline__ uint32_t keys_seen(uint64_t dm, int row, int j0) {
  return static_cast<uint32_t>(((2ull << row) - (1ull << row_first_key(dm, row))) >> j0);
}
// G_tj = exp(cum_t - cum_j) where bit e is set, 0 elsewhere; selected before the exponential: around it the
// selection became a branch per key, half the time of an epilogue (backward, heads of 64: 517 us a launch against 428).
__device__ __forceinline__ float decay_between(float cum_t, float cum_j, uint32_t seen, int e) {
  return __expf((seen >> e) & 1u ? cum_t - cum_j : -INFINITY);
}

// What a thread owns of the 64 x D matrices: D / 4 columns of a row; and of the 64 x 64 ones over two tokens: 16 of the same
// row.
template <int D>
struct Place {
  static constexpr int kCols = D / 4, kVecs = kCols / 8;
  int row, c0, ch;      // ch = c0 / 8
  int j0;
  bool upper;
  uint32_t lanes;       // TMEM address of this warp's lanes
  uint32_t col, jcol;   // where its columns start within an accumulator
  __device__ __forceinline__ Place(int tid, uint32_t tmem) {
    const int warp = tid >> 5, lane = tid & 31, wg = warp >> 2, qw = warp & 3;
    upper = lane >= 16;
    row = qw * 16 + (lane & 15);
    c0 = (upper ? D / 2 : 0) + wg * kCols;
    ch = c0 >> 3;
    j0 = (upper ? 32 : 0) + wg * 16;
    lanes = tmem + (static_cast<uint32_t>(qw * 32) << 16);
    col = wg * kCols;
    jcol = wg * 16;
  }
};
// What it owns of the state (rows value features): with D = 128 the accumulator fills all lanes.
template <int D>
struct StatePlace {
  static constexpr int kCols = D * D / 256;
  int row, c0;
  uint32_t col;
  __device__ __forceinline__ explicit StatePlace(int tid) {
    const int warp = tid >> 5, lane = tid & 31, wg = warp >> 2;
    row = D == 64 ? (warp & 3) * 16 + (lane & 15) : tid & 127;
    c0 = D == 64 ? (lane >= 16 ? 32 : 0) + wg * 16 : wg * 64;
    col = wg * kCols;
  }
};
// uint4 index of the 16-byte vector `ch` of row `r` in lines of D columns
__device__ __forceinline__ int line_at(int r, int ch) { return (ch >> 3) * kSquareVecs + sw_idx(r, ch & 7); }

template <int ROWS>
__device__ __forceinline__ Operand panels(const uint4* m, bool contract_rows) { return Operand{smem_u32(m), ROWS, contract_rows}; }
__device__ __forceinline__ Operand lines(const uint4* m, bool contract_rows) { return sw_operand(smem_u32(m), contract_rows, kBlockBytes); }
// The N side of a product from its row or column n (32 or 64) on.
__device__ __forceinline__ Operand from(Operand b, uint32_t n) {
  if (b.swizzled) b.saddr += b.contract_rows ? (n == 64 ? kBlockBytes : n * 2) : n * 128u;
  else b.saddr += b.contract_rows ? n / 8 * b.rows * 16u : n * 16u;
  return b;
}
template <int K>
__device__ __forceinline__ void contract(uint32_t d, const Operand& a, const Operand& b, uint32_t idesc, bool accumulate, bool leader) {
  if constexpr (K == 64) gemm<4>(d, a, b, idesc, accumulate, leader);
  else gemm128(d, a, b, idesc, accumulate, leader);
}
// D [64 x N] (+)= A B^T over K in halves, at TMEM address `d`; called by one warp.
template <int N, int K>
__device__ __forceinline__ void product(uint32_t d, const Operand& a, const Operand& b, bool accumulate, bool leader) {
  const uint32_t id = idesc_bf16(kC, N / 2, a.contract_rows, b.contract_rows);
  contract<K>(d, a, b, id, accumulate, leader);
  contract<K>(d + kUpperLanes, a, from(b, N / 2), id, accumulate, leader);
}
// The same with all N columns in the lanes of `d`.
template <int N, int K>
__device__ __forceinline__ void product_rows(uint32_t d, const Operand& a, const Operand& b, bool accumulate, bool leader) {
  contract<K>(d, a, b, idesc_bf16(kC, N, a.contract_rows, b.contract_rows), accumulate, leader);
}
// State accumulator [D x D] += A B^T over the 64 tokens.
template <int D>
__device__ __forceinline__ void product_state(uint32_t d, const Operand& a, const Operand& b, bool accumulate, bool leader) {
  if constexpr (D == 64) product<64, 64>(d, a, b, accumulate, leader);
  else gemm<4>(d, a, b, idesc_bf16(D, D, a.contract_rows, b.contract_rows), accumulate, leader);
}
template <int N>
__device__ __forceinline__ void tmem_load(uint32_t taddr, float* x) {   // (the caller waits)
#pragma unroll
  for (int i = 0; i < N; i += 8) tmem_ld8(taddr + i, x + i);
}

// alpha and beta of tokens t0 + 2 lane, t0 + 2 lane + 1 (1 and 0 past the end: such rows leave the state alone).
struct Gates {
  float a[2], b[2];
};
__device__ __forceinline__ Gates load_gates(const float* alpha, const float* beta, size_t bt_base, int H, int h, int t0, int T, int lane) {
  Gates g;
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int t = t0 + 2 * lane + e;
    const bool in = t >= 0 && t < T;
    const size_t i = (bt_base + t) * H + h;
    g.a[e] = in ? __ldg(alpha + i) : 1.f;
    g.b[e] = (in && beta) ? __ldg(beta + i) : 0.f;
  }
  return g;
}
// cum of tokens 2 lane, 2 lane + 1, by one warp.
__device__ __forceinline__ float2 cumulative(const Gates& ga, int lane) {
  const float l1 = __logf(ga.a[1]);
  float s = __logf(ga.a[0]) + l1;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const float o = __shfl_up_sync(0xffffffffu, s, off);
    if (lane >= off) s += o;
  }
  return make_float2(s - l1, s);
}
// cum, g and gam of a chunk, by one warp.
__device__ __forceinline__ void chunk_decay(const Gates& ga, uint64_t dm, int lane, float* cum, float* g, float* gam) {
  const float2 s = cumulative(ga, lane);
  const float last = __shfl_sync(0xffffffffu, s.y, 31);
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int t = 2 * lane + e;
    const float c = e ? s.y : s.x;
    cum[t] = c;
    g[t] = row_live(dm, t) ? __expf(c) : 0.f;
    gam[t] = row_keep(dm, t) ? __expf(last - c) : 0.f;
  }
}

}  // namespace gdelta
}  // namespace mxk
