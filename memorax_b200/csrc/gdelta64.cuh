// Shared pieces of the gated delta-rule kernels for heads of 64 (math in gdelta_common.cuh).
//
// Every matrix of a chunk is 64 x 64 here, so none fills the 128 TMEM lanes of an M = 128 product.  Padded to 128 a head
// took as long as one of 128 features; instead products are M = 64 and cut into two N = 32 halves, the first in lanes
// 0..15 of each warp's TMEM quarter and the second in lanes 16..31.  All 256 threads then own 16 columns of one row, rows
// are tokens (value features only for the state), every sum over features is a few shuffles, and a CTA is small enough for
// two or three to share an SM and hide each other's waits.
#pragma once

#include "gdelta_common.cuh"
#include "tma.cuh"

namespace mxk {
namespace gdelta {
namespace heads64 {

using namespace umma;

constexpr int kThreads64 = 256;
constexpr int kTileVecs = kC * 8;              // uint4 per 64 x 64 bf16 matrix (8 KiB)
// Residual the forward call leaves per (sequence, chunk): the state entering it [k/8][v][8], then U [v/8][t][8].
constexpr int kResidualVecs64 = 2 * kTileVecs;
constexpr uint32_t kSlot = 32;                 // TMEM columns of a 64 x 64 accumulator in halves
constexpr uint32_t kUpperLanes = 16u << 16;

// What a thread owns of every 64 x 64 matrix.
struct Place {
  int row, c0;          // its row, and the first of its 16 columns
  int ch;               // c0 / 8
  bool upper;
  uint32_t tmem;        // its columns of accumulator slot 0
};
__device__ __forceinline__ Place place_of(int tid, uint32_t tmem) {
  const int warp = tid >> 5, lane = tid & 31, wg = warp >> 2, qw = warp & 3;
  Place m;
  m.upper = lane >= 16;
  m.row = qw * 16 + (lane & 15);
  m.c0 = (m.upper ? 32 : 0) + wg * 16;
  m.ch = m.c0 >> 3;
  m.tmem = tmem + (static_cast<uint32_t>(qw * 32) << 16) + wg * 16;
  return m;
}

// Rows (or columns) 32..63 of the N side of a product.
__device__ __forceinline__ Operand second_half(Operand b) {
  if (b.swizzled) b.saddr += b.contract_rows ? 64u : 32u * 128u;
  else b.saddr += b.contract_rows ? 4u * b.rows * 16u : 32u * 16u;
  return b;
}
// D (+)= A B^T, 64 x 64 x 64, in halves at TMEM address `d`; called by one warp.
__device__ __forceinline__ void product(uint32_t d, const Operand& a, const Operand& b, bool accumulate, bool leader) {
  const uint32_t id = idesc_bf16(kC, 32, a.contract_rows, b.contract_rows);
  gemm<4>(d, a, b, id, accumulate, leader);
  gemm<4>(d + kUpperLanes, a, second_half(b), id, accumulate, leader);
}
__device__ __forceinline__ Operand panels(const uint4* m, bool contract_rows) { return Operand{smem_u32(m), kC, contract_rows}; }
__device__ __forceinline__ Operand lines(const uint4* m, bool contract_rows) { return sw_operand(smem_u32(m), contract_rows); }

__device__ __forceinline__ void load16(uint32_t taddr, float* x) {
  tmem_ld8(taddr, x);
  tmem_ld8(taddr + 8, x + 8);
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

struct Forward {
  const float* alpha;
  const float* s0;
  const uint8_t* done;
  float* s_last;
  uint4* residual;      // nullptr: not kept
  const uint4* tprime;  // T' of every chunk, written by the preparation kernel
  int* status;
  int T, H;
  CUtensorMap map_k, map_q, map_v, map_o;
};
struct Backward {
  const float* alpha;
  const float* beta;
  const uint8_t* done;
  const uint4* residual;
  const uint4* tprime;
  const float* ds_last;
  float* dalpha;
  float* dbeta;
  float* ds0;
  int* status;
  int T, H;
  CUtensorMap map_k, map_q, map_do, map_dq, map_dk, map_dv;
};
int launch_forward(const Forward& p, int sequences, cudaStream_t stream);     // gdelta64.cu
int launch_backward(const Backward& p, int sequences, cudaStream_t stream);   // gdelta64_bwd.cu

}  // namespace heads64
}  // namespace gdelta
}  // namespace mxk
