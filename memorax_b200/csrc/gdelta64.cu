// Gated delta rule, forward, heads of 64, on the sm_100a tensor cores (math in gdelta_common.cuh, layout in gdelta64.cuh).
//
// One CTA per (batch, head) sequence walks its 64-token chunks in order; the state S (64 x 64, fp32) stays in registers, 16
// per thread.  Loads arrive a chunk ahead.  Per chunk:
//   products 1: Q K^T, Y = K S_in^T
//   epilogue 1: P = tril(G o QK^T), -g Y (bf16 operands), Q and K rescaled in place (g Q, gam K)
//   products 2: U = T' V - T' (g Y); then O = (g Q) S_in^T, which epilogue 2 need not wait for
//   epilogue 2: U as bf16 operand and residual
//   products 3: O += P U, dS = U^T (gam K)
//   epilogue 3: output tile, S = g_last S + dS
// Bound: the serial chain of three groups of products a chunk, hidden by three CTAs per SM (56 KiB each).
#include "gdelta64.cuh"

namespace mxk {
namespace gdelta {
namespace heads64 {
namespace {

struct Smem {
  uint4 s[kTileVecs];    // S_in                           [k/8][v][8]
  uint4 k[kTileVecs];    // K, after products 1 gam K      (lines)
  uint4 q[kTileVecs];    // Q, after products 1 g Q        (lines)
  uint4 v[kTileVecs];    // V                              (lines)
  uint4 yu[kTileVecs];   // -g Y, then U [v/8][t][8], then the output tile (lines)
  uint4 p[kTileVecs];    // P                              [j/8][t][8]
  uint4 tp[kTileVecs];   // T'                             [j/8][t][8]
  float cum[kC], g[kC], gam[kC];
  uint64_t bar[3];
  uint64_t bar_load;
  uint32_t tmem;
};
static_assert(sizeof(Smem) <= 75 * 1024, "three CTAs per SM");

constexpr uint32_t kTmemCols = 128;
constexpr uint32_t kQK = 0, kO = 0, kY = kSlot, kDS = kSlot, kU = 2 * kSlot;

__device__ __forceinline__ void issue_loads(Smem& sm, const Forward& p, int bh, int b, int h, int c, int nchunks) {
  fence_smem_to_async();   // earlier accesses by threads to the buffers come first
  tma::expect_bytes(&sm.bar_load, 4 * kTileVecs * 16);
  const int t0 = c * kC;
  const uint4* tp = p.tprime + (static_cast<size_t>(bh) * nchunks + c) * kAinvVecs;
  tma::load_plain_tile(sm.k, &p.map_k, &sm.bar_load, t0, h, b);
  tma::load_plain_tile(sm.q, &p.map_q, &sm.bar_load, t0, h, b);
  tma::load_plain_tile(sm.v, &p.map_v, &sm.bar_load, t0, h, b);
  tma::load_bulk(sm.tp, tp, kAinvVecs * 16, &sm.bar_load);
  if (c + 1 < nchunks) {   // the chunk after it: into L2 now
    tma::prefetch_plain_tile(&p.map_k, t0 + kC, h, b);
    tma::prefetch_plain_tile(&p.map_q, t0 + kC, h, b);
    tma::prefetch_plain_tile(&p.map_v, t0 + kC, h, b);
    tma::prefetch_bulk(tp + kAinvVecs, kAinvVecs * 16);
  }
}

__global__ void __launch_bounds__(kThreads64, 3) gdelta64_fwd_kernel(const __grid_constant__ Forward p) {
  enter_kernel();
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int bh = blockIdx.x, b = bh / p.H, h = bh % p.H;
  const int nchunks = (p.T + kC - 1) / kC;

  if (tid == 0) {
#pragma unroll
    for (int i = 0; i < 3; ++i) mbar_init(&sm.bar[i], 1);
    mbar_init(&sm.bar_load, 1);
    mbar_init_fence();
  }
  if (warp == 0) tmem_alloc(&sm.tmem, kTmemCols);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = sm.tmem;
  const Place me = place_of(tid, tmem);
  const size_t state_at = (static_cast<size_t>(bh) * kC + me.row) * kC + me.c0;

  if (tid == 0) issue_loads(sm, p, bh, b, h, 0, nchunks);
  const uint8_t* drow = p.done ? p.done + static_cast<size_t>(b) * p.T : nullptr;
  const size_t bt_base = static_cast<size_t>(b) * p.T;
  Gates gates{};
  if (warp == 1) gates = load_gates(p.alpha, nullptr, bt_base, p.H, h, 0, p.T, lane);
  linattn::DoneFlags flags = linattn::load_done_flags(drow, 0, p.T, lane);
  float s[16];   // S[row][c0 ..], rows are value features
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (p.s0) x = *reinterpret_cast<const float4*>(p.s0 + state_at + 4 * i);
    s[4 * i] = x.x; s[4 * i + 1] = x.y; s[4 * i + 2] = x.z; s[4 * i + 3] = x.w;
  }
  bool timed_out = false;

  for (int c = 0; c < nchunks; ++c) {
    const int t0 = c * kC;
    const uint64_t dm = linattn::done_mask_from_flags(flags);
#pragma unroll
    for (int i = 0; i < 2; ++i) sm.s[(me.ch + i) * kC + me.row] = pack8_bf16(s + 8 * i);
    fence_smem_to_async();
    fence_before_sync();
    __syncthreads();
    if (warp == 0) {
      const bool leader = elect_one();
      if (lane == 0 && p.residual) {   // for the backward pass: the state entering the chunk
        tma::store_bulk(p.residual + (static_cast<size_t>(bh) * nchunks + c) * kResidualVecs64, sm.s, kTileVecs * 16);
        tma::commit_group();
      }
      mbar_wait_flag(&sm.bar_load, c & 1, timed_out);
      fence_after_sync();
      product(tmem + kQK, lines(sm.q, false), lines(sm.k, false), false, leader);
      product(tmem + kY, lines(sm.k, false), panels(sm.s, false), false, leader);
      if (leader) commit(&sm.bar[0]);
      // the previous chunk's output tile (the older bulk group) has left `yu` before epilogue 1 rewrites it
      if (lane == 0) { if (p.residual) tma::wait_group_read<1>(); else tma::wait_group_read<0>(); }
      __syncwarp();
    } else if (warp == 1) {
      chunk_decay(gates, dm, lane, sm.cum, sm.g, sm.gam);
    }
    __syncthreads();
    mbar_wait_flag(&sm.bar_load, c & 1, timed_out);
    mbar_wait_flag(&sm.bar[0], c & 1, timed_out);
    fence_after_sync();

    {
      const uint32_t seen = keys_seen(dm, me.row, me.c0);
      const float cum_t = sm.cum[me.row], gt = sm.g[me.row], gm = sm.gam[me.row];
      float qk[16], y[16];
      load16(me.tmem + kQK, qk);
      load16(me.tmem + kY, y);
      tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        qk[e] *= decay_between(cum_t, sm.cum[me.c0 + e], seen, e);
        y[e] *= -gt;
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int at = (me.ch + i) * kC + me.row, line = sw_idx(me.row, me.ch + i);
        sm.p[at] = pack8_bf16(qk + 8 * i);
        sm.yu[at] = pack8_bf16(y + 8 * i);
        float f[8];
        unpack8_bf16(sm.q[line], f);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] *= gt;
        sm.q[line] = pack8_bf16(f);
        unpack8_bf16(sm.k[line], f);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] *= gm;
        sm.k[line] = pack8_bf16(f);
      }
    }
    fence_smem_to_async();
    fence_before_sync();
    __syncthreads();
    if (warp == 0) {
      const bool leader = elect_one();
      fence_after_sync();
      product(tmem + kU, panels(sm.tp, false), lines(sm.v, true), false, leader);
      product(tmem + kU, panels(sm.tp, false), panels(sm.yu, true), true, leader);
      if (leader) commit(&sm.bar[2]);
      product(tmem + kO, lines(sm.q, false), panels(sm.s, false), false, leader);
    }
    const float g_last = sm.g[kC - 1];
#pragma unroll
    for (int e = 0; e < 16; ++e) s[e] *= g_last;
    mbar_wait_flag(&sm.bar[2], c & 1, timed_out);
    fence_after_sync();

    {
      float u[16];
      load16(me.tmem + kU, u);
      tmem_ld_wait();
      uint4* res = p.residual ? p.residual + (static_cast<size_t>(bh) * nchunks + c) * kResidualVecs64 + kTileVecs : nullptr;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const uint4 x = pack8_bf16(u + 8 * i);
        sm.yu[(me.ch + i) * kC + me.row] = x;
        if (res) res[(me.ch + i) * kC + me.row] = x;
      }
    }
    fence_smem_to_async();
    fence_before_sync();
    __syncthreads();
    if (warp == 0) {
      const bool leader = elect_one();
      fence_after_sync();
      product(tmem + kO, panels(sm.p, false), panels(sm.yu, true), true, leader);
      product(tmem + kDS, panels(sm.yu, true), lines(sm.k, true), false, leader);
      if (leader) commit(&sm.bar[1]);
    }
    mbar_wait_flag(&sm.bar[1], c & 1, timed_out);
    fence_after_sync();
    if (c + 1 < nchunks) {
      if (tid == 0) issue_loads(sm, p, bh, b, h, c + 1, nchunks);
      if (warp == 1) gates = load_gates(p.alpha, nullptr, bt_base, p.H, h, t0 + kC, p.T, lane);
      flags = linattn::load_done_flags(drow, t0 + kC, p.T, lane);
    }
    {
      float o[16], ds[16];
      load16(me.tmem + kO, o);
      load16(me.tmem + kDS, ds);
      tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 16; ++e) s[e] += ds[e];
#pragma unroll
      for (int i = 0; i < 2; ++i) sm.yu[sw_idx(me.row, me.ch + i)] = pack8_bf16(o + 8 * i);
    }
    fence_smem_to_async();
    if (tid == 0) tma::wait_group_read<0>();   // the residual copy has finished reading `s`
    __syncthreads();
    if (tid == 0) {
      tma::store_plain_tile(&p.map_o, sm.yu, t0, h, b);   // rows past the end of the sequence are clipped
      tma::commit_group();
    }
  }
  if (p.s_last) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      *reinterpret_cast<float4*>(p.s_last + state_at + 4 * i) = make_float4(s[4 * i], s[4 * i + 1], s[4 * i + 2], s[4 * i + 3]);
  }
  if (tid == 0) tma::wait_group_all();
  if (timed_out && p.status) atomicExch(p.status, 1);
  fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, kTmemCols);
}

}  // namespace

int launch_forward(const Forward& p, int sequences, cudaStream_t stream) {
  cudaError_t e = cudaFuncSetAttribute(gdelta64_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(sizeof(Smem)));
  if (e != cudaSuccess) return static_cast<int>(e);
  mxk::launch_kernel(gdelta64_fwd_kernel, sequences, kThreads64, sizeof(Smem), stream, p);
  return launch_status();
}

}  // namespace heads64
}  // namespace gdelta
}  // namespace mxk
