// Gated delta rule, backward, heads of 64, on the sm_100a tensor cores (formulas in gdelta_bwd.cu, layout in gdelta64.cuh).
//
// One CTA per (batch, head) sequence walks its chunks right to left; dS (64 x 64, fp32) stays in registers, 16 per thread.
// With j and t tokens, v and k features, and X = dO U^T, W = dR U^T, per chunk:
//   products A: K K^T, Q K^T, S-side (K S_in^T, Q S_in^T), K dS^T, X
//   epilogue A: P = tril(G o QK^T), dO . (S_in q)
//   product  B: P^T dO             epilogue B: dU = P^T dO + gam K dS^T, u . (dS k); gam U and g dO meanwhile
//   product  C: dR = T'^T dU       epilogue C: dV = dR, -g dR, dR . (S_in k), dR . U
//   products D: W; then the terms of dQ, dK and dS_in that do not need it, under
//   epilogue D: dX o G, dL o G, and the row and column sums of E
//   products E: the rest of dQ and dK     epilogue E: output tiles, dS <- g_last dS + increment
// Rows are tokens everywhere, so the sums over features that the decay, beta and gam cotangents need are 16 values a thread
// and one shuffle, and the column sums of E four shuffle steps; no 64 x 64 fp32 matrix goes through shared memory.
// Bound: the serial chain of five groups of products a chunk; two CTAs per SM (108 KiB each) run under each other's.
#include "gdelta64.cuh"

namespace mxk {
namespace gdelta {
namespace heads64 {
namespace {

struct Smem {
  uint4 s[kTileVecs];     // S_in      [k/8][v][8]
  uint4 u[kTileVecs];     // U         [v/8][t][8]   (one bulk copy with s)
  uint4 ds[kTileVecs];    // dS        [k/8][v][8]
  uint4 k[kTileVecs];     // lines
  uint4 q[kTileVecs];     // lines
  uint4 d_o[kTileVecs];   // dO, later g dO          (lines)
  uint4 tp[kTileVecs];    // T'        [j/8][t][8]
  uint4 p[kTileVecs];     // P [j/8][t][8], later gam U [v/8][t][8]
  uint4 r1[kTileVecs];    // dU, later dR [v/8][t][8], later the dQ tile (lines)
  uint4 r2[kTileVecs];    // -g dR     [v/8][t][8]
  uint4 dpg[kTileVecs];   // dX o G    [j/8][t][8], later the dK tile (lines)
  uint4 dlg[kTileVecs];   // dL o G    [j/8][t][8]
  uint4 dv[kTileVecs];    // dV tile   (lines)
  float alpha[kC], beta[kC], cum[kC], g[kC], gam[kC];
  float dg[2][kC], dgam[2][kC], dru[2][kC], rowsum[2][kC], colsum[4][kC];
  float dcum[kC], gg[kC], dgl[8];
  uint64_t bar[3];
  uint64_t bar_load;
  uint32_t tmem;
};
static_assert(sizeof(Smem) <= 113 * 1024, "two CTAs per SM");

constexpr uint32_t kTmemCols = 256;
// Accumulator slots: dQ (lower lanes) and dK (upper lanes) are 64 columns wide and take two.
constexpr uint32_t kKK = 0, kQK = kSlot, kY = 2 * kSlot, kOI = 3 * kSlot, kX2 = 4 * kSlot, kX1 = 5 * kSlot, kX = 6 * kSlot, kDR = 7 * kSlot,
                   kW = kOI, kDQK = kX2, kDS = kDR;

__device__ __forceinline__ void issue_loads(Smem& sm, const Backward& p, int bh, int b, int h, int c, int nchunks) {
  fence_smem_to_async();   // earlier accesses by threads to the buffers come first
  tma::expect_bytes(&sm.bar_load, 6 * kTileVecs * 16);
  const int t0 = c * kC;
  const size_t at = static_cast<size_t>(bh) * nchunks + c;
  const uint4 *res = p.residual + at * kResidualVecs64, *tp = p.tprime + at * kAinvVecs;
  tma::load_plain_tile(sm.k, &p.map_k, &sm.bar_load, t0, h, b);
  tma::load_plain_tile(sm.q, &p.map_q, &sm.bar_load, t0, h, b);
  tma::load_plain_tile(sm.d_o, &p.map_do, &sm.bar_load, t0, h, b);
  tma::load_bulk(sm.s, res, kResidualVecs64 * 16, &sm.bar_load);
  tma::load_bulk(sm.tp, tp, kAinvVecs * 16, &sm.bar_load);
  if (c > 0) {   // the chunk after it (right to left): into L2 now
    tma::prefetch_plain_tile(&p.map_k, t0 - kC, h, b);
    tma::prefetch_plain_tile(&p.map_q, t0 - kC, h, b);
    tma::prefetch_plain_tile(&p.map_do, t0 - kC, h, b);
    tma::prefetch_bulk(res - kResidualVecs64, kResidualVecs64 * 16);
    tma::prefetch_bulk(tp - kAinvVecs, kAinvVecs * 16);
  }
}

__device__ __forceinline__ float other_half(float x) { return x + __shfl_xor_sync(0xffffffffu, x, 16); }

__global__ void __launch_bounds__(kThreads64, 2) gdelta64_bwd_kernel(const __grid_constant__ Backward p) {
  enter_kernel();
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, wg = warp >> 2;
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

  if (tid == 0) issue_loads(sm, p, bh, b, h, nchunks - 1, nchunks);
  const uint8_t* drow = p.done ? p.done + static_cast<size_t>(b) * p.T : nullptr;
  const size_t bt_base = static_cast<size_t>(b) * p.T;
  Gates gates{};
  if (warp == 1) gates = load_gates(p.alpha, p.beta, bt_base, p.H, h, (nchunks - 1) * kC, p.T, lane);
  linattn::DoneFlags flags = linattn::load_done_flags(drow, (nchunks - 1) * kC, p.T, lane);
  float ds[16];   // dS[row][c0 ..], rows are value features
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (p.ds_last) x = *reinterpret_cast<const float4*>(p.ds_last + state_at + 4 * i);
    ds[4 * i] = x.x; ds[4 * i + 1] = x.y; ds[4 * i + 2] = x.z; ds[4 * i + 3] = x.w;
  }
  bool timed_out = false;

  for (int it = 0; it < nchunks; ++it) {
    const int c = nchunks - 1 - it;
    const int t0 = c * kC;
    const uint64_t dm = linattn::done_mask_from_flags(flags);
#pragma unroll
    for (int i = 0; i < 2; ++i) sm.ds[(me.ch + i) * kC + me.row] = pack8_bf16(ds + 8 * i);
    fence_smem_to_async();
    fence_before_sync();
    __syncthreads();
    if (warp == 0) {
      const bool leader = elect_one();
      mbar_wait_flag(&sm.bar_load, it & 1, timed_out);
      fence_after_sync();
      product(tmem + kQK, lines(sm.q, false), lines(sm.k, false), false, leader);
      product(tmem + kOI, lines(sm.q, false), panels(sm.s, false), false, leader);
      product(tmem + kX2, lines(sm.k, false), panels(sm.ds, false), false, leader);
      if (leader) commit(&sm.bar[0]);
      // needed from epilogue C on, complete with product C
      product(tmem + kY, lines(sm.k, false), panels(sm.s, false), false, leader);
      product(tmem + kKK, lines(sm.k, false), lines(sm.k, false), false, leader);
      product(tmem + kX, lines(sm.d_o, false), panels(sm.u, false), false, leader);
      if (lane == 0) tma::wait_group_read<0>();   // the previous chunk's output tiles have left `r1`, `dpg` and `dv`
      __syncwarp();
    } else if (warp == 1) {
      chunk_decay(gates, dm, lane, sm.cum, sm.g, sm.gam);
#pragma unroll
      for (int e = 0; e < 2; ++e) { sm.alpha[2 * lane + e] = gates.a[e]; sm.beta[2 * lane + e] = gates.b[e]; }
    }
    __syncthreads();
    mbar_wait_flag(&sm.bar_load, it & 1, timed_out);
    mbar_wait_flag(&sm.bar[0], 0, timed_out);
    fence_after_sync();

    // ---- epilogue A ----
    const uint32_t seen = keys_seen(dm, me.row, me.c0);
    const float cum_t = sm.cum[me.row], gt = sm.g[me.row], gm = sm.gam[me.row];
    float dg = 0.f;
    {
      float qk[16], oi[16];
      load16(me.tmem + kQK, qk);
      load16(me.tmem + kOI, oi);
      tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 16; ++e) qk[e] *= decay_between(cum_t, sm.cum[me.c0 + e], seen, e);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        sm.p[(me.ch + i) * kC + me.row] = pack8_bf16(qk + 8 * i);
        float f[8];
        unpack8_bf16(sm.d_o[sw_idx(me.row, me.ch + i)], f);
#pragma unroll
        for (int e = 0; e < 8; ++e) dg = fmaf(oi[8 * i + e], f[e], dg);
      }
    }
    fence_smem_to_async();
    fence_before_sync();
    __syncthreads();
    if (warp == 0) {
      const bool leader = elect_one();
      fence_after_sync();
      product(tmem + kX1, panels(sm.p, true), lines(sm.d_o, true), false, leader);
      if (leader) commit(&sm.bar[1]);
    }
    uint4 u2[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) u2[i] = sm.u[(me.ch + i) * kC + me.row];
    mbar_wait_flag(&sm.bar[1], 0, timed_out);
    fence_after_sync();

    // ---- epilogue B ----
    float dgam = 0.f;
    {
      float x1[16], x2[16];
      load16(me.tmem + kX2, x2);   // (dS k_t)[v]
      load16(me.tmem + kX1, x1);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float f[8];
        unpack8_bf16(u2[i], f);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          dgam = fmaf(x2[8 * i + e], f[e], dgam);
          x1[8 * i + e] = fmaf(gm, x2[8 * i + e], x1[8 * i + e]);
        }
        sm.r1[(me.ch + i) * kC + me.row] = pack8_bf16(x1 + 8 * i);
      }
    }
    fence_smem_to_async();
    fence_before_sync();
    __syncthreads();
    if (warp == 0) {
      const bool leader = elect_one();
      fence_after_sync();
      product(tmem + kDR, panels(sm.tp, true), panels(sm.r1, true), false, leader);
      if (leader) commit(&sm.bar[2]);
    }
    // meanwhile: <dS, S_in> for the cotangent of g_last, gam U over P, g dO in place
    {
      float dot = 0.f;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int at = (me.ch + i) * kC + me.row, line = sw_idx(me.row, me.ch + i);
        float f[8];
        unpack8_bf16(sm.s[at], f);
#pragma unroll
        for (int e = 0; e < 8; ++e) dot = fmaf(ds[8 * i + e], f[e], dot);
        unpack8_bf16(u2[i], f);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] *= gm;
        sm.p[at] = pack8_bf16(f);
        unpack8_bf16(sm.d_o[line], f);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] *= gt;
        sm.d_o[line] = pack8_bf16(f);
      }
#pragma unroll
      for (int off = 16; off >= 1; off >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, off);
      if (lane == 0) sm.dgl[warp] = dot;
      const float g_last = sm.g[kC - 1];
#pragma unroll
      for (int e = 0; e < 16; ++e) ds[e] *= g_last;
    }
    mbar_wait_flag(&sm.bar[2], it & 1, timed_out);
    fence_after_sync();

    // ---- epilogue C ----
    {
      float dr[16], y[16], dru = 0.f;
      load16(me.tmem + kDR, dr);
      load16(me.tmem + kY, y);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int at = (me.ch + i) * kC + me.row;
        float f[8];
        unpack8_bf16(u2[i], f);
        const uint4 x = pack8_bf16(dr + 8 * i);
        sm.r1[at] = x;
        sm.dv[sw_idx(me.row, me.ch + i)] = x;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          dru = fmaf(dr[8 * i + e], f[e], dru);
          dg = fmaf(-dr[8 * i + e], y[8 * i + e], dg);
          dr[8 * i + e] *= -gt;
        }
        sm.r2[at] = pack8_bf16(dr + 8 * i);
      }
      dg = other_half(dg);
      dgam = other_half(dgam);
      dru = other_half(dru);
      if (!me.upper) {
        sm.dg[wg][me.row] = dg;
        sm.dgam[wg][me.row] = dgam;
        sm.dru[wg][me.row] = dru;
      }
    }
    fence_smem_to_async();
    fence_before_sync();
    __syncthreads();
    if (warp == 0) {
      const bool leader = elect_one();
      fence_after_sync();
      if (lane == 0) {
        tma::store_plain_tile(&p.map_dv, sm.dv, t0, h, b);   // rows past the end of the sequence are clipped
        tma::commit_group();
      }
      __syncwarp();
      product(tmem + kW, panels(sm.r1, false), panels(sm.u, false), false, leader);
      if (leader) commit(&sm.bar[0]);
      // dQ = g dO S_in, dK = gam U dS - g dR S_in, dS_in - g_last dS = (g dO)^T Q - (g dR)^T K
      const uint32_t id_nt = idesc_bf16(kC, kC, false, true);
      gemm<4>(tmem + kDQK, lines(sm.d_o, false), panels(sm.s, true), id_nt, false, leader);
      gemm<4>(tmem + kUpperLanes + kDQK, panels(sm.p, false), panels(sm.ds, true), id_nt, false, leader);
      gemm<4>(tmem + kUpperLanes + kDQK, panels(sm.r2, false), panels(sm.s, true), id_nt, true, leader);
      product(tmem + kDS, lines(sm.d_o, true), lines(sm.q, true), false, leader);
      product(tmem + kDS, panels(sm.r2, true), lines(sm.k, true), true, leader);
    }
    mbar_wait_flag(&sm.bar[0], 1, timed_out);
    fence_after_sync();

    // ---- epilogue D ----
    {
      float ev[16], rs = 0.f;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float kk[8], qk[8], x[8], w[8];
        tmem_ld8(me.tmem + kKK + 8 * i, kk);
        tmem_ld8(me.tmem + kQK + 8 * i, qk);
        tmem_ld8(me.tmem + kX + 8 * i, x);
        tmem_ld8(me.tmem + kW + 8 * i, w);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int j = me.c0 + 8 * i + e;
          const float gtj = decay_between(cum_t, sm.cum[j], seen, 8 * i + e);
          const float dl = j < me.row ? -w[e] : 0.f;
          ev[8 * i + e] = (x[e] * qk[e] + dl * kk[e]) * gtj;
          rs += ev[8 * i + e];
          x[e] *= gtj;
          w[e] = dl * gtj;
        }
        sm.dpg[(me.ch + i) * kC + me.row] = pack8_bf16(x);
        sm.dlg[(me.ch + i) * kC + me.row] = pack8_bf16(w);
      }
      rs = other_half(rs);
      if (!me.upper) sm.rowsum[wg][me.row] = rs;
      // column sums over this warp's 16 rows: lane l & 15 ends with column c0 + (l & 15)
#pragma unroll
      for (int n = 8; n >= 1; n >>= 1) {
        const bool high = (lane & n) != 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (i >= n) continue;
          const float send = high ? ev[i] : ev[i + n], keep = high ? ev[i + n] : ev[i];
          ev[i] = keep + __shfl_xor_sync(0xffffffffu, send, n);
        }
      }
      sm.colsum[warp & 3][me.c0 + (lane & 15)] = ev[0];
    }
    fence_smem_to_async();
    fence_before_sync();
    __syncthreads();
    if (warp == 0) {
      const bool leader = elect_one();
      fence_after_sync();
      const uint32_t id_nt = idesc_bf16(kC, kC, false, true), id_tt = idesc_bf16(kC, kC, true, true);
      gemm<4>(tmem + kDQK, panels(sm.dpg, false), lines(sm.k, true), id_nt, true, leader);
      gemm<4>(tmem + kUpperLanes + kDQK, panels(sm.dpg, true), lines(sm.q, true), id_tt, true, leader);
      gemm<4>(tmem + kUpperLanes + kDQK, panels(sm.dlg, false), lines(sm.k, true), id_nt, true, leader);
      gemm<4>(tmem + kUpperLanes + kDQK, panels(sm.dlg, true), lines(sm.k, true), id_tt, true, leader);
      if (leader) commit(&sm.bar[1]);
    }
    // meanwhile, warps 2 and 3: the cotangents of alpha and beta
    if (tid >= 64 && tid < 128) {
      const int x = tid - 64;
      const float cs = (sm.colsum[0][x] + sm.colsum[1][x]) + (sm.colsum[2][x] + sm.colsum[3][x]);
      const float gdg = (sm.dgam[0][x] + sm.dgam[1][x]) * sm.gam[x];
      sm.dcum[x] = (sm.rowsum[0][x] + sm.rowsum[1][x]) - cs + (sm.dg[0][x] + sm.dg[1][x]) * sm.g[x] - gdg;
      sm.gg[x] = gdg;
      const float beta = sm.beta[x];
      if (t0 + x < p.T) p.dbeta[(bt_base + t0 + x) * p.H + h] = beta != 0.f ? (sm.dru[0][x] + sm.dru[1][x]) / (beta * beta) : 0.f;
      asm volatile("bar.sync 2, 64;" ::: "memory");   // warps 2 and 3 only
      if (x < 32) {
        float extra = sm.gg[2 * x] + sm.gg[2 * x + 1];
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) extra += __shfl_xor_sync(0xffffffffu, extra, off);
        extra += (((sm.dgl[0] + sm.dgl[1]) + (sm.dgl[2] + sm.dgl[3])) + ((sm.dgl[4] + sm.dgl[5]) + (sm.dgl[6] + sm.dgl[7]))) * sm.g[kC - 1];
        float d0 = sm.dcum[2 * x], d1 = sm.dcum[2 * x + 1];
        if (x == 31) d1 += extra;
        float s = d0 + d1;   // suffix sums over the chunk
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const float o = __shfl_down_sync(0xffffffffu, s, off);
          if (x + off < 32) s += o;
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int i = 2 * x + e;
          if (t0 + i < p.T) p.dalpha[(bt_base + t0 + i) * p.H + h] = ((dm >> i) & 1ull) ? 0.f : (e ? s - d0 : s) / sm.alpha[i];
        }
      }
    }
    mbar_wait_flag(&sm.bar[1], 1, timed_out);
    fence_after_sync();
    if (c > 0) {
      if (tid == 0) issue_loads(sm, p, bh, b, h, c - 1, nchunks);
      if (warp == 1) gates = load_gates(p.alpha, p.beta, bt_base, p.H, h, t0 - kC, p.T, lane);
      flags = linattn::load_done_flags(drow, t0 - kC, p.T, lane);
    }

    // ---- epilogue E: lanes 0..15 hold rows of dQ, lanes 16..31 of dK, 32 columns per warpgroup ----
    {
      uint4* const tile = me.upper ? sm.dpg : sm.r1;
      float x[32], inc[16];
      tmem_ld8(me.tmem + kDQK + wg * 16, x);        // (me.tmem holds wg * 16 already)
      tmem_ld8(me.tmem + kDQK + wg * 16 + 8, x + 8);
      tmem_ld8(me.tmem + kDQK + wg * 16 + 16, x + 16);
      tmem_ld8(me.tmem + kDQK + wg * 16 + 24, x + 24);
      load16(me.tmem + kDS, inc);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 4; ++i) tile[sw_idx(me.row, wg * 4 + i)] = pack8_bf16(x + 8 * i);
#pragma unroll
      for (int e = 0; e < 16; ++e) ds[e] += inc[e];
    }
    fence_smem_to_async();
    fence_before_sync();
    __syncthreads();
    if (tid == 0) {
      tma::store_plain_tile(&p.map_dq, sm.r1, t0, h, b);
      tma::store_plain_tile(&p.map_dk, sm.dpg, t0, h, b);
      tma::commit_group();
    }
  }
  if (p.ds0) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      *reinterpret_cast<float4*>(p.ds0 + state_at + 4 * i) = make_float4(ds[4 * i], ds[4 * i + 1], ds[4 * i + 2], ds[4 * i + 3]);
  }
  if (tid == 0) tma::wait_group_all();
  if (timed_out && p.status) atomicExch(p.status, 1);
  fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, kTmemCols);
}

}  // namespace

int launch_backward(const Backward& p, int sequences, cudaStream_t stream) {
  cudaError_t e = cudaFuncSetAttribute(gdelta64_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(sizeof(Smem)));
  if (e != cudaSuccess) return static_cast<int>(e);
  mxk::launch_kernel(gdelta64_bwd_kernel, sequences, kThreads64, sizeof(Smem), stream, p);
  return launch_status();
}

}  // namespace heads64
}  // namespace gdelta
}  // namespace mxk
