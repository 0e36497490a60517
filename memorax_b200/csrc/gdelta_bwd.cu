// Gated delta rule, backward, on the sm_100a tensor cores (layout in gdelta_common.cuh).
//
// One CTA (256 threads) owns one (batch, head) sequence and walks its 64-token chunks right to left with the fp32 cotangent of
// the state, dS (D x D), resident in tensor memory.  S_in and U of every chunk are the forward call's residual.
// With the chunk quantities of gdelta_common.cuh (A = I + diag(beta) L, P =
// tril(G o QK^T), R = V - diag(g) K S_in^T, U = A^-1 diag(beta) R):
//   dU   = P^T dO + diag(gam) K dS^T            dR = T'^T dU  with T' = A^-1 diag(beta) from the preparation
//                                                kernel (gdelta_prep.cu): a product, no back substitution
//   dV   = dR                                    dbeta_t = (dR_t . U_t) / beta_t^2
//   dP   = tril(dO U^T)                          dL = -stril(dR U^T)
//   dQ   = (dP o G) K + diag(g) dO S_in
//   dK   = (dP o G)^T Q + (dL o G) K + (dL o G)^T K + diag(gam) U dS - diag(g) dR S_in
//   dS_in = g_last dS + (diag(g) dO)^T Q - (diag(g) dR)^T K
//   decay: E = (dP o QK^T + dL o KK^T) o G,  dg_t = do_t.(S_in q_t) - dr_t.(S_in k_t),
//          dgam_j = u_j.(dS k_j),  dg_last += <dS, S_in>;
//          dcum_t = rowsum_t(E) - colsum_t(E) + dg_t g_t - dgam_t gam_t (+ sum_j dgam_j gam_j at t = last),
//          dlog(alpha_i) = sum_{t >= i} dcum_t,  dalpha_i = done_i ? 0 : dlog(alpha_i) / alpha_i.
// With X = dO U^T and W = dR U^T, a chunk is five groups of products, each followed by an epilogue of all threads:
//   A  Q K^T, Q S_in^T, K dS^T (then K S_in^T, K K^T, X, first needed in C and D)   P, dO . (S_in q)
//   B  P^T dO                                      dU, u . (dS k); under C: <dS, S_in>, dS <- g_last dS, gam U, g dO
//   C  dR = T'^T dU                                dV = dR, -g dR, dR . (S_in k), dR . U
//   D  W; under its epilogue the terms of dQ, dK and dS_in that do not need W    dP o G, dL o G, row and column sums of E
//   E  the rest of dQ and dK                       output tiles, bf16 copy of dS
// dQ (lanes 0..15 of every TMEM quarter) and dK (lanes 16..31) share their accumulator columns.
// Bound: that serial chain.  Heads of 64 have two CTAs per SM (108 KiB each) to run it under each other's; heads of 128 fill
// the shared memory of one.  Measured: 512 x 256 steps, 8 heads of 64: 430 us (1308 padded to 128); 128 x 512 steps, 8 heads of
// 128: 462 us (630 with features on the rows and every term of dQ and dK behind the last epilogue).  Four warpgroups instead of
// two for heads of 128: 469.
#include "attention.cuh"
#include "gdelta_common.cuh"

namespace mxk {
namespace {

using namespace gdelta;

struct BwdParams {
  const float* alpha;
  const float* beta;
  const uint8_t* done;
  const uint4* residual;
  const uint4* tprime;                // T' of every chunk (the forward call's workspace)
  const float* ds_last;
  float* dalpha;
  float* dbeta;
  float* ds0;
  int* status;
  int T, H;
  CUtensorMap map_k, map_q, map_do, map_dq, map_dk, map_dv;   // 64-token tiles as lines
};

template <int D>
struct BwdSmem {
  uint4 s[state_vecs(D)];     // S_in      [k/8][v][8]
  uint4 u[tile_vecs(D)];      // U         [v/8][t][8]   (one bulk copy with s)
  uint4 ds[state_vecs(D)];    // dS        [k/8][v][8]
  uint4 k[tile_vecs(D)];      // lines
  uint4 q[tile_vecs(D)];      // lines
  uint4 d_o[tile_vecs(D)];    // dO, later g dO          (lines)
  uint4 tp[kSquareVecs];      // T'        [j/8][t][8], later the dV tile (lines; D = 128: over P too)
  uint4 p[kSquareVecs];       // P         [j/8][t][8], later, D = 64, gam U [v/8][t][8]
  uint4 ug[D == 64 ? 64 : tile_vecs(D)];   // gam U, D = 128
  uint4 r1[tile_vecs(D)];     // dU, later dR [v/8][t][8], later the dQ tile (lines)
  uint4 r2[tile_vecs(D)];     // -g dR     [v/8][t][8]
  uint4 dpg[kSquareVecs];     // dP o G    [j/8][t][8], later the dK tile (lines; D = 128: over dL o G too)
  uint4 dlg[kSquareVecs];     // dL o G    [j/8][t][8]
  float alpha[kC], beta[kC], cum[kC], g[kC], gam[kC];
  float dg[2][kC], dgam[2][kC], dru[2][kC], rowsum[2][kC], colsum[4][kC];
  float dcum[kC], gg[kC], dgl[8];
  uint64_t bar[3];
  uint64_t bar_load;
  uint32_t tmem;
  __device__ __forceinline__ uint4* gam_u() { return D == 64 ? p : ug; }
  __device__ __forceinline__ uint4* dv() { return tp; }
};

template <int D>
struct BwdLayout {
  static constexpr int kPerSm = D == 64 ? 2 : 1;
  static constexpr uint32_t kTmemCols = D == 64 ? 256 : 512;
  static constexpr uint32_t kDS = 0, kKK = D == 64 ? 32 : 128, kQK = kKK + 32, kX = kKK + 64, kY = D == 64 ? 128 : 256, kOI = kY + D / 2,
                            kX2 = kOI + D / 2, kX1 = kX2 + D / 2, kDR = kOI, kW = D == 64 ? kY : kKK + 96, kDQK = kX2;
  static_assert(kPerSm * (sizeof(BwdSmem<D>) + 1024) <= 228 * 1024 && kX1 + D / 2 <= kTmemCols, "CTAs per SM");
};

constexpr int kBwdThreads = 256;

template <int D>
__device__ __forceinline__ void issue_loads(BwdSmem<D>& sm, const BwdParams& p, int bh, int b, int h, int c, int nchunks) {
  fence_smem_to_async();   // earlier accesses by threads to the buffers come first
  tma::expect_bytes(&sm.bar_load, (3 * tile_vecs(D) + residual_vecs(D) + kAinvVecs) * 16);
  const int t0 = c * kC;
  const size_t at = static_cast<size_t>(bh) * nchunks + c;
  const uint4 *res = p.residual + at * residual_vecs(D), *tp = p.tprime + at * kAinvVecs;
#pragma unroll
  for (int i = 0; i < D / 64; ++i) {
    tma::load_plain_tile(sm.k + i * kSquareVecs, &p.map_k, &sm.bar_load, t0, h, b, 64 * i);
    tma::load_plain_tile(sm.q + i * kSquareVecs, &p.map_q, &sm.bar_load, t0, h, b, 64 * i);
    tma::load_plain_tile(sm.d_o + i * kSquareVecs, &p.map_do, &sm.bar_load, t0, h, b, 64 * i);
  }
  tma::load_bulk(sm.s, res, residual_vecs(D) * 16, &sm.bar_load);
  tma::load_bulk(sm.tp, tp, kAinvVecs * 16, &sm.bar_load);
  if (c > 0) {   // the chunk after it (right to left): into L2 now
#pragma unroll
    for (int i = 0; i < D / 64; ++i) {
      tma::prefetch_plain_tile(&p.map_k, t0 - kC, h, b, 64 * i);
      tma::prefetch_plain_tile(&p.map_q, t0 - kC, h, b, 64 * i);
      tma::prefetch_plain_tile(&p.map_do, t0 - kC, h, b, 64 * i);
    }
    tma::prefetch_bulk(res - residual_vecs(D), residual_vecs(D) * 16);
    tma::prefetch_bulk(tp - kAinvVecs, kAinvVecs * 16);
  }
}

__device__ __forceinline__ float other_half(float x) { return x + __shfl_xor_sync(0xffffffffu, x, 16); }

template <int D>
__global__ void __launch_bounds__(kBwdThreads, BwdLayout<D>::kPerSm) gdelta_bwd_kernel(const __grid_constant__ BwdParams p) {
  enter_kernel();
  using L = BwdLayout<D>;
  constexpr int kVecs = Place<D>::kVecs, kCols = Place<D>::kCols, kStateCols = StatePlace<D>::kCols;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  BwdSmem<D>& sm = *reinterpret_cast<BwdSmem<D>*>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, wg = warp >> 2;
  const int bh = blockIdx.x, b = bh / p.H, h = bh % p.H;
  const int nchunks = (p.T + kC - 1) / kC;

  if (tid == 0) {
#pragma unroll
    for (int i = 0; i < 3; ++i) mbar_init(&sm.bar[i], 1);
    mbar_init(&sm.bar_load, 1);
    mbar_init_fence();
  }
  if (warp == 0) tmem_alloc(&sm.tmem, L::kTmemCols);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = sm.tmem;
  const Place<D> me(tid, tmem);
  const StatePlace<D> st(tid);
  const uint32_t state = me.lanes + L::kDS + st.col;
  const size_t state_at = (static_cast<size_t>(bh) * D + st.row) * D + st.c0;

  if (tid == 0) issue_loads<D>(sm, p, bh, b, h, nchunks - 1, nchunks);
  const uint8_t* drow = p.done ? p.done + static_cast<size_t>(b) * p.T : nullptr;
  const size_t bt_base = static_cast<size_t>(b) * p.T;
  Gates gates{};
  if (warp == 1) gates = load_gates(p.alpha, p.beta, bt_base, p.H, h, (nchunks - 1) * kC, p.T, lane);
  linattn::DoneFlags flags = linattn::load_done_flags(drow, (nchunks - 1) * kC, p.T, lane);
#pragma unroll
  for (int c = 0; c < kStateCols; c += 16) {
    float x[16];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
      if (p.ds_last) f = *reinterpret_cast<const float4*>(p.ds_last + state_at + c + 4 * i);
      x[4 * i] = f.x; x[4 * i + 1] = f.y; x[4 * i + 2] = f.z; x[4 * i + 3] = f.w;
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      tmem_st8(state + c + 8 * i, x + 8 * i);
      sm.ds[((st.c0 + c) / 8 + i) * D + st.row] = pack8_bf16(x + 8 * i);
    }
  }
  tmem_st_wait();
  bool timed_out = false;

  for (int it = 0; it < nchunks; ++it) {
    const int c = nchunks - 1 - it;
    const int t0 = c * kC;
    const uint64_t dm = linattn::done_mask_from_flags(flags);
    fence_smem_to_async();   // the bf16 copy of dS is read by products
    fence_before_sync();
    __syncthreads();
    if (warp == 0) {
      const bool leader = elect_one();
      mbar_wait_flag(&sm.bar_load, it & 1, timed_out);
      fence_after_sync();
      product<64, D>(tmem + L::kQK, lines(sm.q, false), lines(sm.k, false), false, leader);
      product<D, D>(tmem + L::kOI, lines(sm.q, false), panels<D>(sm.s, false), false, leader);
      if (leader) commit(&sm.bar[0]);
      product<D, D>(tmem + L::kX2, lines(sm.k, false), panels<D>(sm.ds, false), false, leader);
      product<D, D>(tmem + L::kY, lines(sm.k, false), panels<D>(sm.s, false), false, leader);
      product<64, D>(tmem + L::kKK, lines(sm.k, false), lines(sm.k, false), false, leader);
      product<64, D>(tmem + L::kX, lines(sm.d_o, false), panels<kC>(sm.u, false), false, leader);
      if (lane == 0) tma::wait_group_read<0>();   // the previous chunk's output tiles have left `r1` and `dpg`
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
    const uint32_t seen = keys_seen(dm, me.row, me.j0);
    const float cum_t = sm.cum[me.row], gt = sm.g[me.row], gm = sm.gam[me.row];
    float dg = 0.f;
    {
      float qk[16], oi[kCols];
      tmem_load<16>(me.lanes + L::kQK + me.jcol, qk);
      tmem_load<kCols>(me.lanes + L::kOI + me.col, oi);
      tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 16; ++e) qk[e] *= decay_between(cum_t, sm.cum[me.j0 + e], seen, e);
#pragma unroll
      for (int i = 0; i < 2; ++i) sm.p[((me.j0 >> 3) + i) * kC + me.row] = pack8_bf16(qk + 8 * i);
#pragma unroll
      for (int i = 0; i < kVecs; ++i) {
        float f[8];
        unpack8_bf16(sm.d_o[line_at(me.row, me.ch + i)], f);
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
      product<D, 64>(tmem + L::kX1, panels<kC>(sm.p, true), lines(sm.d_o, true), false, leader);
      if (leader) commit(&sm.bar[1]);
    }
    uint4 u2[kVecs];
#pragma unroll
    for (int i = 0; i < kVecs; ++i) u2[i] = sm.u[(me.ch + i) * kC + me.row];
    mbar_wait_flag(&sm.bar[1], 0, timed_out);
    fence_after_sync();

    // ---- epilogue B ----
    float dgam = 0.f;
    {
      float x1[kCols], x2[kCols];
      tmem_load<kCols>(me.lanes + L::kX2 + me.col, x2);   // (dS k_t)[v]
      tmem_load<kCols>(me.lanes + L::kX1 + me.col, x1);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < kVecs; ++i) {
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
      product<D, 64>(tmem + L::kDR, panels<kC>(sm.tp, true), panels<kC>(sm.r1, true), false, leader);
      if (leader) commit(&sm.bar[2]);
    }
    // meanwhile: <dS, S_in> for the cotangent of g_last, dS <- g_last dS, gam U, g dO in place
    {
      const float g_last = sm.g[kC - 1];
      float dot = 0.f;
      fence_after_sync();
#pragma unroll
      for (int c0 = 0; c0 < kStateCols; c0 += 16) {
        float x[16];
        tmem_load<16>(state + c0, x);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          float f[8];
          unpack8_bf16(sm.s[((st.c0 + c0) / 8 + i) * D + st.row], f);
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            dot = fmaf(x[8 * i + e], f[e], dot);
            x[8 * i + e] *= g_last;
          }
          tmem_st8(state + c0 + 8 * i, x + 8 * i);
        }
      }
#pragma unroll
      for (int off = 16; off >= 1; off >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, off);
      if (lane == 0) sm.dgl[warp] = dot;
#pragma unroll
      for (int i = 0; i < kVecs; ++i) {
        const int line = line_at(me.row, me.ch + i);
        float f[8];
        unpack8_bf16(u2[i], f);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] *= gm;
        sm.gam_u()[(me.ch + i) * kC + me.row] = pack8_bf16(f);
        unpack8_bf16(sm.d_o[line], f);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] *= gt;
        sm.d_o[line] = pack8_bf16(f);
      }
      tmem_st_wait();
    }
    mbar_wait_flag(&sm.bar[2], it & 1, timed_out);
    fence_after_sync();

    // ---- epilogue C ----
    {
      float dr[kCols], y[kCols], dru = 0.f;
      tmem_load<kCols>(me.lanes + L::kDR + me.col, dr);
      tmem_load<kCols>(me.lanes + L::kY + me.col, y);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < kVecs; ++i) {
        const int at = (me.ch + i) * kC + me.row;
        float f[8];
        unpack8_bf16(u2[i], f);
        const uint4 x = pack8_bf16(dr + 8 * i);
        sm.r1[at] = x;
        sm.dv()[line_at(me.row, me.ch + i)] = x;
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
#pragma unroll
        for (int i = 0; i < D / 64; ++i)   // rows past the end of the sequence are clipped
          tma::store_plain_tile(&p.map_dv, sm.dv() + i * kSquareVecs, t0, h, b, 64 * i);
        tma::commit_group();
      }
      __syncwarp();
      product<64, D>(tmem + L::kW, panels<kC>(sm.r1, false), panels<kC>(sm.u, false), false, leader);
      if (leader) commit(&sm.bar[0]);
      // dQ = g dO S_in, dK = gam U dS - g dR S_in, dS_in = g_last dS + (g dO)^T Q - (g dR)^T K
      product_rows<D, D>(tmem + L::kDQK, lines(sm.d_o, false), panels<D>(sm.s, true), false, leader);
      product_rows<D, D>(tmem + kUpperLanes + L::kDQK, panels<kC>(sm.gam_u(), false), panels<D>(sm.ds, true), false, leader);
      product_rows<D, D>(tmem + kUpperLanes + L::kDQK, panels<kC>(sm.r2, false), panels<D>(sm.s, true), true, leader);
      product_state<D>(tmem + L::kDS, lines(sm.d_o, true), lines(sm.q, true), true, leader);
      product_state<D>(tmem + L::kDS, panels<kC>(sm.r2, true), lines(sm.k, true), true, leader);
    }
    mbar_wait_flag(&sm.bar[0], 1, timed_out);
    fence_after_sync();

    // ---- epilogue D ----
    {
      float ev[16], rs = 0.f;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float kk[8], qk[8], x[8], w[8];
        tmem_ld8(me.lanes + L::kKK + me.jcol + 8 * i, kk);
        tmem_ld8(me.lanes + L::kQK + me.jcol + 8 * i, qk);
        tmem_ld8(me.lanes + L::kX + me.jcol + 8 * i, x);
        tmem_ld8(me.lanes + L::kW + me.jcol + 8 * i, w);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int j = me.j0 + 8 * i + e;
          const float gtj = decay_between(cum_t, sm.cum[j], seen, 8 * i + e);
          const float dl = j < me.row ? -w[e] : 0.f;
          ev[8 * i + e] = (x[e] * qk[e] + dl * kk[e]) * gtj;
          rs += ev[8 * i + e];
          x[e] *= gtj;
          w[e] = dl * gtj;
        }
        sm.dpg[((me.j0 >> 3) + i) * kC + me.row] = pack8_bf16(x);
        sm.dlg[((me.j0 >> 3) + i) * kC + me.row] = pack8_bf16(w);
      }
      rs = other_half(rs);
      if (!me.upper) sm.rowsum[wg][me.row] = rs;
      // column sums over this warp's 16 rows: lane l & 15 ends with key j0 + (l & 15)
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
      sm.colsum[warp & 3][me.j0 + (lane & 15)] = ev[0];
    }
    fence_smem_to_async();
    fence_before_sync();
    __syncthreads();
    if (warp == 0) {
      const bool leader = elect_one();
      fence_after_sync();
      product_rows<D, 64>(tmem + L::kDQK, panels<kC>(sm.dpg, false), lines(sm.k, true), true, leader);
      product_rows<D, 64>(tmem + kUpperLanes + L::kDQK, panels<kC>(sm.dpg, true), lines(sm.q, true), true, leader);
      product_rows<D, 64>(tmem + kUpperLanes + L::kDQK, panels<kC>(sm.dlg, false), lines(sm.k, true), true, leader);
      product_rows<D, 64>(tmem + kUpperLanes + L::kDQK, panels<kC>(sm.dlg, true), lines(sm.k, true), true, leader);
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
      if (tid == 0) {
        tma::wait_group_read<0>();   // the dV tile has left `tp`
        issue_loads<D>(sm, p, bh, b, h, c - 1, nchunks);
      }
      if (warp == 1) gates = load_gates(p.alpha, p.beta, bt_base, p.H, h, t0 - kC, p.T, lane);
      flags = linattn::load_done_flags(drow, t0 - kC, p.T, lane);
    }

    // ---- epilogue E: lanes 0..15 hold rows of dQ, lanes 16..31 of dK, half of the columns per warpgroup ----
    {
      uint4* const tile = me.upper ? sm.dpg : sm.r1;
#pragma unroll
      for (int c0 = 0; c0 < D / 2; c0 += 32) {
        float x[32];
        tmem_load<32>(me.lanes + L::kDQK + wg * (D / 2) + c0, x);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 4; ++i) tile[line_at(me.row, (wg * (D / 2) + c0) / 8 + i)] = pack8_bf16(x + 8 * i);
      }
#pragma unroll
      for (int c0 = 0; c0 < kStateCols; c0 += 16) {
        float x[16];
        tmem_load<16>(state + c0, x);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 2; ++i) sm.ds[((st.c0 + c0) / 8 + i) * D + st.row] = pack8_bf16(x + 8 * i);
        if (c == 0 && p.ds0) {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            *reinterpret_cast<float4*>(p.ds0 + state_at + c0 + 4 * i) = make_float4(x[4 * i], x[4 * i + 1], x[4 * i + 2], x[4 * i + 3]);
        }
      }
    }
    fence_smem_to_async();
    fence_before_sync();
    __syncthreads();
    if (tid == 0) {
#pragma unroll
      for (int i = 0; i < D / 64; ++i) {
        tma::store_plain_tile(&p.map_dq, sm.r1 + i * kSquareVecs, t0, h, b, 64 * i);
        tma::store_plain_tile(&p.map_dk, sm.dpg + i * kSquareVecs, t0, h, b, 64 * i);
      }
      tma::commit_group();
    }
  }
  if (tid == 0) tma::wait_group_all();
  if (timed_out && p.status) atomicExch(p.status, 1);
  fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, L::kTmemCols);
}

template <int D>
int launch_backward(const BwdParams& p, int sequences, cudaStream_t stream) {
  cudaError_t e = cudaFuncSetAttribute(gdelta_bwd_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(sizeof(BwdSmem<D>)));
  if (e != cudaSuccess) return static_cast<int>(e);
  mxk::launch_kernel(gdelta_bwd_kernel<D>, sequences, kBwdThreads, sizeof(BwdSmem<D>), stream, p);
  return launch_status();
}

}  // namespace

namespace gdelta {

int backward(const void* q, const void* k, const void* v, const float* alpha, const float* beta,
                        const void* d_o, const void* chunk_states, const void* workspace, const uint8_t* done,
                        const float* ds_last,
                        void* dq, void* dk, void* dv, long long ld_dv, float* dalpha, float* dbeta, float* ds0, int* status,
                        int B, int T, int H, int d, cudaStream_t stream) {
  if (!q || !k || !v || !alpha || !beta || !d_o || !chunk_states || !workspace || !dq || !dk || !dv || !dalpha || !dbeta)
    return MXK_ERR_NULL;
  if (B <= 0 || T <= 0 || H <= 0 || static_cast<long long>(B) * H > 0x7fffffffLL) return MXK_ERR_DIMS;
  if (d != 128 && d != 64) return MXK_ERR_UNSUPPORTED;
  for (const void* ptr : {q, k, v, d_o, chunk_states, workspace, (const void*)dq, (const void*)dk, (const void*)dv,
                          (const void*)ds_last, (const void*)ds0})
    if (ptr && !aligned16(ptr)) return MXK_ERR_ALIGN;
  BwdParams prm{alpha, beta, done, static_cast<const uint4*>(chunk_states), static_cast<const uint4*>(workspace), ds_last, dalpha, dbeta, ds0,
                status, T, H};
  if (!tma::make_sw_map(&prm.map_k, k, B, T, H, kC, d) || !tma::make_sw_map(&prm.map_q, q, B, T, H, kC, d) ||
      !tma::make_sw_map(&prm.map_do, d_o, B, T, H, kC, d) || !tma::make_sw_map(&prm.map_dq, dq, B, T, H, kC, d) ||
      !tma::make_sw_map(&prm.map_dk, dk, B, T, H, kC, d) || !tma::make_sw_map(&prm.map_dv, dv, B, T, H, kC, d, ld_dv))
    return MXK_ERR_UNSUPPORTED;
  return d == 64 ? launch_backward<64>(prm, B * H, stream) : launch_backward<128>(prm, B * H, stream);
}

}  // namespace gdelta
}  // namespace mxk

extern "C" {

int mxk_gdelta_bf16_bwd(const void* q, const void* k, const void* v, const float* alpha, const float* beta,
                        const void* d_o, const void* chunk_states, const void* workspace, const uint8_t* done,
                        const float* ds_last,
                        void* dq, void* dk, void* dv, float* dalpha, float* dbeta, float* ds0, int* status,
                        int B, int T, int H, int d, mxk_stream_t stream) {
  return mxk::gdelta::backward(q, k, v, alpha, beta, d_o, chunk_states, workspace, done, ds_last, dq, dk, dv, 0, dalpha, dbeta, ds0,
                               status, B, T, H, d, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
