// Gated delta rule, forward, on the sm_100a tensor cores (math and layout in gdelta_common.cuh).
//
// One CTA (256 threads) owns one (batch, head) sequence and walks its 64-token chunks in order with the fp32 state S (D x D)
// resident in tensor memory; K, Q, V (128-byte-swizzled lines) arrive by TMA one chunk ahead, as does the chunk's
// T' = (I + diag(beta) L)^-1 diag(beta) from the preparation kernel (gdelta_prep.cu), so the state-serial chain holds no
// triangular solve, only products:
//   products 1: Q K^T, Y = K S_in^T (one warp computes the chunk's decay meanwhile)
//   epilogue 1: P = tril(G o QK^T), -g Y (bf16 operands), Q and K rescaled in place (g Q, gam K)
//   products 2: U = T' V - T' (g Y), then O = (g Q) S_in^T, which epilogue 2 need not wait for; S <- g_last S meanwhile
//   epilogue 2: U as bf16 operand and as the backward pass's residual
//   products 3: O += P U, S += U^T (gam K)
//   epilogue 3: output tile (one TMA store), bf16 operand copy of the new state
// Bound: the serial chain of three groups of products a chunk, hidden by two (D = 128) or three (D = 64) CTAs per SM.
// Measured: 512 x 256 steps, 8 heads of 64: 222 us (408 padded to 128); 128 x 512 steps, 8 heads of 128: 222 us (229 with
// features on the rows).
#include <cstddef>

#include "attention.cuh"
#include "gdelta_common.cuh"

namespace mxk {
namespace {

using namespace gdelta;

struct FwdParams {
  const float* alpha;
  const float* s0;
  const uint8_t* done;
  float* s_last;
  uint4* residual;            // nullptr: not kept
  const uint4* tprime;        // T' of every chunk, written by the preparation kernel
  int* status;
  int T, H;
  CUtensorMap map_k, map_q, map_v, map_o;   // 64-token tiles as lines
};

template <int D>
struct FwdSmem {
  uint4 s[state_vecs(D)];    // S_in                           [k/8][v][8]
  uint4 k[tile_vecs(D)];     // K, after products 1 gam K      (lines)
  uint4 q[tile_vecs(D)];     // Q, after products 1 g Q        (lines)
  uint4 v[tile_vecs(D)];     // V                              (lines)
  uint4 yu[tile_vecs(D)];    // -g Y, then U [v/8][t][8], then the output tile (lines)
  uint4 p[kSquareVecs];      // P                              [j/8][t][8]
  uint4 tp[kSquareVecs];     // T'                             [j/8][t][8]
  float cum[kC], g[kC], gam[kC];
  uint64_t bar[3];
  uint64_t bar_load;
  uint32_t tmem;
};
template <int D>
struct FwdLayout {
  static constexpr int kPerSm = D == 64 ? 3 : 2;
  static constexpr uint32_t kTmemCols = D == 64 ? 128 : 256;
  // Q K^T shares the columns of U, and O those of Y
  static constexpr uint32_t kS = 0, kY = D == 64 ? 32 : 128, kU = kY + D / 2, kQK = kU, kO = kY;
  static_assert(kPerSm * (sizeof(FwdSmem<D>) + 1024) <= 228 * 1024 && kPerSm * kTmemCols <= 512, "CTAs per SM");
};

constexpr int kFwdThreads = 256;

template <int D>
__device__ __forceinline__ void issue_loads(FwdSmem<D>& sm, const FwdParams& p, int bh, int b, int h, int c, int nchunks) {
  fence_smem_to_async();   // earlier accesses by threads to the buffers come first
  tma::expect_bytes(&sm.bar_load, (3 * tile_vecs(D) + kAinvVecs) * 16);
  const int t0 = c * kC;
  const uint4* tp = p.tprime + (static_cast<size_t>(bh) * nchunks + c) * kAinvVecs;
#pragma unroll
  for (int i = 0; i < D / 64; ++i) {
    tma::load_plain_tile(sm.k + i * kSquareVecs, &p.map_k, &sm.bar_load, t0, h, b, 64 * i);
    tma::load_plain_tile(sm.q + i * kSquareVecs, &p.map_q, &sm.bar_load, t0, h, b, 64 * i);
    tma::load_plain_tile(sm.v + i * kSquareVecs, &p.map_v, &sm.bar_load, t0, h, b, 64 * i);
  }
  tma::load_bulk(sm.tp, tp, kAinvVecs * 16, &sm.bar_load);
  if (c + 1 < nchunks) {   // the chunk after it: into L2 now
#pragma unroll
    for (int i = 0; i < D / 64; ++i) {
      tma::prefetch_plain_tile(&p.map_k, t0 + kC, h, b, 64 * i);
      tma::prefetch_plain_tile(&p.map_q, t0 + kC, h, b, 64 * i);
      tma::prefetch_plain_tile(&p.map_v, t0 + kC, h, b, 64 * i);
    }
    tma::prefetch_bulk(tp + kAinvVecs, kAinvVecs * 16);
  }
}

template <int D>
__global__ void __launch_bounds__(kFwdThreads, FwdLayout<D>::kPerSm) gdelta_fwd_kernel(const __grid_constant__ FwdParams p) {
  enter_kernel();
  using L = FwdLayout<D>;
  constexpr int kVecs = Place<D>::kVecs, kStateCols = StatePlace<D>::kCols;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  FwdSmem<D>& sm = *reinterpret_cast<FwdSmem<D>*>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
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
  const uint32_t state = me.lanes + L::kS + st.col;
  const size_t state_at = (static_cast<size_t>(bh) * D + st.row) * D + st.c0;

  if (tid == 0) issue_loads<D>(sm, p, bh, b, h, 0, nchunks);
  const uint8_t* drow = p.done ? p.done + static_cast<size_t>(b) * p.T : nullptr;
  const size_t bt_base = static_cast<size_t>(b) * p.T;
  Gates gates{};
  if (warp == 1) gates = load_gates(p.alpha, nullptr, bt_base, p.H, h, 0, p.T, lane);
  linattn::DoneFlags flags = linattn::load_done_flags(drow, 0, p.T, lane);
#pragma unroll
  for (int c = 0; c < kStateCols; c += 16) {
    float x[16];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
      if (p.s0) f = *reinterpret_cast<const float4*>(p.s0 + state_at + c + 4 * i);
      x[4 * i] = f.x; x[4 * i + 1] = f.y; x[4 * i + 2] = f.z; x[4 * i + 3] = f.w;
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      tmem_st8(state + c + 8 * i, x + 8 * i);
      sm.s[((st.c0 + c) / 8 + i) * D + st.row] = pack8_bf16(x + 8 * i);
    }
  }
  tmem_st_wait();
  bool timed_out = false;

  for (int c = 0; c < nchunks; ++c) {
    const int t0 = c * kC;
    const uint64_t dm = linattn::done_mask_from_flags(flags);
    fence_smem_to_async();   // the bf16 state copy is read by a bulk copy and by products
    fence_before_sync();
    __syncthreads();
    if (warp == 0) {
      const bool leader = elect_one();
      if (lane == 0 && p.residual) {   // for the backward pass: the state entering the chunk
        tma::store_bulk(p.residual + (static_cast<size_t>(bh) * nchunks + c) * residual_vecs(D), sm.s, state_vecs(D) * 16);
        tma::commit_group();
      }
      mbar_wait_flag(&sm.bar_load, c & 1, timed_out);
      fence_after_sync();
      product<64, D>(tmem + L::kQK, lines(sm.q, false), lines(sm.k, false), false, leader);
      product<D, D>(tmem + L::kY, lines(sm.k, false), panels<D>(sm.s, false), false, leader);
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
      const uint32_t seen = keys_seen(dm, me.row, me.j0);
      const float cum_t = sm.cum[me.row], gt = sm.g[me.row], gm = sm.gam[me.row];
      float qk[16], y[8 * kVecs];
      tmem_load<16>(me.lanes + L::kQK + me.jcol, qk);
      tmem_load<8 * kVecs>(me.lanes + L::kY + me.col, y);
      tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 16; ++e) qk[e] *= decay_between(cum_t, sm.cum[me.j0 + e], seen, e);
#pragma unroll
      for (int i = 0; i < 2; ++i) sm.p[((me.j0 >> 3) + i) * kC + me.row] = pack8_bf16(qk + 8 * i);
#pragma unroll
      for (int i = 0; i < kVecs; ++i) {
        const int line = line_at(me.row, me.ch + i);
        float f[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = -gt * y[8 * i + e];
        sm.yu[(me.ch + i) * kC + me.row] = pack8_bf16(f);
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
      product<D, 64>(tmem + L::kU, panels<kC>(sm.tp, false), lines(sm.v, true), false, leader);
      product<D, 64>(tmem + L::kU, panels<kC>(sm.tp, false), panels<kC>(sm.yu, true), true, leader);
      if (leader) commit(&sm.bar[2]);
      product<D, D>(tmem + L::kO, lines(sm.q, false), panels<D>(sm.s, false), false, leader);
    }
    {
      const float g_last = sm.g[kC - 1];
      fence_after_sync();
#pragma unroll
      for (int c0 = 0; c0 < kStateCols; c0 += 16) {
        float x[16];
        tmem_load<16>(state + c0, x);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e) x[e] *= g_last;
        tmem_st8(state + c0, x);
        tmem_st8(state + c0 + 8, x + 8);
      }
      tmem_st_wait();
    }
    mbar_wait_flag(&sm.bar[2], c & 1, timed_out);
    fence_after_sync();

    {
      uint4* res = p.residual ? p.residual + (static_cast<size_t>(bh) * nchunks + c) * residual_vecs(D) + state_vecs(D) : nullptr;
      float u[8 * kVecs];
      tmem_load<8 * kVecs>(me.lanes + L::kU + me.col, u);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < kVecs; ++i) {
        const uint4 x = pack8_bf16(u + 8 * i);
        sm.yu[(me.ch + i) * kC + me.row] = x;
        if (res) res[(me.ch + i) * kC + me.row] = x;
      }
    }
    if (tid == 0) tma::wait_group_read<0>();   // the residual copy has finished reading `s` (rewritten in epilogue 3)
    fence_smem_to_async();
    fence_before_sync();
    __syncthreads();
    if (warp == 0) {
      const bool leader = elect_one();
      fence_after_sync();
      product<D, 64>(tmem + L::kO, panels<kC>(sm.p, false), panels<kC>(sm.yu, true), true, leader);
      product_state<D>(tmem + L::kS, panels<kC>(sm.yu, true), lines(sm.k, true), true, leader);
      if (leader) commit(&sm.bar[1]);
    }
    mbar_wait_flag(&sm.bar[1], c & 1, timed_out);
    fence_after_sync();
    const bool last = c + 1 == nchunks;
    if (!last) {
      if (tid == 0) issue_loads<D>(sm, p, bh, b, h, c + 1, nchunks);
      if (warp == 1) gates = load_gates(p.alpha, nullptr, bt_base, p.H, h, t0 + kC, p.T, lane);
      flags = linattn::load_done_flags(drow, t0 + kC, p.T, lane);
    }
    {
      float o[8 * kVecs];
      tmem_load<8 * kVecs>(me.lanes + L::kO + me.col, o);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < kVecs; ++i) sm.yu[line_at(me.row, me.ch + i)] = pack8_bf16(o + 8 * i);
    }
#pragma unroll
    for (int c0 = 0; c0 < kStateCols; c0 += 16) {
      float x[16];
      tmem_load<16>(state + c0, x);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 2; ++i) sm.s[((st.c0 + c0) / 8 + i) * D + st.row] = pack8_bf16(x + 8 * i);
      if (last && p.s_last) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<float4*>(p.s_last + state_at + c0 + 4 * i) = make_float4(x[4 * i], x[4 * i + 1], x[4 * i + 2], x[4 * i + 3]);
      }
    }
    fence_smem_to_async();
    fence_before_sync();
    __syncthreads();
    if (tid == 0) {
#pragma unroll
      for (int i = 0; i < D / 64; ++i)   // rows past the end of the sequence are clipped
        tma::store_plain_tile(&p.map_o, sm.yu + i * kSquareVecs, t0, h, b, 64 * i);
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
int launch_forward(const FwdParams& p, int sequences, cudaStream_t stream) {
  cudaError_t e = cudaFuncSetAttribute(gdelta_fwd_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(sizeof(FwdSmem<D>)));
  if (e != cudaSuccess) return static_cast<int>(e);
  mxk::launch_kernel(gdelta_fwd_kernel<D>, sequences, kFwdThreads, sizeof(FwdSmem<D>), stream, p);
  return launch_status();
}

}  // namespace

namespace gdelta {

int forward(const void* q, const void* k, const void* v, long long ld_v, const float* alpha, const float* beta,
            const float* s0, const uint8_t* done, void* o, float* s_last, void* chunk_states,
            void* workspace, size_t workspace_bytes, int* status, int B, int T, int H, int d,
            cudaStream_t stream) {
  if (!q || !k || !v || !alpha || !beta || !o) return MXK_ERR_NULL;
  if (B <= 0 || T <= 0 || H <= 0 || static_cast<long long>(B) * H > 0x7fffffffLL) return MXK_ERR_DIMS;
  if (d != 128 && d != 64) return MXK_ERR_UNSUPPORTED;
  for (const void* ptr : {q, k, v, (const void*)o, (const void*)chunk_states, (const void*)s0, (const void*)s_last})
    if (ptr && !aligned16(ptr)) return MXK_ERR_ALIGN;
  if (!workspace || workspace_bytes < mxk_gdelta_workspace_bytes(B, T, H, d)) return MXK_ERR_WORKSPACE;
  if (!aligned16(workspace)) return MXK_ERR_ALIGN;
  FwdParams prm{alpha, s0, done, s_last, static_cast<uint4*>(chunk_states), static_cast<const uint4*>(workspace), status, T, H};
  if (!tma::make_sw_map(&prm.map_k, k, B, T, H, kC, d) || !tma::make_sw_map(&prm.map_q, q, B, T, H, kC, d) ||
      !tma::make_sw_map(&prm.map_v, v, B, T, H, kC, d, ld_v) || !tma::make_sw_map(&prm.map_o, o, B, T, H, kC, d))
    return MXK_ERR_UNSUPPORTED;
  const int st = launch_prep(k, alpha, beta, done, workspace, status, B, T, H, d, stream);
  if (st != MXK_OK) return st;
  return d == 64 ? launch_forward<64>(prm, B * H, stream) : launch_forward<128>(prm, B * H, stream);
}

}  // namespace gdelta
}  // namespace mxk

extern "C" {

size_t mxk_gdelta_chunk_states_bytes(int B, int T, int H, int d) {
  if (B <= 0 || T <= 0 || H <= 0 || (d != 128 && d != 64)) return 0;
  const size_t nchunks = (static_cast<size_t>(T) + mxk::gdelta::kC - 1) / mxk::gdelta::kC;
  return static_cast<size_t>(B) * H * nchunks * mxk::gdelta::residual_vecs(d) * sizeof(uint4);
}

size_t mxk_gdelta_workspace_bytes(int B, int T, int H, int d) {
  if (B <= 0 || T <= 0 || H <= 0 || (d != 128 && d != 64)) return 0;
  const size_t nchunks = (static_cast<size_t>(T) + mxk::gdelta::kC - 1) / mxk::gdelta::kC;
  return static_cast<size_t>(B) * H * nchunks * mxk::gdelta::kAinvVecs * sizeof(uint4);
}

int mxk_gdelta_bf16_fwd(const void* q, const void* k, const void* v, const float* alpha, const float* beta,
                        const float* s0, const uint8_t* done, void* o, float* s_last, void* chunk_states,
                        void* workspace, size_t workspace_bytes, int* status, int B, int T, int H, int d,
                        mxk_stream_t stream) {
  return mxk::gdelta::forward(q, k, v, 0, alpha, beta, s0, done, o, s_last, chunk_states, workspace, workspace_bytes, status, B, T,
                              H, d, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
