// Gated delta rule, chunk-parallel preparation: everything of the chunked form that does not depend on
// the carried state, computed for all chunks at once so that the state-serial kernels need no
// triangular solve.
//
// Persistent CTAs (128 threads) over the (batch, head, 64-token chunk) items, the next item's K, gates and resets in flight
// under the present one's solve (a CTA per item took 21 k cycles, most of them waits;
// 128 x 512 steps, 8 heads of 128: 145 -> 104 us).  With the chunk quantities of
// gdelta_common.cuh (L = strict_tril(G o K K^T), A = I + diag(beta) L):
//   K K^T  on the tensor core (two N = 32 halves, so that each thread owns 32 keys of one token row),
//   N = -beta L in fp32 in shared memory, transposed,
//   A^-1 = (I - N)^-1 in fp32 by block recursion, every step using all four warps and no step longer than a
//          16-row chain: the four 16 x 16 diagonal blocks by forward substitution (one column per thread),
//          then  X_pq = X_pp N_pq X_qq  for the two 16 x 16 blocks under the diagonal of each 32 x 32 half,
//          then the same formula for the lower-left 32 x 32 block (the inverse of a block lower-triangular
//          matrix [[A11, 0], [A21, A22]] has -A22^-1 A21 A11^-1 there, and A21 = -N21).  A column-per-thread
//          substitution over all 64 rows would leave three warps idle behind a 63-step dependent chain.
//   T' = A^-1 diag(beta) leaves as bf16 in tensor-core operand order, [j/8][t][8] with t the row and
//          j the column.
// The forward kernel then forms U = T' (V - diag(g) K S_in^T) and the backward kernel dR = T'^T dU as
// plain tensor-core products.
#include "gdelta_common.cuh"
#include "tma.cuh"

namespace mxk {
namespace {

using namespace umma;
using namespace gdelta;

struct PrepParams {
  const float* alpha;
  const float* beta;
  const uint8_t* done;
  uint4* ainv;   // out: T', kAinvVecs uint4 per (b, h, chunk)
  int* status;
  int T, H, nchunks, items;
  int blocks;          // 64-column blocks of a head: 1 or 2
  CUtensorMap map_k;   // 64-token tiles as SW tiles (two 64-column blocks)
};

// Row stride of the fp32 matrices: rows 16-byte aligned, and eight of them spread their 16-byte vectors over all banks.
// Scalar accesses at an odd stride made 950 shared-memory wavefronts a warp and chunk, these make about 380.
constexpr int kXS = kC + 4;
// lt[j][t]; rows from 32 on shifted by 16 so that a warp, writing rows j and j + 32 at once, meets no bank twice
__device__ __forceinline__ int lt_at(int j) { return j * kC + (j & 32) / 2; }

struct PrepSmem {
  union {
    float lt[kC * kC + 16];   // lt[j][t] = N[t][j] = -beta_t L_tj
    uint4 tp[kAinvVecs];      // the staged bf16 T', [j/8][t][8]
  };
  float x[kC * kXS];          // A^-1, row-major; its upper right 32 x 32 block, zero by definition, holds M = N_pq X_qq
  float cum[kC], beta[kC];
  uint64_t bar_load, bar_mma;
  uint32_t tmem;
  alignas(1024) uint4 k[2 * kSquareVecs];   // K, SW tiles (one or two 64-column blocks)
};
constexpr int smem_bytes(int blocks) { return static_cast<int>(offsetof(PrepSmem, k)) + blocks * kSquareVecs * 16; }
static_assert(smem_bytes(1) <= 44 * 1024 && smem_bytes(2) <= 56 * 1024, "five CTAs per SM for heads of 64, four for 128");

#ifdef MXK_TIMING
}  // namespace
__device__ unsigned long long g_gdp_phase_cycles[16];
namespace {
#define MXK_TP(i) do { if (tid == 0 && (blockIdx.x % 37) == 0) { const long long now_ = clock64(); atomicAdd(&g_gdp_phase_cycles[i], (unsigned long long)(now_ - t_prev_)); t_prev_ = now_; } } while (0)
#else
#define MXK_TP(i) do {} while (0)
#endif
constexpr uint32_t kPrepTmemCols = 32;
constexpr int kThreads = 128;

// acc[0 .. 1] += a * (four consecutive values)
__device__ __forceinline__ void axpy(float a, float4 x, float2* acc) {
  const float2 a2 = make_float2(a, a);
  acc[0] = __ffma2_rn(a2, make_float2(x.x, x.y), acc[0]);
  acc[1] = __ffma2_rn(a2, make_float2(x.z, x.w), acc[1]);
}

__global__ void __launch_bounds__(kThreads, 5) gdelta_prep_kernel(const __grid_constant__ PrepParams p) {
  enter_kernel();
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  PrepSmem& sm = *reinterpret_cast<PrepSmem*>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool upper = lane >= 16;
  const int row = warp * 16 + (lane & 15);   // token row owned in the accumulator

#ifdef MXK_TIMING
  long long t_prev_ = clock64();
#endif
  if (tid == 0) {
    mbar_init(&sm.bar_load, 1);
    mbar_init(&sm.bar_mma, 1);
    mbar_init_fence();
  }
  if (warp == 0) tmem_alloc(&sm.tmem, kPrepTmemCols);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = sm.tmem;
  const uint32_t lane_base = tmem + (static_cast<uint32_t>(warp * 32) << 16);
  bool timed_out = false;
  MXK_TP(0);

  Gates gates{};
  linattn::DoneFlags flags;
  const auto fetch = [&](int item) {
    const int c = item % p.nchunks, bh = item / p.nchunks, b = bh / p.H, h = bh % p.H, t0 = c * kC;
    if (tid == 0) {
      tma::expect_bytes(&sm.bar_load, p.blocks * kSquareVecs * 16);
      for (int i = 0; i < p.blocks; ++i) tma::load_plain_tile(sm.k + i * kSquareVecs, &p.map_k, &sm.bar_load, t0, h, b, 64 * i);
    }
    if (warp == 1) gates = load_gates(p.alpha, p.beta, static_cast<size_t>(b) * p.T, p.H, h, t0, p.T, lane);
    flags = linattn::load_done_flags(p.done ? p.done + static_cast<size_t>(b) * p.T : nullptr, t0, p.T, lane);
  };
  float* const xm = sm.x;
  float* const mm = sm.x + 32;
  for (int i = tid; i < kC * kXS / 4; i += kThreads) reinterpret_cast<float4*>(xm)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  fetch(blockIdx.x);

  int turn = 0;
  for (int item = blockIdx.x; item < p.items; item += gridDim.x, ++turn) {
    const uint64_t dm = linattn::done_mask_from_flags(flags);
    if (warp == 0) {
      const bool leader = elect_one();
      const uint32_t id_half = idesc_bf16(kC, 32, false, false);
      mbar_wait_flag(&sm.bar_load, turn & 1, timed_out);
      fence_after_sync();
      // keys 0..31 land in lanes 0..15 of each warp's TMEM quarter, keys 32..63 in lanes 16..31 of the same columns
      for (int i = 0; i < p.blocks; ++i) {
        const uint32_t at = smem_u32(sm.k + i * kSquareVecs);
        gemm<4>(tmem, sw_operand(at, false), sw_operand(at, false), id_half, i > 0, leader);
        gemm<4>(tmem + kUpperLanes, sw_operand(at, false), sw_operand(at + 32 * 128, false), id_half, i > 0, leader);
      }
      if (leader) commit(&sm.bar_mma);
      if (tid == 0) tma::wait_group_read<0>();   // the previous T' has left `tp`
      __syncwarp();
    } else if (warp == 1) {
      const float2 cum = cumulative(gates, lane);
      *reinterpret_cast<float2*>(&sm.cum[2 * lane]) = cum;
      *reinterpret_cast<float2*>(&sm.beta[2 * lane]) = make_float2(gates.b[0], gates.b[1]);
    }
    __syncthreads();
    MXK_TP(1);
    mbar_wait_flag(&sm.bar_mma, turn & 1, timed_out);
    fence_after_sync();
    if (item + gridDim.x < p.items) fetch(item + gridDim.x);   // (K has been read)
    MXK_TP(3);

    // -beta L, transposed: every thread owns 32 keys of its token row
    {
      const float cum_t = sm.cum[row], nb = -sm.beta[row];
      const int j0 = upper ? 32 : 0;
      const uint32_t seen = keys_seen(dm, row, j0) & ~static_cast<uint32_t>((1ull << row) >> j0);   // (strictly earlier keys)
      float* const dst = &sm.lt[lt_at(j0) + row];
      float kk[32];
      tmem_ld_row<32>(lane_base, kk);
#pragma unroll
      for (int e4 = 0; e4 < 32; e4 += 4) {
        const float4 c4 = *reinterpret_cast<const float4*>(&sm.cum[j0 + e4]);
        const float cj[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
        for (int e = e4; e < e4 + 4; ++e) dst[e * kC] = nb * decay_between(cum_t, cj[e - e4], seen, e) * kk[e];
      }
      fence_before_sync();
    }
    __syncthreads();

    MXK_TP(4);
    // ---- A^-1 = (I - N)^-1 by block recursion (N[t][j] = lt[j][t]) ----
    const auto vec = [](const float* at) { return *reinterpret_cast<const float4*>(at); };
    // (1) the four 16 x 16 diagonal blocks: thread (p, c) solves column c of block p
    if (tid < kC) {
      const int p0 = (tid >> 4) * 16, c = tid & 15;
      float xc[16];
#pragma unroll
      for (int t = 0; t < 16; ++t) xc[t] = (t == c) ? 1.f : 0.f;
#pragma unroll
      for (int jj = 0; jj < 15; ++jj) {
        const float uj = xc[jj];
#pragma unroll
        for (int m = (jj + 1) / 4; m < 4; ++m) {   // (rows up to jj of this column are zero)
          const float4 l = vec(&sm.lt[lt_at(p0 + jj) + p0 + 4 * m]);
          xc[4 * m] = fmaf(l.x, uj, xc[4 * m]);
          xc[4 * m + 1] = fmaf(l.y, uj, xc[4 * m + 1]);
          xc[4 * m + 2] = fmaf(l.z, uj, xc[4 * m + 2]);
          xc[4 * m + 3] = fmaf(l.w, uj, xc[4 * m + 3]);
        }
      }
#pragma unroll
      for (int t = 0; t < 16; ++t) xm[(p0 + t) * kXS + p0 + c] = xc[t];
    }
    __syncthreads();
    // (2) X_pq = X_pp (N_pq X_qq) for (p, q) = (1, 0) and (3, 2): 64 threads per pair, thread = (row r, 4 columns)
    {
      const int pair = tid >> 6, r = tid & 15, c0 = ((tid >> 4) & 3) * 4;
      const int q0 = pair * 32, p0 = q0 + 16;
      float2 acc[2] = {}, out[2] = {};
#pragma unroll
      for (int kk = 0; kk < 16; ++kk) {
        const float a = sm.lt[lt_at(q0 + kk) + p0 + r];          // N[p0 + r][q0 + kk]
        axpy(a, vec(&xm[(q0 + kk) * kXS + q0 + c0]), acc);
      }
      *reinterpret_cast<float4*>(&mm[(pair * 16 + r) * kXS + c0]) = make_float4(acc[0].x, acc[0].y, acc[1].x, acc[1].y);
      __syncthreads();
#pragma unroll
      for (int k4 = 0; k4 < 4; ++k4) {
        const float4 a = vec(&xm[(p0 + r) * kXS + p0 + 4 * k4]);   // X_pp[r][4 k4 ..]
        const float* const mr = &mm[(pair * 16 + 4 * k4) * kXS + c0];
        axpy(a.x, vec(mr), out);
        axpy(a.y, vec(mr + kXS), out);
        axpy(a.z, vec(mr + 2 * kXS), out);
        axpy(a.w, vec(mr + 3 * kXS), out);
      }
      __syncthreads();   // every read of mm and of the diagonal blocks is done before anything is overwritten
      *reinterpret_cast<float4*>(&xm[(p0 + r) * kXS + q0 + c0]) = make_float4(out[0].x, out[0].y, out[1].x, out[1].y);
    }
    __syncthreads();
    // (3) the lower-left 32 x 32 block: X_PQ = X_PP (N_PQ X_QQ), thread = (row r of 32, 8 columns)
    {
      const int r = tid & 31, c0 = (tid >> 5) * 8;
      float2 acc[4] = {}, out[4] = {};
#pragma unroll 8
      for (int kk = 0; kk < 32; ++kk) {
        const float a = sm.lt[lt_at(kk) + 32 + r];                 // N[32 + r][kk]
        axpy(a, vec(&xm[kk * kXS + c0]), acc);
        axpy(a, vec(&xm[kk * kXS + c0 + 4]), acc + 2);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
        *reinterpret_cast<float4*>(&mm[r * kXS + c0 + 4 * i]) = make_float4(acc[2 * i].x, acc[2 * i].y, acc[2 * i + 1].x, acc[2 * i + 1].y);
      __syncthreads();
#pragma unroll 2
      for (int k4 = 0; k4 < 8; ++k4) {
        const float4 a4 = vec(&xm[(32 + r) * kXS + 32 + 4 * k4]);   // X_PP[r][4 k4 ..]
        const float a[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          axpy(a[e], vec(&mm[(4 * k4 + e) * kXS + c0]), out);
          axpy(a[e], vec(&mm[(4 * k4 + e) * kXS + c0 + 4]), out + 2);
        }
      }
      // (the block written here is read by nobody above)
#pragma unroll
      for (int i = 0; i < 2; ++i)
        *reinterpret_cast<float4*>(&xm[(32 + r) * kXS + c0 + 4 * i]) = make_float4(out[2 * i].x, out[2 * i].y, out[2 * i + 1].x, out[2 * i + 1].y);
    }
    __syncthreads();
    MXK_TP(5);
    // T' = A^-1 diag(beta) as bf16, [j/8][t][8]: thread (t, half) packs four groups of eight columns
    {
      uint4* out = sm.tp;
      const int t = tid & 63, g0 = (tid >> 6) * 4;
#pragma unroll
      for (int gq = 0; gq < 4; ++gq) {
        const int j = (g0 + gq) * 8;
        float f[8];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float4 x = vec(&xm[t * kXS + j + 4 * i]), be = vec(&sm.beta[j + 4 * i]);
          f[4 * i] = x.x * be.x; f[4 * i + 1] = x.y * be.y; f[4 * i + 2] = x.z * be.z; f[4 * i + 3] = x.w * be.w;
        }
        if (t < 32 && j >= 32) {   // (M was there)
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] = 0.f;
        }
        out[(g0 + gq) * kC + t] = pack8_bf16(f);
      }
    }
    fence_smem_to_async();
    __syncthreads();
    MXK_TP(6);
    if (tid == 0) {
      tma::store_bulk(p.ainv + static_cast<size_t>(item) * kAinvVecs, sm.tp, kAinvVecs * 16);
      tma::commit_group();
    }
    MXK_TP(7);
  }
  if (tid == 0) tma::wait_group_all();
  if (timed_out && p.status) atomicExch(p.status, 1);
  fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, kPrepTmemCols);
}

}  // namespace

#ifdef MXK_TIMING
}  // namespace mxk
extern "C" int mxk_debug_gdp_phase_cycles(unsigned long long* out, int reset) {
  if (reset) {
    unsigned long long z[16] = {};
    return (int)cudaMemcpyToSymbol(mxk::g_gdp_phase_cycles, z, sizeof(z));
  }
  return (int)cudaMemcpyFromSymbol(out, mxk::g_gdp_phase_cycles, 16 * sizeof(unsigned long long));
}
namespace mxk {
#endif

namespace gdelta {

int launch_prep(const void* k, const float* alpha, const float* beta, const uint8_t* done, void* ainv, int* status,
                int B, int T, int H, int d, cudaStream_t stream) {
  PrepParams prm;
  prm.alpha = alpha;
  prm.beta = beta;
  prm.done = done;
  prm.ainv = static_cast<uint4*>(ainv);
  prm.status = status;
  prm.T = T; prm.H = H;
  prm.nchunks = (T + kC - 1) / kC;
  prm.blocks = d / 64;
  if (!tma::make_sw_map(&prm.map_k, k, B, T, H, kC, d)) return MXK_ERR_UNSUPPORTED;
  const long long items = static_cast<long long>(B) * H * prm.nchunks;
  const int most = kNumSMs * (prm.blocks == 1 ? 5 : 4);   // one wave
  if (items > 0x7fffffffLL - most) return MXK_ERR_DIMS;
  prm.items = static_cast<int>(items);
  cudaError_t e = cudaFuncSetAttribute(gdelta_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes(2));
  if (e != cudaSuccess) return static_cast<int>(e);
  mxk::launch_kernel(gdelta_prep_kernel, static_cast<unsigned>(items < most ? items : most), kThreads, smem_bytes(prm.blocks), stream, prm);
  return launch_status();
}

}  // namespace gdelta
}  // namespace mxk
