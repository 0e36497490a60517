// bf16 matrix products on tcgen05 for the layers' middle sizes, where a library call costs more on the host (about 30 us
// through the framework) than the product takes: operands by TMA in swizzled tiles, contracted over either index without
// transposing, batched (the block-diagonal projections of a head), split along long contractions (weight gradients).
//
// One persistent CTA per SM: warp 0 issues the TMA loads (4 stages of 64 k), warp 1 the MMAs (M = 128, N = 64 or 128),
// warps 2..5 drain the accumulators, double-buffered in tensor memory, one row per thread with 32-byte stores.
// Bound: L2 -> SM bandwidth at these tiles (a 128 x 128 x 64 step reads 32 KB for 256 cycles of the pipe), which is why
// the largest products stay with the library's two-SM tiles.
#include <cuda_bf16.h>

#include "gemm16.cuh"
#include "mxk_common.cuh"
#include "tma.cuh"
#include "umma.cuh"

namespace mxk {
namespace gemm16 {
namespace {

using namespace umma;

constexpr int kBM = 128, kBK = 64, kStages = 4, kThreads = 192;

struct Params {
  CUtensorMap map_a, map_b;
  __nv_bfloat16* c;
  const __nv_bfloat16* bias;
  float* partial;        // [split][batch][M][N] when splits > 1
  long long ldc, c_batch_stride;
  int batch, M, N, K, k_split, splits;
  bool accumulate;
  int vec;               // elements of C per aligned access to a row: 16, 8 or 1
  int* status;
};

template <int BN>
struct Layout {
  static constexpr int kA = kBM * kBK * 2, kB = BN * kBK * 2, kStage = kA + kB;
  static constexpr int kBars = kStages * kStage;
  static constexpr int kBytes = kBars + 128;
};

__device__ __forceinline__ void load_tile(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
          smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

template <int BN, bool A_ROWS, bool B_ROWS>
__global__ void __launch_bounds__(kThreads, 1) gemm16_kernel(const __grid_constant__ Params p) {
  enter_kernel(((p.M + kBM - 1) / kBM) * ((p.N + BN - 1) / BN) * p.batch * p.splits <= static_cast<int>(gridDim.x));
  using L = Layout<BN>;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* const full = reinterpret_cast<uint64_t*>(smem + L::kBars);
  uint64_t* const empty = full + kStages;
  uint64_t* const acc_full = empty + kStages;
  uint64_t* const acc_empty = acc_full + 2;
  uint32_t* const slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], 4); }
    mbar_init_fence();
  }
  if (warp == 1) tmem_alloc(slot, 2 * BN);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = *slot;
  bool timed_out = false;
  const int mt = (p.M + kBM - 1) / kBM, nt = (p.N + BN - 1) / BN, per_split = mt * nt * p.batch;
  const int tiles = per_split * p.splits;

  if (warp == 0) {
    int stage = 0;
    uint32_t parity = 1;
    const bool leader = elect_one();
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
      const int sp = tile / per_split, r = tile % per_split, z = r / (mt * nt);
      const int n0 = (r % nt) * BN, m0 = (r / nt % mt) * kBM;
      const int k_end = min(p.K, (sp + 1) * p.k_split);
      for (int k0 = sp * p.k_split; k0 < k_end; k0 += kBK) {
        mbar_wait_flag(&empty[stage], parity, timed_out);
        if (leader) {
          uint8_t* const sa = smem + stage * L::kStage;
          uint8_t* const sb = sa + L::kA;
          tma::expect_bytes(&full[stage], L::kStage);
          if (A_ROWS) {
#pragma unroll
            for (int j = 0; j < kBM / 64; ++j) load_tile(sa + j * 8192, &p.map_a, &full[stage], m0 + 64 * j, k0, z);
          } else {
            load_tile(sa, &p.map_a, &full[stage], k0, m0, z);
          }
          if (B_ROWS) {
#pragma unroll
            for (int j = 0; j < BN / 64; ++j) load_tile(sb + j * 8192, &p.map_b, &full[stage], n0 + 64 * j, k0, z);
          } else {
            load_tile(sb, &p.map_b, &full[stage], k0, n0, z);
          }
        }
        __syncwarp();
        if (++stage == kStages) { stage = 0; parity ^= 1; }
      }
    }
  } else if (warp == 1) {
    const bool leader = elect_one();
    const uint32_t idesc = idesc_bf16(kBM, BN, A_ROWS, B_ROWS);
    int stage = 0, turn = 0;
    uint32_t parity = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++turn) {
      const int sp = tile / per_split;
      const int k_end = min(p.K, (sp + 1) * p.k_split);
      const int buf = turn & 1;
      mbar_wait_flag(&acc_empty[buf], ((turn >> 1) & 1) ^ 1, timed_out);
      fence_after_sync();
      bool first = true;
      for (int k0 = sp * p.k_split; k0 < k_end; k0 += kBK) {
        mbar_wait_flag(&full[stage], parity, timed_out);
        fence_after_sync();
        const uint32_t sa = smem_u32(smem + stage * L::kStage), sb = sa + L::kA;
        gemm<kBK / 16>(tmem + buf * BN, sw_operand(sa, A_ROWS, 8192), sw_operand(sb, B_ROWS, 8192), idesc, !first, leader);
        first = false;
        if (leader) commit(&empty[stage]);
        if (++stage == kStages) { stage = 0; parity ^= 1; }
      }
      if (leader) commit(&acc_full[buf]);
    }
    for (int s = 0; s < kStages; ++s) {   // commits still on their way to this CTA's barriers
      mbar_wait_flag(&empty[stage], parity ^ 1, timed_out);
      if (++stage == kStages) { stage = 0; parity ^= 1; }
    }
  } else {
    const int sub = warp & 3;   // tensor-memory lanes this warp may read
    int turn = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++turn) {
      const int sp = tile / per_split, r = tile % per_split, z = r / (mt * nt);
      const int n0 = (r % nt) * BN, m = (r / nt % mt) * kBM + sub * 32 + lane;
      const bool in = m < p.M;
      const int buf = turn & 1;
      mbar_wait_flag(&acc_full[buf], (turn >> 1) & 1, timed_out);
      fence_after_sync();
      const uint32_t src = tmem + buf * BN + (static_cast<uint32_t>(sub * 32) << 16);
#pragma unroll 1
      for (int c = 0; c < BN; c += 16) {
        if (n0 + c >= p.N) break;
        float v[16];
        __syncwarp();
        tmem_ld8(src + c, v);
        tmem_ld8(src + c + 8, v + 8);
        tmem_ld_wait();
        const int n = n0 + c, valid = in ? p.N - n : 0;
        if (valid > 0) {
          if (p.splits > 1) {
            float* const dst = p.partial + ((static_cast<size_t>(sp) * p.batch + z) * p.M + m) * p.N + n;
            if (valid >= 16 && p.N % 8 == 0) {
#pragma unroll
              for (int h = 0; h < 16; h += 8)
                asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst + h), "f"(v[h]), "f"(v[h + 1]), "f"(v[h + 2]),
                             "f"(v[h + 3]), "f"(v[h + 4]), "f"(v[h + 5]), "f"(v[h + 6]), "f"(v[h + 7])
                             : "memory");
            } else {
#pragma unroll
              for (int e = 0; e < 16; ++e)
                if (e < valid) dst[e] = v[e];
            }
          } else {
            __nv_bfloat16* const dst = p.c + z * p.c_batch_stride + m * p.ldc + n;
            if (p.bias) {
#pragma unroll
              for (int e = 0; e < 16; ++e)
                if (e < valid) v[e] += __bfloat162float(p.bias[n + e]);
            }
            // (sums into existing rows, and rows on 16 bytes only, element by element: 26 us at 6000 x 768 x 8 instead of 11,
            // 14 at 4 x 6000 x 64 x 128 instead of 7)
            if (valid >= 16 && p.vec >= 8) {
              if (p.accumulate) {
                float had[16];
                unpack8_bf16(*reinterpret_cast<const uint4*>(dst), had);
                unpack8_bf16(*reinterpret_cast<const uint4*>(dst + 8), had + 8);
#pragma unroll
                for (int e = 0; e < 16; ++e) v[e] += had[e];
              }
              if (p.vec == 16) {
                uint32_t w[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) w[e] = pack_bf16(v[2 * e], v[2 * e + 1]);
                asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]),
                             "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                             : "memory");
              } else {
                *reinterpret_cast<uint4*>(dst) = pack8_bf16(v);
                *reinterpret_cast<uint4*>(dst + 8) = pack8_bf16(v + 8);
              }
            } else {
#pragma unroll
              for (int e = 0; e < 16; ++e) {
                if (e >= valid) continue;
                if (p.accumulate) v[e] += __bfloat162float(dst[e]);
                dst[e] = __float2bfloat16(v[e]);
              }
            }
          }
        }
      }
      fence_before_sync();
      __syncwarp();
      if (lane == 0) arrive(&acc_empty[buf]);
    }
  }
  if (timed_out && p.status) atomicExch(p.status, 1);
  fence_before_sync();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, 2 * BN);
}

// Four elements a thread; of many splits every eighth goes to one of eight threads (one thread for all of the 37 to 74 splits of a
// narrow weight gradient: 18 to 32 us), and their sums are added in a fixed order.  `kVec`: rows of four elements on aligned places.
// (An element a thread, always eight to an element: 4096 x 256 x 768 in two splits took 30 us with its product, 8.5 now.)
template <int kParts, int kVec>
__global__ void __launch_bounds__(256) reduce_splits_kernel(const float* __restrict__ partial, int splits, long long all, int M, int N,
                                                            const __nv_bfloat16* __restrict__ bias, __nv_bfloat16* __restrict__ c,
                                                            long long ldc, long long c_batch_stride, bool accumulate) {
  enter_kernel();
  constexpr int kLanes = 256 / kParts;
  __shared__ float red[kParts > 1 ? kParts : 1][kLanes][kVec];
  const int tx = threadIdx.x % kLanes, ty = threadIdx.x / kLanes;
  const long long i = (static_cast<long long>(blockIdx.x) * kLanes + tx) * kVec;
  float v[kVec] = {};
  if (i < all) {
    const float* const from = partial + i;
#pragma unroll 8
    for (int k = ty; k < splits; k += kParts) {
      if constexpr (kVec == 4) {
        const float4 u = *reinterpret_cast<const float4*>(from + k * all);
        v[0] += u.x; v[1] += u.y; v[2] += u.z; v[3] += u.w;
      } else {
        v[0] += from[k * all];
      }
    }
  }
  if constexpr (kParts > 1) {
#pragma unroll
    for (int e = 0; e < kVec; ++e) red[ty][tx][e] = v[e];
    __syncthreads();
    if (ty != 0) return;
#pragma unroll
    for (int k = 1; k < kParts; ++k)
#pragma unroll
      for (int e = 0; e < kVec; ++e) v[e] += red[k][tx][e];
  }
  if (i >= all) return;
  const int n = static_cast<int>(i % N);
  const long long row = i / N;
  __nv_bfloat16* const dst = c + row / M * c_batch_stride + row % M * ldc + n;
#pragma unroll
  for (int e = 0; e < kVec; ++e) {
    if (bias) v[e] += __bfloat162float(bias[n + e]);
    if (accumulate) v[e] += __bfloat162float(dst[e]);
  }
  if constexpr (kVec == 4) *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
  else *dst = __float2bfloat16(v[0]);
}
template <int kParts>
void reduce_splits(const Params& p, cudaStream_t stream) {
  const long long all = static_cast<long long>(p.batch) * p.M * p.N;
  const bool vec = p.N % 4 == 0 && p.ldc % 4 == 0 && p.c_batch_stride % 4 == 0 && reinterpret_cast<uintptr_t>(p.c) % 8 == 0;
  const long long per_block = 256 / kParts * (vec ? 4 : 1);
  mxk::launch_kernel(vec ? reduce_splits_kernel<kParts, 4> : reduce_splits_kernel<kParts, 1>, static_cast<unsigned>((all + per_block - 1) / per_block), 256, 0, stream, p.partial, p.splits, all,
                     p.M, p.N, p.bias, p.c, p.ldc, p.c_batch_stride, p.accumulate);
}

// Narrow tiles where wide ones would leave SMs idle; a contraction is split when even those do and each part still has
// four stages.
struct Plan {
  int bn, splits, k_split;
};
Plan plan(int batch, int M, int N, int K) {
  const long long mt = static_cast<long long>(batch) * ((M + kBM - 1) / kBM);
  const int kb = (K + kBK - 1) / kBK, most = kb / 4 > 1 ? kb / 4 : 1;
  Plan pl{128, 1, 0};
  if (N <= 64 || mt * ((N + 127) / 128) * most < kNumSMs) pl.bn = 64;
  const long long t = mt * ((N + pl.bn - 1) / pl.bn);
  if (t < kNumSMs && most > 1) pl.splits = static_cast<int>(min(static_cast<long long>(most), kNumSMs / t));   // one wave
  const int per = (kb + pl.splits - 1) / pl.splits;
  pl.k_split = per * kBK;
  pl.splits = (kb + per - 1) / per;
  return pl;
}

bool encode(CUtensorMap* map, const Matrix& m, int cols, int rows, int batch, int box_rows) {
  tma::EncodeTiledFn enc = tma::encode_tiled_fn();
  if (!enc) return false;
  const cuuint64_t dims[3] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(batch)};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(m.ld) * 2, static_cast<cuuint64_t>(batch > 1 ? m.batch_stride : m.ld) * 2};
  const cuuint32_t box[3] = {64, static_cast<cuuint32_t>(box_rows), 1};
  const cuuint32_t elem[3] = {1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(m.ptr), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN, bool A_ROWS, bool B_ROWS>
int launch(const Params& p, cudaStream_t stream) {
  if (const int st = allow_smem<gemm16_kernel<BN, A_ROWS, B_ROWS>, Layout<BN>::kBytes>(); st != MXK_OK) return st;
  const long long tiles = static_cast<long long>((p.M + kBM - 1) / kBM) * ((p.N + BN - 1) / BN) * p.batch * p.splits;
  mxk::launch_kernel(gemm16_kernel<BN, A_ROWS, B_ROWS>, static_cast<unsigned>(min(tiles, static_cast<long long>(kNumSMs))), kThreads, Layout<BN>::kBytes, stream, p);
  return launch_status();
}
template <int BN>
int launch_bn(const Params& p, bool a_rows, bool b_rows, cudaStream_t s) {
  if (a_rows) return b_rows ? launch<BN, true, true>(p, s) : launch<BN, true, false>(p, s);
  return b_rows ? launch<BN, false, true>(p, s) : launch<BN, false, false>(p, s);
}

}  // namespace

size_t workspace_bytes(int batch, int M, int N, int K) {
  if (batch <= 0 || M <= 0 || N <= 0 || K <= 0) return 0;
  const Plan pl = plan(batch, M, N, K);
  return pl.splits > 1 ? static_cast<size_t>(pl.splits) * batch * M * N * sizeof(float) : 0;
}

int run(const Matrix& a, bool a_rows, const Matrix& b, bool b_rows, const void* bias, void* c, long long ldc,
        long long c_batch_stride, bool accumulate, int batch, int M, int N, int K, void* ws, size_t ws_bytes, int* status,
        cudaStream_t stream) {
  if (!a.ptr || !b.ptr || !c) return MXK_ERR_NULL;
  if (batch <= 0 || M <= 0 || N <= 0 || K <= 0) return MXK_ERR_DIMS;
  if (!aligned16(a.ptr) || !aligned16(b.ptr) || a.ld % 8 || b.ld % 8 || a.batch_stride % 8 || b.batch_stride % 8) return MXK_ERR_ALIGN;
  const Plan pl = plan(batch, M, N, K);
  if (pl.splits > 1 && (!ws || reinterpret_cast<uintptr_t>(ws) % 32 || ws_bytes < workspace_bytes(batch, M, N, K))) return MXK_ERR_WORKSPACE;
  Params p{};
  if (!encode(&p.map_a, a, a_rows ? M : K, a_rows ? K : M, batch, a_rows ? kBK : kBM) ||
      !encode(&p.map_b, b, b_rows ? N : K, b_rows ? K : N, batch, b_rows ? kBK : pl.bn))
    return MXK_ERR_UNSUPPORTED;
  p.c = static_cast<__nv_bfloat16*>(c);
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.partial = static_cast<float*>(ws);
  p.ldc = ldc;
  p.c_batch_stride = c_batch_stride;
  p.batch = batch; p.M = M; p.N = N; p.K = K;
  p.k_split = pl.k_split; p.splits = pl.splits;
  p.accumulate = accumulate;
  const auto rows_on = [&](int elements) { return reinterpret_cast<uintptr_t>(c) % (2 * elements) == 0 && ldc % elements == 0 && c_batch_stride % elements == 0; };
  p.vec = rows_on(16) ? 16 : rows_on(8) ? 8 : 1;
  p.status = status;
  const int st = pl.bn == 128 ? launch_bn<128>(p, a_rows, b_rows, stream) : launch_bn<64>(p, a_rows, b_rows, stream);
  if (st != MXK_OK || pl.splits == 1) return st;
  if (pl.splits > 8) reduce_splits<8>(p, stream);
  else reduce_splits<1>(p, stream);
  return launch_status();
}

}  // namespace gemm16
}  // namespace mxk
