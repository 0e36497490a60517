// bf16 matrix products on tcgen05 for the layers' middle sizes, where a library call costs more on the host (about 30 us
// through the framework) than the product takes: operands by TMA in swizzled tiles, contracted over either index without
// transposing, batched (the block-diagonal projections of a head), split along long contractions (weight gradients).
//
// One persistent CTA per SM: warp 0 issues the TMA loads (4 stages of 64 k), warp 1 the MMAs (M = 128, N = 64 or 128),
// warps 2..5 drain the accumulators, double-buffered in tensor memory, one row per thread with 32-byte stores.
// Bound: L2 -> SM bandwidth at these tiles (a 128 x 128 x 64 step reads 32 KB for 256 cycles of the pipe), which is why
// the largest products stay with the library's two-SM tiles.
#include <cuda_bf16.h>

#include <algorithm>

#include "gemm16.cuh"
#include "mxk_common.cuh"
#include "tma.cuh"
#include "umma.cuh"

namespace mxk {
namespace gemm16 {
namespace {

using namespace umma;

constexpr int kBM = 128, kBK = 64, kStages = 4, kThreads = 192;

struct Problem {
  CUtensorMap map_a, map_b;
  __nv_bfloat16* c;
  const __nv_bfloat16* bias;
  float* partial;        // [split][batch][M][N] when splits > 1
  long long ldc, c_batch_stride;
  int batch, M, N, K, k_split, splits;
  bool accumulate;
  int vec;               // elements of C per aligned access to a row: 16, 8 or 1
  int first_tile;        // of the launch's
};
template <int kCount>
struct Params {
  Problem problem[kCount];
  int count, tiles;
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
// Sixteen elements of a row on 32 or on 16 bytes.
__device__ __forceinline__ void store16(__nv_bfloat16* dst, const uint32_t* w, bool on32) {
  if (on32) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]),
                 "r"(w[5]), "r"(w[6]), "r"(w[7])
                 : "memory");
  } else {
    reinterpret_cast<uint4*>(dst)[0] = make_uint4(w[0], w[1], w[2], w[3]);
    reinterpret_cast<uint4*>(dst)[1] = make_uint4(w[4], w[5], w[6], w[7]);
  }
}
__device__ __forceinline__ void arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// The tile of a launch that a role works at.
template <int BN>
struct Tile {
  int q = 0;   // problem
  int sp, z, m0, n0, k0, k_end;
  template <int kCount>
  __device__ __forceinline__ const Problem& at(const Params<kCount>& all, int tile) {
    if (kCount > 1)
      while (q + 1 < all.count && tile >= all.problem[q + 1].first_tile) ++q;
    const Problem& p = all.problem[q];
    const int mt = (p.M + kBM - 1) / kBM, nt = (p.N + BN - 1) / BN, per_split = mt * nt * p.batch, i = tile - p.first_tile, r = i % per_split;
    sp = i / per_split;
    z = r / (mt * nt);
    n0 = (r % nt) * BN;
    m0 = (r / nt % mt) * kBM;
    k0 = sp * p.k_split;
    k_end = min(p.K, k0 + p.k_split);
    return p;
  }
};

// kCount: several problems of the same orders share a launch (a chain of short ones waits for the host: the mLSTM layer's five weight
// gradients in one launch and one sum of their splits instead of ten).
template <int BN, bool A_ROWS, bool B_ROWS, int kCount>
__global__ void __launch_bounds__(kThreads, 1) gemm16_kernel(const __grid_constant__ Params<kCount> all) {
  enter_kernel(all.tiles <= static_cast<int>(gridDim.x));
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
  const int tiles = all.tiles;
  Tile<BN> at;

  if (warp == 0) {
    int stage = 0;
    uint32_t parity = 1;
    const bool leader = elect_one();
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
      const Problem& p = at.at(all, tile);
      const int n0 = at.n0, m0 = at.m0, z = at.z;
      for (int k0 = at.k0; k0 < at.k_end; k0 += kBK) {
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
      at.at(all, tile);
      const int buf = turn & 1;
      mbar_wait_flag(&acc_empty[buf], ((turn >> 1) & 1) ^ 1, timed_out);
      fence_after_sync();
      bool first = true;
      for (int k0 = at.k0; k0 < at.k_end; k0 += kBK) {
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
      const Problem& p = at.at(all, tile);
      const int sp = at.sp, z = at.z, n0 = at.n0, m = at.m0 + sub * 32 + lane;
      const bool in = m < p.M;
      const int buf = turn & 1;
      const uint32_t src = tmem + buf * BN + (static_cast<uint32_t>(sub * 32) << 16);
      if (p.accumulate && p.splits == 1 && p.vec >= 8 && !p.bias && n0 + BN <= p.N) {
        // a whole row of the tile to be added to: all of it is on its way while the product is formed (32 bytes after another
        // left HBM waiting: 65536 x 1536 x 16 211 us, 16 bytes 143, 102 now)
        __nv_bfloat16* const dst = p.c + z * p.c_batch_stride + m * p.ldc + n0;
        uint32_t had[BN / 16][8];
        if (in) {
#pragma unroll
          for (int i = 0; i < BN / 16; ++i) {
            uint32_t* const h = had[i];
            if (p.vec == 16) {
              asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                           : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3]), "=r"(h[4]), "=r"(h[5]), "=r"(h[6]), "=r"(h[7])
                           : "l"(dst + 16 * i)
                           : "memory");
            } else {
              const uint4 x = reinterpret_cast<const uint4*>(dst)[2 * i], y = reinterpret_cast<const uint4*>(dst)[2 * i + 1];
              h[0] = x.x; h[1] = x.y; h[2] = x.z; h[3] = x.w;
              h[4] = y.x; h[5] = y.y; h[6] = y.z; h[7] = y.w;
            }
          }
        }
        mbar_wait_flag(&acc_full[buf], (turn >> 1) & 1, timed_out);
        fence_after_sync();
#pragma unroll
        for (int i = 0; i < BN / 16; ++i) {
          float v[16];
          __syncwarp();
          tmem_ld8(src + i * 16, v);
          tmem_ld8(src + i * 16 + 8, v + 8);
          tmem_ld_wait();
          if (in) {
            uint32_t w[8];
#pragma unroll
            for (int e = 0; e < 8; ++e)
              w[e] = pack_bf16(v[2 * e] + __uint_as_float(had[i][e] << 16), v[2 * e + 1] + __uint_as_float(had[i][e] & 0xffff0000u));
            store16(dst + 16 * i, w, p.vec == 16);
          }
        }
        fence_before_sync();
        __syncwarp();
        if (lane == 0) arrive(&acc_empty[buf]);
        continue;
      }
      mbar_wait_flag(&acc_full[buf], (turn >> 1) & 1, timed_out);
      fence_after_sync();
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
              uint32_t w[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) w[e] = pack_bf16(v[2 * e], v[2 * e + 1]);
              store16(dst, w, p.vec == 16);
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
  if (timed_out && all.status) atomicExch(all.status, 1);
  fence_before_sync();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, 2 * BN);
}

// Four elements a thread; of many splits every eighth goes to one of eight threads (one thread for all of the 37 to 74 splits of a
// narrow weight gradient: 18 to 32 us), and their sums are added in a fixed order.  `kVec`: rows of four elements on aligned places.
// (An element a thread, always eight to an element: 4096 x 256 x 768 in two splits took 30 us with its product, 8.5 now.)
struct Sum {
  const float* partial;
  const __nv_bfloat16* bias;
  __nv_bfloat16* c;
  long long all, ldc, c_batch_stride;   // all: elements
  int splits, M, N, first_block;
  bool accumulate;
};
template <int kCount>
struct Sums {
  Sum sum[kCount];
  int count;
};
template <int kParts, int kVec, int kCount>
__global__ void __launch_bounds__(256) reduce_splits_kernel(const __grid_constant__ Sums<kCount> sums) {
  enter_kernel();
  constexpr int kLanes = 256 / kParts;
  __shared__ float red[kParts > 1 ? kParts : 1][kLanes][kVec];
  int q = 0;
  if (kCount > 1)
    while (q + 1 < sums.count && static_cast<int>(blockIdx.x) >= sums.sum[q + 1].first_block) ++q;
  const Sum& p = sums.sum[q];
  const int tx = threadIdx.x % kLanes, ty = threadIdx.x / kLanes;
  const long long i = (static_cast<long long>(blockIdx.x - p.first_block) * kLanes + tx) * kVec;
  float v[kVec] = {};
  if (i < p.all) {
    const float* const from = p.partial + i;
#pragma unroll 8
    for (int k = ty; k < p.splits; k += kParts) {
      if constexpr (kVec == 4) {
        const float4 u = *reinterpret_cast<const float4*>(from + k * p.all);
        v[0] += u.x; v[1] += u.y; v[2] += u.z; v[3] += u.w;
      } else {
        v[0] += from[k * p.all];
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
  if (i >= p.all) return;
  const int n = static_cast<int>(i % p.N);
  const long long row = i / p.N;
  __nv_bfloat16* const dst = p.c + row / p.M * p.c_batch_stride + row % p.M * p.ldc + n;
#pragma unroll
  for (int e = 0; e < kVec; ++e) {
    if (p.bias) v[e] += __bfloat162float(p.bias[n + e]);
    if (p.accumulate) v[e] += __bfloat162float(dst[e]);
  }
  if constexpr (kVec == 4) *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
  else *dst = __float2bfloat16(v[0]);
}

bool by_fours(const Problem& p) { return p.N % 4 == 0 && p.ldc % 4 == 0 && p.c_batch_stride % 4 == 0 && reinterpret_cast<uintptr_t>(p.c) % 8 == 0; }

template <int kParts, int kVec, int kCount>
void launch_sums(const Params<kCount>& params, cudaStream_t stream) {
  Sums<kCount> sums{};
  long long blocks = 0;
  for (int i = 0; i < params.count; ++i) {
    const Problem& p = params.problem[i];
    if (p.splits == 1) continue;
    const long long all = static_cast<long long>(p.batch) * p.M * p.N;
    sums.sum[sums.count++] = {p.partial, p.bias, p.c, all, p.ldc, p.c_batch_stride, p.splits, p.M, p.N, static_cast<int>(blocks), p.accumulate};
    blocks += (all + 256 / kParts * kVec - 1) / (256 / kParts * kVec);
  }
  mxk::launch_kernel(reduce_splits_kernel<kParts, kVec, kCount>, static_cast<unsigned>(blocks), 256, 0, stream, sums);
}
template <int kCount>
void reduce_splits(const Params<kCount>& params, cudaStream_t stream) {
  int most = 1;
  bool fours = true;
  for (int i = 0; i < params.count; ++i)
    if (params.problem[i].splits > 1) {
      most = std::max(most, params.problem[i].splits);
      fours &= by_fours(params.problem[i]);
    }
  if (most == 1) return;
  if (fours) most > 8 ? launch_sums<8, 4>(params, stream) : launch_sums<1, 4>(params, stream);
  else most > 8 ? launch_sums<8, 1>(params, stream) : launch_sums<1, 1>(params, stream);
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

template <int BN, bool A_ROWS, bool B_ROWS, int kCount>
int launch(const Params<kCount>& p, cudaStream_t stream) {
  if (const int st = allow_smem<gemm16_kernel<BN, A_ROWS, B_ROWS, kCount>, Layout<BN>::kBytes>(); st != MXK_OK) return st;
  mxk::launch_kernel(gemm16_kernel<BN, A_ROWS, B_ROWS, kCount>, static_cast<unsigned>(std::min(p.tiles, kNumSMs)), kThreads, Layout<BN>::kBytes, stream, p);
  return launch_status();
}
template <int BN, int kCount>
int launch(const Params<kCount>& p, bool a_rows, bool b_rows, cudaStream_t s) {
  if (a_rows) return b_rows ? launch<BN, true, true>(p, s) : launch<BN, true, false>(p, s);
  return b_rows ? launch<BN, false, true>(p, s) : launch<BN, false, false>(p, s);
}

// What a launch is told of a job; MXK_OK, or what is wrong with it.
int fill(Problem& p, const Job& j, bool a_rows, bool b_rows, const Plan& pl, float* partial) {
  if (!j.a.ptr || !j.b.ptr || !j.c) return MXK_ERR_NULL;
  if (j.batch <= 0 || j.M <= 0 || j.N <= 0 || j.K <= 0) return MXK_ERR_DIMS;
  if (!aligned16(j.a.ptr) || !aligned16(j.b.ptr) || j.a.ld % 8 || j.b.ld % 8 || j.a.batch_stride % 8 || j.b.batch_stride % 8) return MXK_ERR_ALIGN;
  if (!encode(&p.map_a, j.a, a_rows ? j.M : j.K, a_rows ? j.K : j.M, j.batch, a_rows ? kBK : kBM) ||
      !encode(&p.map_b, j.b, b_rows ? j.N : j.K, b_rows ? j.K : j.N, j.batch, b_rows ? kBK : pl.bn))
    return MXK_ERR_UNSUPPORTED;
  p.c = static_cast<__nv_bfloat16*>(j.c);
  p.bias = static_cast<const __nv_bfloat16*>(j.bias);
  p.partial = partial;
  p.ldc = j.ldc;
  p.c_batch_stride = j.c_batch_stride;
  p.batch = j.batch; p.M = j.M; p.N = j.N; p.K = j.K;
  p.k_split = pl.k_split; p.splits = pl.splits;
  p.accumulate = j.accumulate;
  const auto rows_on = [&](int elements) { return reinterpret_cast<uintptr_t>(j.c) % (2 * elements) == 0 && j.ldc % elements == 0 && j.c_batch_stride % elements == 0; };
  p.vec = rows_on(16) ? 16 : rows_on(8) ? 8 : 1;
  return MXK_OK;
}
int tiles_of(const Job& j, int bn) { return (j.M + kBM - 1) / kBM * ((j.N + bn - 1) / bn) * j.batch; }
int steps_of(const Job& j) { return (j.K + kBK - 1) / kBK; }
size_t partial_floats(const Job& j, const Plan& pl) { return pl.splits > 1 ? (static_cast<size_t>(pl.splits) * j.batch * j.M * j.N + 7) / 8 * 8 : 0; }

// The most steps of a tile's contraction in a launch of several problems: those with which the SMs' rounds of tiles take the fewest
// (three more for a tile's begin and end).
Plan plan_in_group(const Job* jobs, int count, int i) {
  int longest = 1;
  for (int q = 0; q < count; ++q) longest = std::max(longest, steps_of(jobs[q]));
  long long best = -1;
  int cap = longest;
  for (int n = 1; n <= 32 && longest / n >= 4; ++n) {
    const int steps = (longest + n - 1) / n;
    long long tiles = 0;
    for (int q = 0; q < count; ++q) tiles += static_cast<long long>(tiles_of(jobs[q], 64)) * ((steps_of(jobs[q]) + steps - 1) / steps);
    const long long cost = (tiles + kNumSMs - 1) / kNumSMs * (steps + 3);
    if (best < 0 || cost < best) { best = cost; cap = steps; }
  }
  const int steps = steps_of(jobs[i]), parts = (steps + cap - 1) / cap, per = (steps + parts - 1) / parts;
  return {64, (steps + per - 1) / per, per * kBK};
}

}  // namespace

size_t workspace_bytes(int batch, int M, int N, int K) {
  if (batch <= 0 || M <= 0 || N <= 0 || K <= 0) return 0;
  const Plan pl = plan(batch, M, N, K);
  return pl.splits > 1 ? static_cast<size_t>(pl.splits) * batch * M * N * sizeof(float) : 0;
}

int run(const Job& job, bool a_rows, bool b_rows, void* ws, size_t ws_bytes, int* status, cudaStream_t stream) {
  if (job.batch <= 0 || job.M <= 0 || job.N <= 0 || job.K <= 0) return MXK_ERR_DIMS;
  const Plan pl = plan(job.batch, job.M, job.N, job.K);
  if (pl.splits > 1 && (!ws || reinterpret_cast<uintptr_t>(ws) % 32 || ws_bytes < workspace_bytes(job.batch, job.M, job.N, job.K))) return MXK_ERR_WORKSPACE;
  Params<1> p{};
  if (const int st = fill(p.problem[0], job, a_rows, b_rows, pl, static_cast<float*>(ws)); st != MXK_OK) return st;
  p.count = 1;
  p.tiles = tiles_of(job, pl.bn) * pl.splits;
  p.status = status;
  if (const int st = pl.bn == 128 ? launch<128>(p, a_rows, b_rows, stream) : launch<64>(p, a_rows, b_rows, stream); st != MXK_OK) return st;
  reduce_splits(p, stream);
  return launch_status();
}

size_t group_workspace_bytes(const Job* jobs, int count) {
  size_t floats = 0;
  for (int i = 0; i < count; ++i) floats += partial_floats(jobs[i], plan_in_group(jobs, count, i));
  return floats * sizeof(float);
}

int run_group(const Job* jobs, int count, bool a_rows, bool b_rows, void* ws, size_t ws_bytes, int* status, cudaStream_t stream) {
  if (count < 1 || count > kMaxGroup) return MXK_ERR_DIMS;
  for (int i = 0; i < count; ++i)
    if (jobs[i].batch <= 0 || jobs[i].M <= 0 || jobs[i].N <= 0 || jobs[i].K <= 0) return MXK_ERR_DIMS;
  if (const size_t need = group_workspace_bytes(jobs, count); need && (!ws || reinterpret_cast<uintptr_t>(ws) % 32 || ws_bytes < need)) return MXK_ERR_WORKSPACE;
  Params<kMaxGroup> p{};
  float* partial = static_cast<float*>(ws);
  for (int i = 0; i < count; ++i) {
    const Plan pl = plan_in_group(jobs, count, i);
    if (const int st = fill(p.problem[i], jobs[i], a_rows, b_rows, pl, partial); st != MXK_OK) return st;
    partial += partial_floats(jobs[i], pl);
    p.problem[i].first_tile = p.tiles;
    p.tiles += tiles_of(jobs[i], 64) * pl.splits;
  }
  p.count = count;
  p.status = status;
  if (const int st = launch<64>(p, a_rows, b_rows, stream); st != MXK_OK) return st;
  reduce_splits(p, stream);
  return launch_status();
}

}  // namespace gemm16
}  // namespace mxk
