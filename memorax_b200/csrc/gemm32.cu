// float32 matrix products on the tensor cores (tcgen05): contractions of at most 255 elements, and the host side of all of them.
// (Longer ones: gemm32_long.cu, gemm32_long_outer.cu.)
//
// A float32 number is the exact sum of three bf16 numbers (8 + 8 + 8 mantissa bits: hi + mid + lo), so a product
// of float32 matrices is a sum of bf16 products accumulated in float32.  The six largest of the nine are kept;
// the dropped ones (mid*lo, lo*mid, lo*lo) are below 2^-26 of |a||b|, i.e. below the rounding of a float32 product.
//
// Bound: the tensor pipe at six bf16 products per float32 product (1.66 PFLOP/s / 6 = 277 TFLOP/s; a plain float32
// FMA kernel stops at about 65 here).  At M = 128, N = 256 the pipe reads 96 bytes of shared memory per cycle and
// the conversion below writes 48, against 128 available, so shared memory binds a little before the pipe does.
//
// One persistent CTA per SM, warp-specialised:
//   epilogue   accumulators (TMEM) -> global in whole lines, see to_lines()
//   producers  global float32 -> registers (a stage ahead) -> three bf16 planes in shared memory
//   1 warp     issues the MMAs (12 per stage of 32 k)
// Eight warps each for the first two; where one CTA converts both operands alone, 12 producers and 4 epilogue warps.
// Weights are split once, by split_weights, into images of the shared-memory stage, which arrive by one bulk copy per
// stage.  A gradient of a weight contracts two activations and converts both.
// Operand planes are in the panel format of umma.cuh, which serves contraction over columns and over rows alike, so
// nothing is transposed.
//
// Precision: the tensor core truncates when it adds to a float32 accumulator (measured: the error grows linearly with
// the number of additions, 3.3e-6 of the result's norm after 192), so the five small products go to an accumulator of
// their own, whose truncations are 2^-8 as large.  Errors against float64 are then those of a float32 FMA kernel.
#include <algorithm>

#include "gemm32_common.cuh"
#include "tma.cuh"

namespace mxk {
namespace gemm32 {
namespace {

using namespace umma;

constexpr int kBM = 128, kBK = 32;

struct Params {
  const float* a;
  long long lda;
  const uint8_t* image;   // kOuter: unused
  const float* b;         // kOuter only
  long long ldb;
  bool a_wide, b_wide;    // 32-byte aligned rows
  float* c;
  long long ldc;
  int c_vec;
  int M, N, K;
  Epilogue ep;
  int ep_vec;
  int* status;
};

// BN = 256: two CTAs share a 256 x 256 tile (cta_group::2), each with its 128 rows of A and half of the rows of B.
template <int BN>
struct Layout {
  static constexpr bool kPair = BN == 256;
  static constexpr int kRowsB = kPair ? BN / 2 : BN;   // rows of B in this CTA
  static constexpr int kStages = BN == 64 ? 5 : 4;
  static constexpr int kPlaneA = kBM * kBK * 2, kPlaneB = kRowsB * kBK * 2;   // bytes
  static constexpr int kStage = 3 * (kPlaneA + kPlaneB);
  static constexpr int kBarriers = kStages * kStage;
  static constexpr int kBytes = kBarriers + 256;
  // two accumulators of BN columns; a second pair, where TMEM has room for it, lets a tile's epilogue run under the
  // next tile's products
  static constexpr int kAccs = BN == 256 ? 1 : 2;
  static constexpr uint32_t kTmem = kAccs * 2 * BN;
};

// One operand tile of a stage: `ROWS` contracted over its rows ([kBK][EXT]) or its columns ([EXT][kBK]); split into
// blocks of 8 rows x 32 columns, one block per warp and turn: a lane owns 8 consecutive columns of a row, eight
// consecutive lanes own eight rows (conflict-free 16-byte shared stores, whole 128-byte lines of global memory).
template <bool ROWS, int EXT, int WARPS>
struct Tile {
  static constexpr int kRows = ROWS ? kBK : EXT;
  static constexpr int kBlocks = EXT * kBK / 256;
  static constexpr int kTurns = (kBlocks + WARPS - 1) / WARPS;
  float x[kTurns][8];
  const float* ptr[kTurns];   // this lane's vector of the block about to be loaded
  __device__ static __forceinline__ void coords(int block, int lane, int& r, int& c) {
    const int rb = ROWS ? (block & 3) : block, cb = ROWS ? (block >> 2) : 0;
    r = rb * 8 + (lane & 7);
    c = cb * 32 + (lane >> 3) * 8;
  }
  // ext0: the tile's first index along EXT, k0: along the contraction
  __device__ __forceinline__ void begin(const float* base, long long ld, int warp, int lane, int ext0, int k0) {
#pragma unroll
    for (int i = 0; i < kTurns; ++i) {
      int r, c;
      coords(warp + i * WARPS, lane, r, c);
      ptr[i] = base + static_cast<long long>(r + (ROWS ? k0 : ext0)) * ld + (c + (ROWS ? ext0 : k0));
    }
  }
  __device__ __forceinline__ void advance(long long ld) {
#pragma unroll
    for (int i = 0; i < kTurns; ++i) ptr[i] += ROWS ? kBK * ld : static_cast<long long>(kBK);
  }
  // `inner`: the whole tile lies inside the matrix and its rows are 32-byte aligned
  __device__ __forceinline__ void load(int i, bool inner, int warp, int lane, int ext0, int ext_end, int k0, int k_end) {
    const int block = warp + i * WARPS;
    if (kBlocks % WARPS != 0 && block >= kBlocks) return;
    if (inner) {
      load8(ptr[i], 8, 8, x[i]);
    } else {
      int r, c;
      coords(block, lane, r, c);
      const int row = r + (ROWS ? k0 : ext0), col = c + (ROWS ? ext0 : k0);
      const bool in = row < (ROWS ? k_end : ext_end);
      load8(ptr[i], in ? (ROWS ? ext_end : k_end) - col : 0, 1, x[i]);
    }
  }
  __device__ __forceinline__ void store(int i, uint8_t* plane0, int warp, int lane) {
    constexpr int kPlane = EXT * kBK * 2;
    const int block = warp + i * WARPS;
    if (kBlocks % WARPS != 0 && block >= kBlocks) return;
    int r, c;
    coords(block, lane, r, c);
    uint4 hi, mid, lo;
    split8(x[i], hi, mid, lo);
    uint8_t* const dst = plane0 + ((c >> 3) * kRows + r) * 16;
    *reinterpret_cast<uint4*>(dst) = hi;
    *reinterpret_cast<uint4*>(dst + kPlane) = mid;
    *reinterpret_cast<uint4*>(dst + 2 * kPlane) = lo;
  }
};

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* out) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) out[i] = __uint_as_float(r[i]);
}

// v: 32 consecutive columns of row `lane`.  Afterwards v[8 j ..] are columns 8 (lane & 3) .. + 7 of row (lane & 28) + j, so
// that a store instruction writes whole 128-byte lines: with a row per lane it touched 32 lines for 32 bytes each, and a
// 128 x 256 accumulator took 7.9 k cycles to drain instead of the 5 k that its bytes need.
__device__ __forceinline__ void to_lines(float* v, int lane) {
#pragma unroll
  for (int o = 1; o <= 2; o <<= 1) {
    const bool high = (lane & o) != 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (u & o) continue;
#pragma unroll
      for (int e = 0; e < 8; ++e) {   // units u and u + o: keep one, trade the other
        float &a = v[u * 8 + e], &b = v[(u + o) * 8 + e];
        const float got = __shfl_xor_sync(0xffffffffu, high ? a : b, o);
        a = high ? got : a;
        b = high ? b : got;
      }
    }
  }
}

// kOuter: C = A^T B, both operands contracted over their rows and converted here; else C = A W^T, W from its image.
template <int BN, bool kOuter>
struct Roles {
  // (a seventeenth warp is the last that leaves 96 registers a thread)
  static constexpr int kProducerWarps = !kOuter || BN == 256 ? 8 : 12, kEpilogueWarps = kOuter && BN != 256 ? 4 : 8;
  static constexpr int kMmaWarp = kProducerWarps + kEpilogueWarps;
  static constexpr int kThreads = 32 * (kMmaWarp + 1);
};

template <int BN, bool kOuter>
__global__ void __launch_bounds__(Roles<BN, kOuter>::kThreads, 1) gemm32_kernel(const __grid_constant__ Params p) {
  using L = Layout<BN>;
  constexpr bool kPair = L::kPair;
  constexpr int kTileM = kPair ? 2 * kBM : kBM;
  const int mt = (p.M + kTileM - 1) / kTileM, nt = (p.N + BN - 1) / BN;
  const int tiles = mt * nt;
  const int first_tile = kPair ? blockIdx.x / 2 : blockIdx.x, tile_step = kPair ? gridDim.x / 2 : gridDim.x;
  enter_kernel(tiles <= tile_step);
  const int rank = kPair ? static_cast<int>(cluster_rank()) : 0;
  using R = Roles<BN, kOuter>;
  constexpr int kProducerWarps = R::kProducerWarps, kEpilogueWarps = R::kEpilogueWarps, kMmaWarp = R::kMmaWarp;
  constexpr int kColumnParts = kEpilogueWarps / 4;   // epilogue warps that share the rows, and the columns between them
  using TileA = Tile<kOuter, kBM, kProducerWarps>;
  using TileB = Tile<true, L::kRowsB, kProducerWarps>;
  constexpr int kStages = L::kStages;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* const bars = reinterpret_cast<uint64_t*>(smem + L::kBarriers);
  uint64_t* const full = bars;                 // producers (and the image's bulk copy) -> MMA
  uint64_t* const empty = bars + kStages;      // MMA -> producers
  uint64_t* const acc_full = bars + 2 * kStages;       // MMA -> epilogue
  uint64_t* const acc_empty = bars + 2 * kStages + 2;  // epilogue -> MMA
  uint64_t* const peer_full = bars + 2 * kStages + 4;  // rank 0: the other CTA's stage is full
  uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(bars + 3 * kStages + 4);
  const auto wait = [](uint64_t* bar, uint32_t parity, bool& timed_out) {
    if (kPair) mbar_wait_cluster_flag(bar, parity, timed_out);
    else mbar_wait_flag(bar, parity, timed_out);
  };
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(&full[s], kProducerWarps + (kOuter ? 0 : 1)); mbar_init(&empty[s], 1); mbar_init(&peer_full[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], kEpilogueWarps * (kPair ? 2 : 1)); }
    mbar_init_fence();
  }
  if (warp == kMmaWarp) {
    if (kPair) tmem_alloc_pair(tmem_slot, L::kTmem);
    else tmem_alloc(tmem_slot, L::kTmem);
  }
  fence_before_sync();
  __syncthreads();
  if (kPair) cluster_sync();   // the other CTA's barriers are there
  fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  bool timed_out = false;

  if (warp >= kEpilogueWarps && warp < kMmaWarp) {
    // ------------------------------------------------------------ producers
    const int pw = warp - kEpilogueWarps;
    const int k_images = (p.K + kBK - 1) / kBK;
    int tile = first_tile;
    int stage = 0;
    uint32_t parity = 1;   // a fresh barrier's previous phase counts as complete
    TileA ta;
    TileB tb;
    const int k_end = p.K;
    int m0 = 0, n0 = 0, k0 = 0;
    bool a_inner = false, b_inner = false;
    auto tile_begin = [&](int t) {
      n0 = (t % nt) * BN + rank * L::kRowsB;   // of this CTA's part of B
      m0 = (t / nt) * kTileM + rank * kBM;
      k0 = 0;
      ta.begin(p.a, p.lda, pw, lane, m0, k0);
      if (kOuter) tb.begin(p.b, p.ldb, pw, lane, n0, k0);
    };
    auto bounds = [&]() {
      const bool k_in = k0 + kBK <= k_end;
      a_inner = p.a_wide && k_in && m0 + kBM <= p.M;
      b_inner = p.b_wide && k_in && n0 + L::kRowsB <= p.N;
    };
    if (tile < tiles) {
      tile_begin(tile);
      bounds();
#pragma unroll
      for (int i = 0; i < TileA::kTurns; ++i) ta.load(i, a_inner, pw, lane, m0, p.M, k0, k_end);
      if (kOuter) {
#pragma unroll
        for (int i = 0; i < TileB::kTurns; ++i) tb.load(i, b_inner, pw, lane, n0, p.N, k0, k_end);
      }
    }
    while (tile < tiles) {
      const uint8_t* const image = kOuter ? nullptr : p.image + (static_cast<size_t>(n0 / L::kRowsB) * k_images + k0 / kBK) * (3 * L::kPlaneB);
      // the block after this one, whose loads are issued as this one's registers are released
      k0 += kBK;
      if (k0 >= k_end) {
        tile += tile_step;
        if (tile < tiles) tile_begin(tile);
      } else {
        ta.advance(p.lda);
        if (kOuter) tb.advance(p.ldb);
      }
      const bool more = tile < tiles;
      bounds();
      wait(&empty[stage], parity, timed_out);
      uint8_t* const base = smem + stage * L::kStage;
      if (!kOuter && pw == 0 && lane == 0) {
        tma::expect_bytes(&full[stage], 3 * L::kPlaneB);
        tma::load_bulk(base + 3 * L::kPlaneA, image, 3 * L::kPlaneB, &full[stage]);
      }
#pragma unroll
      for (int i = 0; i < TileA::kTurns; ++i) {
        ta.store(i, base, pw, lane);
        if (more) ta.load(i, a_inner, pw, lane, m0, p.M, k0, k_end);
      }
      if (kOuter) {
#pragma unroll
        for (int i = 0; i < TileB::kTurns; ++i) {
          tb.store(i, base + 3 * L::kPlaneA, pw, lane);
          if (more) tb.load(i, b_inner, pw, lane, n0, p.N, k0, k_end);
        }
      }
      fence_smem_to_async();
      __syncwarp();
      if (lane == 0) arrive(&full[stage]);
      if (++stage == kStages) { stage = 0; parity ^= 1; }
    }
  } else if (warp == kMmaWarp) {
    // ------------------------------------------------------------ tensor core
    const bool leader = elect_one();
    const uint32_t idesc = idesc_bf16(kTileM, BN, kOuter, kOuter);
    int stage = 0;
    uint32_t parity = 0;
    int turn = 0;
    for (int tile = first_tile; tile < tiles; tile += tile_step, ++turn) {
      const int blocks = (p.K + kBK - 1) / kBK;
      const int buf = turn % L::kAccs;
      if (rank == 0) wait(&acc_empty[buf], ((turn / L::kAccs) & 1) ^ 1, timed_out);
      fence_after_sync();
      const uint32_t acc = tmem + buf * 2 * BN, acc_small = acc + BN;
      for (int kb = 0; kb < blocks; ++kb) {
        wait(&full[stage], parity, timed_out);
        if (kPair && rank != 0) {   // this CTA's stage is full: the other one issues
          if (leader) arrive_at_leader(&peer_full[stage]);
          __syncwarp();
          if (++stage == kStages) { stage = 0; parity ^= 1; }
          continue;
        }
        if (kPair) wait(&peer_full[stage], parity, timed_out);
        fence_after_sync();
        const uint32_t sa = smem_u32(smem + stage * L::kStage), sb = sa + 3 * L::kPlaneA;
        constexpr uint32_t kRowsA = kOuter ? kBK : kBM, kRowsB = kOuter ? kBK : L::kRowsB;
        const Operand a0{sa, kRowsA, kOuter}, a1{sa + L::kPlaneA, kRowsA, kOuter}, a2{sa + 2 * L::kPlaneA, kRowsA, kOuter};
        const Operand b0{sb, kRowsB, kOuter}, b1{sb + L::kPlaneB, kRowsB, kOuter}, b2{sb + 2 * L::kPlaneB, kRowsB, kOuter};
        const auto product = [&](uint32_t d, const Operand& a, const Operand& b, bool accumulate) {
          if (kPair) gemm_pair<kBK / 16>(d, a, b, idesc, accumulate, leader);
          else gemm<kBK / 16>(d, a, b, idesc, accumulate, leader);
        };
        product(acc_small, a2, b0, kb > 0);
        product(acc_small, a0, b2, true);
        product(acc_small, a1, b1, true);
        product(acc_small, a1, b0, true);
        product(acc_small, a0, b1, true);
        product(acc, a0, b0, kb > 0);
        if (leader) (kPair ? commit_pair : commit)(&empty[stage]);
        if (++stage == kStages) { stage = 0; parity ^= 1; }
      }
      if (leader && rank == 0) (kPair ? commit_pair : commit)(&acc_full[buf]);
    }
    // the last commits may still be on their way to barriers in this CTA's shared memory
    for (int s = 0; s < kStages; ++s) {
      wait(&empty[stage], parity ^ 1, timed_out);
      if (++stage == kStages) { stage = 0; parity ^= 1; }
    }
  } else if (warp < kEpilogueWarps) {
    // ------------------------------------------------------------ epilogue
    int turn = 0;
    for (int tile = first_tile; tile < tiles; tile += tile_step, ++turn) {
      const int n0 = (tile % nt) * BN, m0 = (tile / nt) * kTileM + rank * kBM;
      const int m = m0 + (warp & 3) * 32 + (lane & 28);   // first of the four rows this lane stores, see to_lines()
      const int buf = turn % L::kAccs;
      wait(&acc_full[buf], (turn / L::kAccs) & 1, timed_out);
      fence_after_sync();
      const uint32_t src = tmem + buf * 2 * BN + (static_cast<uint32_t>((warp & 3) * 32) << 16);
#pragma unroll 1
      for (int c = (warp >> 2) * (BN / kColumnParts); c < ((warp >> 2) + 1) * (BN / kColumnParts); c += 32) {
        if (n0 + c >= p.N) break;
        float v[32];
        __syncwarp();
        tmem_ld32(src + c, v);
#pragma unroll
        for (int h = 0; h < 32; h += 16) {
          float w[16];
          tmem_ld8(src + BN + c + h, w);
          tmem_ld8(src + BN + c + h + 8, w + 8);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 16; ++e) v[h + e] += w[e];
        }
        to_lines(v, lane);
        const int n = n0 + c + (lane & 3) * 8;
        float* dst = p.c + m * p.ldc + n;
#pragma unroll
        for (int j = 0; j < 4; ++j, dst += p.ldc) {
          const int valid = m + j < p.M ? p.N - n : 0;
          if (valid <= 0) continue;
          float* const x = v + j * 8;
          if (p.ep.bias) {
#pragma unroll
            for (int e = 0; e < 8; ++e)
              if (e < valid) x[e] += __ldg(p.ep.bias + n + e);
          }
          if (p.ep.add) {
            float ad[8];
            load8(p.ep.add + (m + j) * p.ep.ld_add + n, valid, p.ep_vec, ad);
#pragma unroll
            for (int e = 0; e < 8; ++e)
              x[e] = fmaf(ad[e], (p.ep.add_scale && e < valid) ? __ldg(p.ep.add_scale + n + e) : 1.f, x[e]);
          }
          store8(dst, valid, p.c_vec, x);
        }
      }
      fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        if (kPair) arrive_at_leader(&acc_empty[buf]);
        else arrive(&acc_empty[buf]);
      }
    }
  }

  if (timed_out && p.status) atomicExch(p.status, 1);
  fence_before_sync();
  __syncthreads();
  if (kPair) cluster_sync();   // nothing reaches into the other CTA any more
  if (warp == kMmaWarp) {
    if (kPair) tmem_dealloc_pair(tmem, L::kTmem);
    else tmem_dealloc(tmem, L::kTmem);
  }
}

// C = sum over splits of the partial products (fixed order: bit-reproducible) + epilogue
__global__ void __launch_bounds__(256) reduce_splits_kernel(const float* __restrict__ partial, int splits, int M, int N,
                                                            float* __restrict__ c, long long ldc, Epilogue ep) {
  enter_kernel();
  const long long n_all = static_cast<long long>(M) * N;
  const long long i = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x;
  if (i >= n_all) return;
  float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
  int s = 0;
  for (; s + 4 <= splits; s += 4) {
    s0 += partial[(s + 0) * n_all + i];
    s1 += partial[(s + 1) * n_all + i];
    s2 += partial[(s + 2) * n_all + i];
    s3 += partial[(s + 3) * n_all + i];
  }
  for (; s < splits; ++s) s0 += partial[s * n_all + i];
  float acc = (s0 + s1) + (s2 + s3);
  const int m = static_cast<int>(i / N), n = static_cast<int>(i % N);
  if (ep.bias) acc += ep.bias[n];
  if (ep.add) acc = fmaf(ep.add[m * ep.ld_add + n], ep.add_scale ? ep.add_scale[n] : 1.f, acc);
  c[m * ldc + n] = acc;
}

int reduce_splits(const float* partial, int splits, int M, int N, float* c, long long ldc, const Epilogue& ep, cudaStream_t stream) {
  const long long n_all = static_cast<long long>(M) * N;
  mxk::launch_kernel(reduce_splits_kernel, static_cast<unsigned>((n_all + 255) / 256), 256, 0, stream, partial, splits, M, N, c, ldc, ep);
  return launch_status();
}

// Width of a tile: 256 columns halve the shared-memory traffic per product, but only where enough tiles are left to give every SM
// one.  Narrower tiles are the only way to occupy more SMs.
int tile_columns(int M, int N) {
  const auto tiles = [&](int bn) {   // CTAs that one pass over C occupies
    const int tm = bn == 256 ? 2 * kBM : kBM;
    return static_cast<long long>((M + tm - 1) / tm) * ((N + bn - 1) / bn) * (tm / kBM);
  };
  int bn = N <= 64 ? 64 : N <= 128 || M <= 128 ? 128 : 256;
  while (bn > 64 && tiles(bn) < kNumSMs) bn /= 2;
  return bn;
}

template <int BN, bool kOuter>
int launch(const Params& p, int tiles, cudaStream_t stream) {
  if (const int st = allow_smem<gemm32_kernel<BN, kOuter>, Layout<BN>::kBytes>(); st != MXK_OK) return st;
  mxk::launch_kernel_clusters(gemm32_kernel<BN, kOuter>, Layout<BN>::kPair ? 2 : 1, min(tiles, kNumSMs), Roles<BN, kOuter>::kThreads,
                              Layout<BN>::kBytes, stream, p);
  return launch_status();
}

template <bool kOuter>
int run(Params& p, cudaStream_t stream) {
  const int bn = tile_columns(p.M, p.N), tm = bn == 256 ? 2 * kBM : kBM;
  p.c_vec = vec_of(p.c, p.ldc);
  p.ep_vec = p.ep.add ? vec_of(p.ep.add, p.ep.ld_add) : 1;
  p.a_wide = vec_of(p.a, p.lda) == 8;
  p.b_wide = kOuter && vec_of(p.b, p.ldb) == 8;
  const int tiles = ((p.M + tm - 1) / tm) * ((p.N + bn - 1) / bn) * (tm / kBM);   // in CTAs
  return bn == 256 ? launch<256, kOuter>(p, tiles, stream) : bn == 128 ? launch<128, kOuter>(p, tiles, stream) : launch<64, kOuter>(p, tiles, stream);
}

struct SplitParams {
  WeightJob job[4];
  int first_block[6];   // of the four images and of lambda; past the last block for what is not asked for
  LambdaJob lambda;
};

// One thread per eight k of a weight row: reads them (zero past the matrix), writes one vector of each plane.
__global__ void __launch_bounds__(256) split_weights_kernel(const __grid_constant__ SplitParams sp) {
  enter_kernel();
  int j = 0;
  while (static_cast<int>(blockIdx.x) >= sp.first_block[j + 1]) ++j;
  if (j == 4) {
    const int n = (blockIdx.x - sp.first_block[4]) * 256 + threadIdx.x;
    if (n < sp.lambda.N) {
      const float r = expf(-expf(sp.lambda.nu_log[n]));
      float s, c;
      sincosf(expf(sp.lambda.theta_log[n]), &s, &c);
      reinterpret_cast<float2*>(sp.lambda.lambda)[n] = make_float2(r * c, r * s);
    }
    return;
  }
  const WeightJob& jb = sp.job[j];
  const bool of_long = jb.K > kShortK;
  const int bn = jb.bn, bk = of_long ? longk::kBK : kBK, kb = (jb.K + bk - 1) / bk, groups = bk / 8;
  const long long id = static_cast<long long>(blockIdx.x - sp.first_block[j]) * 256 + threadIdx.x;
  // id = ((n_tile * kb + k_block) * groups + k_group) * bn + n: consecutive threads write (nearly) consecutive vectors
  const int n_in = static_cast<int>(id % bn);
  const long long rest = id / bn;
  const int kg = static_cast<int>(rest % groups), k_block = static_cast<int>(rest / groups % kb);
  const int n_tile = static_cast<int>(rest / groups / kb);
  if (n_tile * bn >= jb.N) return;
  float x[8];
  weight_vector(jb, n_tile * bn + n_in, k_block * groups + kg, x);
  uint4 hi, mid, lo;
  split8(x, hi, mid, lo);
  // a tile of a pair of CTAs is cut into the halves that the two hold
  const int cut = of_long ? longk::rows_of(bn) : bn == 256 ? 128 : bn, part = n_tile * (bn / cut) + n_in / cut, row = n_in % cut;
  uint4* const dst = static_cast<uint4*>(jb.image) + (static_cast<size_t>(part) * kb + k_block) * (3 * cut * groups) + kg * cut +
                     (of_long ? (row & ~31) + longk::placed(row & 31) : row);
  dst[0] = hi;
  dst[cut * groups] = mid;
  dst[2 * cut * groups] = lo;
}

}  // namespace

int tile_width(int M, int N, int K) { return K > kShortK ? longk::plan(M, N, K).bn : tile_columns(M, N); }

size_t image_bytes(int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  const int bn = tile_width(M, N, K);
  const int bk = K > kShortK ? longk::kBK : kBK;
  return static_cast<size_t>((N + bn - 1) / bn) * ((K + bk - 1) / bk) * (3 * bn * bk * 2);
}

int split_weights(const WeightJob* jobs, int count, const LambdaJob& lambda, cudaStream_t stream) {
  if (count < 0 || count > 4) return MXK_ERR_DIMS;
  SplitParams sp{};
  for (int j = 0; j < count; ++j) {
    const WeightJob& jb = jobs[j];
    if (!jb.image || jb.w.count < 1) return MXK_ERR_NULL;
    if (!aligned16(jb.image)) return MXK_ERR_ALIGN;
    sp.job[j] = jb;
    const int bk = jb.K > kShortK ? longk::kBK : kBK;
    const long long vectors = static_cast<long long>((jb.N + jb.bn - 1) / jb.bn) * jb.bn * ((jb.K + bk - 1) / bk) * (bk / 8);
    sp.first_block[j + 1] = sp.first_block[j] + static_cast<int>((vectors + 255) / 256);
  }
  for (int j = count; j < 4; ++j) sp.first_block[j + 1] = sp.first_block[count];
  const int blocks = sp.first_block[4] + (lambda.N + 255) / 256;
  sp.first_block[5] = 0x7fffffff;
  sp.lambda = lambda;
  if (blocks == 0) return MXK_OK;
  mxk::launch_kernel(split_weights_kernel, blocks, 256, 0, stream, sp);
  return launch_status();
}

size_t workspace_bytes(int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  // (of a weight's product or of two activations')
  const int splits = K > kShortK ? std::max(longk::plan(M, N, K).splits, longk::plan_outer(M, N, K).splits) : 1;
  return splits > 1 ? static_cast<size_t>(splits) * M * N * sizeof(float) : 0;
}

int run_weights(const float* a, long long lda, const void* image, float* c, long long ldc, int M, int N, int K,
                const Epilogue& ep, float* ws, size_t ws_bytes, int* status, cudaStream_t stream) {
  if (!a || !image || !c) return MXK_ERR_NULL;
  if (M <= 0 || N <= 0 || K <= 0) return MXK_ERR_DIMS;
  if (!aligned16(image)) return MXK_ERR_ALIGN;
  if (K > kShortK) {
    const longk::Plan pl = longk::plan(M, N, K);
    if (pl.splits > 1 && (!ws || ws_bytes < static_cast<size_t>(pl.splits) * M * N * sizeof(float))) return MXK_ERR_WORKSPACE;
    const int st = longk::launch_weights(pl, a, lda, image, c, ldc, M, N, K, ep, ws, status, stream);
    return st != MXK_OK || pl.splits == 1 ? st : reduce_splits(ws, pl.splits, M, N, c, ldc, ep, stream);
  }
  Params p{};
  p.a = a; p.lda = lda;
  p.image = static_cast<const uint8_t*>(image);
  p.c = c; p.ldc = ldc;
  p.M = M; p.N = N; p.K = K;
  p.ep = ep;
  p.status = status;
  return run<false>(p, stream);
}

int run_outer(const float* a, long long lda, const float* b, long long ldb, float* c, long long ldc, int M, int N, int K,
              float* ws, size_t ws_bytes, int* partials, int* status, cudaStream_t stream) {
  if (!a || !b || !c) return MXK_ERR_NULL;
  if (M <= 0 || N <= 0 || K <= 0) return MXK_ERR_DIMS;
  if (K > kShortK) {
    const longk::Plan pl = longk::plan_outer(M, N, K);
    if (pl.splits > 1 && (!ws || ws_bytes < static_cast<size_t>(pl.splits) * M * N * sizeof(float))) return MXK_ERR_WORKSPACE;
    const int st = longk::launch_outer(pl, a, lda, b, ldb, c, ldc, M, N, K, ws, status, stream);
    if (partials) *partials = pl.splits;
    return st != MXK_OK || pl.splits == 1 || partials ? st : reduce_splits(ws, pl.splits, M, N, c, ldc, {}, stream);
  }
  Params p{};
  p.a = a; p.lda = lda;
  p.b = b; p.ldb = ldb;
  p.c = c; p.ldc = ldc;
  p.M = M; p.N = N; p.K = K;
  p.status = status;
  if (partials) *partials = 1;
  return run<true>(p, stream);
}

}  // namespace gemm32
}  // namespace mxk
