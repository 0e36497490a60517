// float32 products of two activations, C = A^T B (the gradient of a weight), contractions of more than kShortK tokens, on the tensor cores:
// three bf16 planes and six products as in gemm32_long.cu.
//
// Both operands are contracted over their rows and converted here.  The accumulators live for one stage, two in contractions from 512 on
// (eight truncating additions), and are then added to float32 sums in registers.  Errors against float64, relative 2-norm, normal entries: 1.4e-7 at
// 8192 tokens, 1.9e-7 at 65536 (drained every 512 tokens: 4.2e-7 and 4.75e-7).
//
// Bound: shared memory.  A stage of 256 x 128 is 1536 cycles of the tensor pipe, but 48 KB copied in and read by the producers, 72 KB of planes
// written and 192 KB read by the pipe (A and both halves of B for six products): 2800 cycles at 128 bytes.
// Measured with the sum of the splits (the form of gemm32.cu): 1024 x 256 over 65536 tokens 203 us (204), 1024 x 512 over 24000 153 us (148),
// 520 x 512 over 8192 53 us (50).
//
// One persistent CTA per SM, pairs on tiles of 256 x 128, or alone on 128 x 64:
//   8 warps    epilogue: accumulators (TMEM) -> sums in registers -> global
//   12 warps   producers: 32 columns x 32 tokens of a stage each, eight warps for A and four for B
//   1 warp     issues the MMAs (24 per stage of 64 tokens), 1 warp the copies of both float32 tiles (TMA)
#include <algorithm>

#include "gemm32_common.cuh"

namespace mxk {
namespace gemm32 {
namespace longk {
namespace {

using namespace umma;

constexpr int kLongRuns = 512;   // tokens from which on the accumulators live for two stages

struct Params {
  CUtensorMap map_a, map_b;   // kWide: boxes of 64 tokens x 32 columns
  const float *a, *b;
  long long lda, ldb;
  float* c;
  long long ldc;
  int c_vec;             // floats per aligned access to a row
  int M, N, K;
  int k_split;           // tokens per split (a multiple of kBK)
  int splits;            // more than one: c is [splits][M][N]
  int run;               // stages that the accumulators live for
  int zero;              // 0, which the compiler does not know
  int* status;
};

// kPair: two CTAs share a tile of 256 rows (cta_group::2), each with 128 columns of A and 64 of B.
template <bool kPair>
struct Config {
  static constexpr int kTileM = kPair ? 2 * kBM : kBM, kBN = kPair ? 128 : 64, kColsB = 64;   // columns of B in this CTA
  static constexpr int kPlaneA = kBM * kBK * 2, kPlaneB = kColsB * kBK * 2;   // bytes
  static constexpr int kStage = 3 * (kPlaneA + kPlaneB), kStages = 2;
  static constexpr int kBox = 32 * kBK * 4, kRaw = (kBM + kColsB) / 32 * kBox, kRaws = 1;   // float32 tiles: boxes of 32 columns, rows of 128 bytes
  static constexpr int kSets = 2;   // accumulators: kBN columns for hi*hi and kBN for the small products, twice
  static constexpr uint32_t kTmem = kSets * 2 * kBN;
  static constexpr int kRawAt = kStages * kStage;
  static constexpr int kBarriers = kRawAt + kRaws * kRaw;
  static constexpr int kBytes = kBarriers + (2 * kStages + 2 * kRaws + 2 * kSets + 2) * 8;
  static constexpr int kEpilogueWarps = 8, kProducerWarps = 12, kWarpsA = 8;
  static constexpr int kMmaWarp = kEpilogueWarps + kProducerWarps, kRawWarp = kMmaWarp + 1;
  static constexpr int kThreads = 32 * (kMmaWarp + 4);   // warpgroups deal registers: 768 threads of 80
  static constexpr int kRegsEpilogue = 104, kRegsProducer = 80, kRegsMma = 32;
  static_assert(kEpilogueWarps * kRegsEpilogue + kProducerWarps * kRegsProducer + 4 * kRegsMma == kThreads / 32 * 80, "the launch's registers");
};

template <bool kPair, bool kWide>
__global__ void __launch_bounds__(Config<kPair>::kThreads, 1) gemm32_long_outer_kernel(const __grid_constant__ Params p) {
  using L = Config<kPair>;
  constexpr int kStages = L::kStages, kSets = L::kSets, kTileM = L::kTileM, BN = L::kBN;
  constexpr int kEpilogueWarps = L::kEpilogueWarps, kProducerWarps = L::kProducerWarps, kMmaWarp = L::kMmaWarp;
  const int mt = (p.M + kTileM - 1) / kTileM, nt = (p.N + BN - 1) / BN;
  const int tiles = mt * nt * p.splits;
  const int first_tile = kPair ? blockIdx.x / 2 : blockIdx.x, tile_step = kPair ? gridDim.x / 2 : gridDim.x;
  enter_kernel(tiles <= tile_step && p.k_split <= 1024);
  const int rank = kPair ? static_cast<int>(cluster_rank()) : 0;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* const full = reinterpret_cast<uint64_t*>(smem + L::kBarriers);   // rank 0: producers of both CTAs -> MMA
  uint64_t* const empty = full + kStages;        // MMA -> producers
  uint64_t* const acc_full = empty + kStages;    // MMA -> epilogue
  uint64_t* const acc_empty = acc_full + kSets;  // epilogue -> MMA
  uint64_t* const raw_full = acc_empty + kSets;  // copies -> producers, the float32 tiles
  uint64_t* const raw_empty = raw_full + L::kRaws;
  uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(raw_empty + L::kRaws);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(&full[s], kProducerWarps * (kPair ? 2 : 1)); mbar_init(&empty[s], 1); }
    for (int s = 0; s < kSets; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], kEpilogueWarps * (kPair ? 2 : 1)); }
    for (int s = 0; s < L::kRaws; ++s) { mbar_init(&raw_full[s], 1); mbar_init(&raw_empty[s], kProducerWarps); }
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
  // (of a pair, either CTA arrives on the other's barriers)
  const auto wait = [&](uint64_t* bar, uint32_t parity) { (kPair ? mbar_wait_cluster_flag : mbar_wait_flag)(bar, parity, timed_out); };
  const auto k_length = [&](int tile) {
    const int sp = tile / (mt * nt);
    return min(p.K, (sp + 1) * p.k_split) - sp * p.k_split;
  };
  if (warp < kEpilogueWarps) {
    // ------------------------------------------------------------ epilogue
    more_registers<L::kRegsEpilogue>();
    constexpr int kChunks = BN / 64;   // of 32 columns
    const int col0 = (warp >> 2) * (BN / 2), row0 = (warp & 3) * 32 + (lane >> 2);   // this thread: rows row0 + 8 i
    float sum[kChunks][4][8];          // [2 j + e]: column 32 c + 8 j + 2 (lane % 4) + e
    int turn = 0;   // accumulators
    for (int tile = first_tile; tile < tiles; tile += tile_step) {
      const int mn = tile % (mt * nt), sp = tile / (mt * nt);
      const int n0 = (mn % nt) * BN + col0, m0 = (mn / nt) * kTileM + rank * kBM + row0;
      const int stages = (k_length(tile) + kBK - 1) / kBK;
#pragma unroll
      for (int c = 0; c < kChunks; ++c)
#pragma unroll
        for (int i = 0; i < 32; ++i) sum[c][i >> 3][i & 7] = 0.f;
#pragma unroll 1
      for (int stage = 0; stage < stages; stage += p.run, ++turn) {
        const int set = turn % kSets;
        wait(&acc_full[set], (turn / kSets) & 1);
        fence_after_sync();
        const uint32_t src = tmem + set * 2 * BN + col0 + (static_cast<uint32_t>((warp & 3) * 32) << 16);
#pragma unroll
        for (int c = 0; c < kChunks; ++c)
#pragma unroll
          for (int h = 0; h < 2; ++h) {   // rows 16 h + lane / 4, + 8
            uint32_t r[16], q[16];
            tmem_ld_16x32(src + c * 32 + (static_cast<uint32_t>(16 * h) << 16), r);
            tmem_ld_16x32(src + BN + c * 32 + (static_cast<uint32_t>(16 * h) << 16), q);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
              for (int i = 0; i < 4; ++i) sum[c][2 * h + (i >> 1)][2 * j + (i & 1)] += __uint_as_float(r[4 * j + i]) + __uint_as_float(q[4 * j + i]);
          }
        fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          if (kPair) arrive_read(&acc_empty[set]);
          else arrive(&acc_empty[set]);
        }
      }
      float* const dst = p.c + (p.splits > 1 ? static_cast<size_t>(sp) * p.M * p.N : 0);
#pragma unroll
      for (int c = 0; c < kChunks; ++c)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int n = n0 + c * 32 + j * 8 + (lane & 3) * 2;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int m = m0 + 8 * i;
            if (m >= p.M || n >= p.N) continue;
            float* const out = dst + m * p.ldc + n;
            if (p.c_vec >= 4 && n + 1 < p.N) {
              *reinterpret_cast<float2*>(out) = make_float2(sum[c][i][2 * j], sum[c][i][2 * j + 1]);
            } else {
              out[0] = sum[c][i][2 * j];
              if (n + 1 < p.N) out[1] = sum[c][i][2 * j + 1];
            }
          }
        }
    }
  } else if (warp < kMmaWarp) {
    // ------------------------------------------------------------ producers
    fewer_registers<L::kRegsProducer>();
    // A warp converts 32 columns x 32 tokens, a column a lane, and leaves vectors of eight tokens: what was contracted over rows
    // becomes K-major on the way.
    const int pw = warp - kEpilogueWarps;
    const bool is_b = pw >= L::kWarpsA;
    const int block = is_b ? pw & 1 : pw & 3, half = is_b ? (pw - L::kWarpsA) >> 1 : pw >> 2;
    const int col = block * 32 + lane, rows = is_b ? L::kColsB : kBM, plane = is_b ? L::kPlaneB : L::kPlaneA;
    int stage = 0, raw = 0;
    uint32_t parity = 1, raw_parity = 0;
    float x[32];
    const auto load = [&](int tile, int seg) {
      if (kWide) {
        wait(&raw_full[raw], raw_parity);
        const uint8_t* const src = smem + L::kRawAt + raw * L::kRaw + ((is_b ? kBM / 32 : 0) + block) * L::kBox + half * 4096 + (lane & 3) * 4;
#pragma unroll
        for (int i = 0; i < 32; ++i) x[i] = read_once(src + i * 128 + ((lane >> 2) ^ (i & 7)) * 16);
        // the tiles may be overwritten once every lane has its values: the vote takes all of them, and the arrival the vote
        uint32_t seen = 0;
#pragma unroll
        for (int i = 0; i < 32; ++i) seen |= __float_as_uint(x[i]);
        const int off = __any_sync(0xffffffffu, seen == 1u) ? p.zero : 0;
        if (lane == 0) arrive(&raw_empty[raw] + off);
        if (++raw == L::kRaws) { raw = 0; raw_parity ^= 1; }
      } else {
        const int mn = tile % (mt * nt), k = tile / (mt * nt) * p.k_split + half * 32 + seg;
        const int c = (is_b ? (mn % nt) * BN + rank * L::kColsB : (mn / nt) * kTileM + rank * kBM) + col, end = is_b ? p.N : p.M;
        const long long ld = is_b ? p.ldb : p.lda;
        const float* const from = (is_b ? p.b : p.a) + k * ld + c;
#pragma unroll
        for (int i = 0; i < 32; ++i) x[i] = k + i < p.K && c < end ? __ldg(from + i * ld) : 0.f;
      }
    };
    if (first_tile < tiles) load(first_tile, 0);
    for (int tile = first_tile; tile < tiles; tile += tile_step) {
      const int k_len = k_length(tile);
#pragma unroll 1
      for (int seg = 0; seg < k_len; seg += kBK) {
        wait(&empty[stage], parity);
        uint8_t* const dst = smem + stage * L::kStage + (is_b ? 3 * L::kPlaneA : 0) + (half * 4 * rows + col) * 16;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint4 hi, mid, lo;
          split8(x + 8 * j, hi, mid, lo);
          *reinterpret_cast<uint4*>(dst + j * rows * 16) = hi;
          *reinterpret_cast<uint4*>(dst + j * rows * 16 + plane) = mid;
          *reinterpret_cast<uint4*>(dst + j * rows * 16 + 2 * plane) = lo;
        }
        fence_smem_to_async();
        __syncwarp();
        if (lane == 0) {
          if (kPair) arrive_written(&full[stage]);
          else arrive(&full[stage]);
        }
        // (not before the arrival: there is one float32 tile, and the next may not have come yet; 65536 tokens of 1024 x 256 206 -> 203 us)
        if (seg + kBK < k_len) load(tile, seg + kBK);
        else if (tile + tile_step < tiles) load(tile + tile_step, 0);
        if (++stage == kStages) { stage = 0; parity ^= 1; }
      }
    }
  } else {
    fewer_registers<L::kRegsMma>();   // (a whole warpgroup's)
    if (warp == kMmaWarp) {
      // ---------------------------------------------------------- tensor core
      const bool leader = elect_one();
      const uint32_t idesc = idesc_bf16(kTileM, BN, false, false);
      int slot = 0, turn = 0;
      uint32_t parity = 0;
      const auto done = [&](uint64_t* bar) {
        if (leader) (kPair ? commit_pair : commit)(bar);
      };
      for (int tile = first_tile; tile < tiles; tile += tile_step) {
        const int k_len = k_length(tile);
        int run = 0;   // stages in the accumulators
        for (int seg = 0; seg < k_len; seg += kBK) {
          if (rank != 0) {   // the other CTA issues; its commits reach this one's barriers
            wait(&empty[slot], parity);
            if (++slot == kStages) { slot = 0; parity ^= 1; }
            continue;
          }
          wait(&full[slot], parity);
          const int set = turn % kSets;
          if (run == 0) wait(&acc_empty[set], ((turn / kSets) & 1) ^ 1);
          fence_after_sync();
          const uint32_t sa = smem_u32(smem + slot * L::kStage), sb = sa + 3 * L::kPlaneA, acc = tmem + set * 2 * BN, low = acc + BN;
          const auto a = [&](int i) { return Operand{sa + i * L::kPlaneA, kBM, false}; };   // hi, mid, lo
          const auto b = [&](int i) { return Operand{sb + i * L::kPlaneB, L::kColsB, false}; };
          const int steps = min(kBK, k_len - seg + 15) / 16;   // of 16 tokens
          const auto product = [&](uint32_t d, const Operand& x, const Operand& y, bool accumulate) {
            const uint64_t dx = x.desc(0), dy = y.desc(0);
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k)
              if (leader && k < steps)
                (kPair ? mma_bf16_pair : mma_bf16)(d, dx + static_cast<uint64_t>(k * x.advance()), dy + static_cast<uint64_t>(k * y.advance()), idesc,
                                                  (accumulate || k > 0) ? 1u : 0u);
          };
          product(low, a(2), b(0), run > 0);
          product(low, a(0), b(2), true);
          product(low, a(1), b(1), true);
          product(low, a(1), b(0), true);
          product(low, a(0), b(1), true);
          product(acc, a(0), b(0), run > 0);
          done(&empty[slot]);
          if (++run == p.run || seg + kBK >= k_len) {
            done(&acc_full[set]);
            ++turn;
            run = 0;
          }
          if (++slot == kStages) { slot = 0; parity ^= 1; }
        }
      }
      // the last commits may still be on their way to barriers in this CTA's shared memory
      for (int s = 0; rank == 0 && s < kStages; ++s) {
        wait(&empty[slot], parity ^ 1);
        if (++slot == kStages) { slot = 0; parity ^= 1; }
      }
    } else if (kWide && warp == L::kRawWarp && lane == 0) {
      // ---------------------------------------------------------- float32 tiles
      int raw = 0;
      uint32_t parity = 1;
      for (int tile = first_tile; tile < tiles; tile += tile_step) {
        const int mn = tile % (mt * nt), m0 = mn / nt * kTileM + rank * kBM, n0 = mn % nt * BN + rank * L::kColsB, k0 = tile / (mt * nt) * p.k_split;
        const int k_len = k_length(tile);
        for (int seg = 0; seg < k_len; seg += kBK) {
          wait(&raw_empty[raw], parity);
          uint8_t* dst = smem + L::kRawAt + raw * L::kRaw;
          tma::expect_bytes(&raw_full[raw], L::kRaw);
          for (int c = 0; c < kBM; c += 32, dst += L::kBox) load_box(dst, &p.map_a, &raw_full[raw], m0 + c, k0 + seg);   // zeros past the matrix
          for (int c = 0; c < L::kColsB; c += 32, dst += L::kBox) load_box(dst, &p.map_b, &raw_full[raw], n0 + c, k0 + seg);
          if (++raw == L::kRaws) { raw = 0; parity ^= 1; }
        }
      }
    }
    __syncwarp();
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

int tile_m(int bn) { return bn == 64 ? kBM : 2 * kBM; }
int tile_ctas(int bn) { return bn == 64 ? 1 : 2; }

template <bool kPair, bool kWide>
int launch(const Params& p, long long ctas, cudaStream_t stream) {
  using L = Config<kPair>;
  if (const int st = allow_smem<gemm32_long_outer_kernel<kPair, kWide>, L::kBytes>(); st != MXK_OK) return st;
  mxk::launch_kernel_clusters(gemm32_long_outer_kernel<kPair, kWide>, kPair ? 2 : 1, static_cast<unsigned>(std::min(ctas, static_cast<long long>(kNumSMs))),
                              L::kThreads, L::kBytes, stream, p);
  return launch_status();
}

}  // namespace

// Pairs, unless one SM's tile is all there is.  The contraction is split so that the SMs' rounds of tiles take the fewest stages (three
// more for a tile's begin and end), each part four stages at least: 1024 x 512 x 24000 in nine parts, two rounds of 42 stages, instead of
// one round of 94 on 64 of the 74 pairs.
Plan plan_outer(int M, int N, int K) {
  Plan pl{M <= 128 || N <= 64 ? 64 : 128, 1, 0};
  const auto ctas = [&] { return static_cast<long long>((M + tile_m(pl.bn) - 1) / tile_m(pl.bn)) * ((N + pl.bn - 1) / pl.bn) * tile_ctas(pl.bn); };
  const int kblocks = (K + kBK - 1) / kBK, most = std::max(1, kblocks / 4);
  if (pl.bn == 128 && ctas() * most < kNumSMs) pl.bn = 64;
  const long long tiles = ctas() / tile_ctas(pl.bn), slots = kNumSMs / tile_ctas(pl.bn);
  if (tiles < slots) {
    long long best = -1;
    for (int n = 1; n <= most && n <= 32; ++n) {
      const long long cost = (tiles * n + slots - 1) / slots * ((kblocks + n - 1) / n + 3);
      if (best < 0 || cost < best) { best = cost; pl.splits = n; }
    }
  }
  const int per = (kblocks + pl.splits - 1) / pl.splits;
  pl.k_split = per * kBK;
  pl.splits = (kblocks + per - 1) / per;
  return pl;
}

int launch_outer(const Plan& pl, const float* a, long long lda, const float* b, long long ldb, float* c, long long ldc, int M, int N, int K, float* partial,
                 int* status, cudaStream_t stream) {
  Params p{};
  p.a = a; p.lda = lda;
  p.b = b; p.ldb = ldb;
  p.c = pl.splits > 1 ? partial : c;
  p.ldc = pl.splits > 1 ? N : ldc;
  p.c_vec = vec_of(p.c, p.ldc);
  p.M = M; p.N = N; p.K = K;
  p.k_split = pl.k_split; p.splits = pl.splits;
  p.run = K < kLongRuns ? 1 : 2;
  p.status = status;
  const bool wide = vec_of(a, lda) >= 4 && vec_of(b, ldb) >= 4;
  if (wide) {
    tma::EncodeTiledFn enc = tma::encode_tiled_fn();
    const auto map = [&](CUtensorMap* m, const float* q, int cols, long long ld) {
      const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(K)}, strides[1] = {static_cast<cuuint64_t>(ld) * 4};
      const cuuint32_t box[2] = {32, kBK}, elem[2] = {1, 1};
      return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(q), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                 CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    if (!enc || !map(&p.map_a, a, M, lda) || !map(&p.map_b, b, N, ldb)) return MXK_ERR_UNSUPPORTED;
  }
  const long long ctas = static_cast<long long>((M + tile_m(pl.bn) - 1) / tile_m(pl.bn)) * ((N + pl.bn - 1) / pl.bn) * pl.splits * tile_ctas(pl.bn);
  if (pl.bn == 128) return wide ? launch<true, true>(p, ctas, stream) : launch<true, false>(p, ctas, stream);
  return wide ? launch<false, true>(p, ctas, stream) : launch<false, false>(p, ctas, stream);
}

}  // namespace longk
}  // namespace gemm32
}  // namespace mxk
