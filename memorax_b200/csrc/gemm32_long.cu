// float32 products with a weight on the tensor cores (tcgen05), contractions of more than kShortK elements.
//
// A float32 number is the exact sum of three bf16 numbers, and the six largest of the nine products are formed, as in gemm32.cu.  (Two
// scaled float16 numbers take three products, 124 and 106 us at the sizes below, but an element 2^25 below the largest of its row is then
// lost, and with it an output where the large one meets a zero: padding that holds a sentinel, a feature without a weight.)
//
// Precision: the tensor core truncates when it adds to a float32 accumulator (3e-8 of the sum per addition of 16 k), so the hi*hi
// accumulator lives for one stage of 64 k, two at a tile's begin (under the stores of the tile before) and in contractions from 384 on, and is
// summed up in float32 registers; the five small products have an accumulator of their own, whose truncations are 2^-8 as large, for at
// most kLowRun stages.  Errors against float64, relative 2-norm (drained every 512 k, in brackets):
//   65536 x 1024 x 256    normal entries 1.05e-7 (2.3e-7)
//   65536 x 256 x 1024                   1.34e-7 (4.7e-7)    lognormal, sigma 3: 1.3e-7 (4.3e-7)
//   24000 x 1024 x 512                   1.27e-7 (4.7e-7)                        1.2e-7 (3.7e-7)
//
// Bound: the tensor pipe at six products (24 MMAs, 3072 cycles a stage of 256 columns) and, beside it, shared memory: 192 KB read by the
// pipe, 80 KB of tiles and 48 KB of planes written and 32 KB of float32 read, 2750 cycles at 128 bytes.
// Measured with the splitting of the weight (the form of gemm32.cu, whose producers read global memory): 65536 x 1024 x 256 142 us (187),
// 65536 x 256 x 1024 145 us (183), 24000 x 1024 x 512 118 us (133), 65536 x 128 x 256 37.5 us (50), 8192 x 520 x 512 52 us (52).
//
// One persistent CTA per SM, warp-specialised:
//   8 warps    epilogue: accumulators (TMEM) -> sums in registers -> global, whole lines
//   8 warps    producers: float32 tiles, one or two stages ahead in shared memory -> bf16 planes
//   1 warp     issues the MMAs (24 per stage of 64 k), 1 warp the copies of the weight's image, 1 warp those of A (TMA)
// Registers are dealt out by setmaxnreg: a thread of the epilogue holds up to 128 sums.
#include <algorithm>

#include "gemm32_common.cuh"
#include "tma.cuh"

namespace mxk {
namespace gemm32 {
namespace longk {
namespace {

using namespace umma;

constexpr int kLongRuns = 384; // from here on the hi*hi accumulator lives for two stages
constexpr int kFirstRun = 2;   // and always a tile's first: the epilogue is still at the tile before
constexpr int kLowRun = 8;     // stages that the accumulator of the small products lives for

struct Params {
  CUtensorMap map_a;     // kWide: boxes of 128 rows x 32 k
  const float* a;
  long long lda;
  const uint8_t* image;
  float* c;
  long long ldc;
  int c_vec;             // floats per aligned access to a row
  bool vectors;          // eight of C's, four of what is added
  int M, N, K;
  int k_split;           // k per split (a multiple of kBK)
  int splits;            // more than one: c is [splits][M][N]
  int run;               // stages that the hi*hi accumulator lives for after a tile's first run
  int zero;              // 0, which the compiler does not know
  Epilogue ep;           // of a contraction that is not split
  int* status;
};

// kPair: two CTAs share a tile of 256 rows (cta_group::2), each with its 128 rows of A and half of the rows of W.
template <int BN>
struct Config {
  static constexpr bool kPair = BN != 64;
  static constexpr int kTileM = kPair ? 2 * kBM : kBM;
  static constexpr int kRowsB = rows_of(BN);   // rows of W in this CTA
  static constexpr int kPlaneA = kBM * kBK * 2, kPlaneB = kRowsB * kBK * 2;   // bytes
  static constexpr int kStage = 3 * (kPlaneA + kPlaneB), kStages = 2;
  static constexpr int kRaw = kBM * kBK * 4, kRaws = kRowsB == 128 ? 1 : 2;   // float32 tiles of A: two halves of 32 k, rows of 128 bytes
  // accumulators: BN columns for hi*hi and BN for the small products, twice where TMEM has room
  static constexpr int kSets = BN == 256 ? 1 : 2;
  static constexpr uint32_t kTmem = kSets * 2 * BN;
  static constexpr int kRawAt = kStages * kStage;
  static constexpr int kBarriers = kRawAt + kRaws * kRaw;
  static constexpr int kBytes = kBarriers + (3 * kStages + 2 * kRaws + 4 * kSets + 2) * 8;
  static constexpr int kEpilogueWarps = 8, kProducerWarps = 8;
  static constexpr int kMmaWarp = kEpilogueWarps + kProducerWarps, kImageWarp = kMmaWarp + 1, kRawWarp = kMmaWarp + 2;
  static constexpr int kThreads = 32 * (kMmaWarp + 4);   // warpgroups deal registers: 640 threads of 96
  static constexpr int kRegsEpilogue = BN == 256 ? 168 : 152, kRegsProducer = BN == 256 ? 56 : 64, kRegsMma = BN == 256 ? 32 : 48;
  static_assert(kEpilogueWarps * kRegsEpilogue + kProducerWarps * kRegsProducer + 4 * kRegsMma == kThreads / 32 * 96, "the launch's registers");
};

// The tiles of a CTA (pair), one after the other: `n` fastest, then `m`, then the split.  (Taken apart by divisions for every tile, the
// coordinates cost the epilogue 1 to 3 %.)
struct Walk {
  int n, m, sp;
  int step_n, step_m, step_sp;
  __device__ __forceinline__ Walk(int first, int step, int nt, int mt)
      : n(first % nt), m(first / nt % mt), sp(first / nt / mt), step_n(step % nt), step_m(step / nt % mt), step_sp(step / nt / mt) {}
  __device__ __forceinline__ void next(int nt, int mt) {
    n += step_n; m += step_m; sp += step_sp;
    if (n >= nt) { n -= nt; ++m; }
    if (m >= mt) { m -= mt; ++sp; }
  }
};

// kWide: rows of A begin on 16-byte boundaries; where they do not, the producers read them element by element.  kEp: something is
// added on the way out.
// (The instruction cache is small beside this much unrolled code: what is rare is a rolled loop over a copy of the sums in
// local memory, or another instantiation.)
template <int BN, bool kWide, bool kEp>
__global__ void __launch_bounds__(Config<BN>::kThreads, 1) gemm32_long_kernel(const __grid_constant__ Params p) {
  using L = Config<BN>;
  constexpr bool kPair = L::kPair;
  constexpr int kStages = L::kStages, kSets = L::kSets, kTileM = L::kTileM, kRowsB = L::kRowsB;
  constexpr int kEpilogueWarps = L::kEpilogueWarps, kProducerWarps = L::kProducerWarps, kMmaWarp = L::kMmaWarp;
  const int mt = (p.M + kTileM - 1) / kTileM, nt = (p.N + BN - 1) / BN;
  const int tiles = mt * nt * p.splits;
  const int first_tile = kPair ? blockIdx.x / 2 : blockIdx.x, tile_step = kPair ? gridDim.x / 2 : gridDim.x;
  enter_kernel(tiles <= tile_step && p.k_split <= 1024);
  const int rank = kPair ? static_cast<int>(cluster_rank()) : 0;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* const full = reinterpret_cast<uint64_t*>(smem + L::kBarriers);   // producers and the image's copy -> MMA; rank 1: the copy alone
  uint64_t* const empty = full + kStages;          // MMA -> producers, copies
  uint64_t* const peer_full = empty + kStages;     // rank 0: the other CTA's part of the image is there
  uint64_t* const main_full = peer_full + kStages; // MMA -> epilogue, the hi*hi accumulator
  uint64_t* const main_empty = main_full + kSets;  // epilogue -> MMA
  uint64_t* const low_full = main_empty + kSets;   // the same for the small products
  uint64_t* const low_empty = low_full + kSets;
  uint64_t* const raw_full = low_empty + kSets;    // copies -> producers, a float32 tile
  uint64_t* const raw_empty = raw_full + L::kRaws;
  uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(raw_empty + L::kRaws);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(&full[s], (rank == 0 ? kProducerWarps * (kPair ? 2 : 1) : 0) + 1); mbar_init(&empty[s], 1); mbar_init(&peer_full[s], 1); }
    for (int s = 0; s < kSets; ++s) {
      mbar_init(&main_full[s], 1); mbar_init(&low_full[s], 1);
      mbar_init(&main_empty[s], kEpilogueWarps * (kPair ? 2 : 1)); mbar_init(&low_empty[s], kEpilogueWarps * (kPair ? 2 : 1));
    }
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
  const auto k_length = [&](const Walk& at) { return min(p.K - at.sp * p.k_split, p.k_split); };
  if (warp < kEpilogueWarps) {
    // ------------------------------------------------------------ epilogue
    more_registers<L::kRegsEpilogue>();
    constexpr int kChunks = BN / 64;   // of 32 columns
    const int col0 = (warp >> 2) * (BN / 2), row0 = (warp & 3) * 32 + (lane >> 2);   // this thread: rows row0 + 8 i
    float sum[kChunks][4][8];          // columns 32 c + 8 (lane % 4) + e
    int main_turn = 0, low_turn = 0;   // accumulators
    Walk at(first_tile, tile_step, nt, mt);
    for (int tile = first_tile; tile < tiles; tile += tile_step, at.next(nt, mt)) {
      const int sp = at.sp, n0 = at.n * BN + col0, m0 = at.m * kTileM + rank * kBM + row0, stages = (k_length(at) + kBK - 1) / kBK;
#pragma unroll
      for (int c = 0; c < kChunks; ++c)
#pragma unroll
        for (int i = 0; i < 32; ++i) sum[c][i >> 3][i & 7] = 0.f;
      bool low = false;
#pragma unroll 1
      for (int stage = 0;;) {   // one accumulator a turn: hi*hi of a run of stages, the small products of kLowRun of them
        const int turn = low ? low_turn : main_turn, set = turn % kSets;
        wait((low ? low_full : main_full) + set, (turn / kSets) & 1);
        fence_after_sync();
        const uint32_t src = tmem + set * 2 * BN + (low ? BN : 0) + col0 + (static_cast<uint32_t>((warp & 3) * 32) << 16);
#pragma unroll
        for (int c = 0; c < kChunks; ++c)
#pragma unroll
          for (int h = 0; h < 2; ++h) {   // rows 16 h + lane / 4, + 8
            uint32_t r[16];
            tmem_ld_16x32(src + c * 32 + (static_cast<uint32_t>(16 * h) << 16), r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
              for (int i = 0; i < 4; ++i) sum[c][2 * h + (i >> 1)][2 * j + (i & 1)] += __uint_as_float(r[4 * j + i]);
          }
        fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          uint64_t* const bar = (low ? low_empty : main_empty) + set;
          if (kPair) arrive_read(bar);
          else arrive(bar);
        }
        if (low) {
          ++low_turn;
          low = false;
          if (stage == stages) break;
        } else {
          ++main_turn;
          stage = min(stage + (stage == 0 ? kFirstRun : p.run), stages);
          low = stage % kLowRun == 0 || stage == stages;
        }
      }
      float* const dst = p.c + (p.splits > 1 ? static_cast<size_t>(sp) * p.M * p.N : 0);
      if (p.vectors && m0 - row0 + kBM <= p.M && n0 + BN / 2 <= p.N) {   // a whole tile
        float* out = dst + m0 * p.ldc + n0 + (lane & 3) * 8;
#pragma unroll
        for (int c = 0; c < kChunks; ++c, out += 32) {
#pragma unroll
          for (int h = 0; h < 2 && kEp; ++h) {   // four columns
            const int n = n0 + c * 32 + (lane & 3) * 8 + 4 * h;
            float bias[4], scale[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              bias[e] = p.ep.bias ? __ldg(p.ep.bias + n + e) : 0.f;
              scale[e] = p.ep.add_scale ? __ldg(p.ep.add_scale + n + e) : 1.f;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              float* const x = sum[c][i] + 4 * h;
              const float4 ad = p.ep.add ? __ldg(reinterpret_cast<const float4*>(p.ep.add + (m0 + 8 * i) * p.ep.ld_add + n)) : make_float4(0.f, 0.f, 0.f, 0.f);
              x[0] = fmaf(ad.x, scale[0], x[0] + bias[0]);
              x[1] = fmaf(ad.y, scale[1], x[1] + bias[1]);
              x[2] = fmaf(ad.z, scale[2], x[2] + bias[2]);
              x[3] = fmaf(ad.w, scale[3], x[3] + bias[3]);
            }
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) store8(out + 8 * i * p.ldc, 8, 8, sum[c][i]);
        }
      } else {
        float copy[kChunks * 32];
#pragma unroll
        for (int i = 0; i < kChunks * 32; ++i) copy[i] = sum[i >> 5][i >> 3 & 3][i & 7];
#pragma unroll 1
        for (int c = 0; c < kChunks; ++c) {   // a vector of eight columns of four rows, all that is read for it on its way at once (one element
          // after element: 2023 x 16 x 256 with 16 columns added held the launch for 4 us more)
          const int n = n0 + c * 32 + (lane & 3) * 8, left = p.N - n;
          float bias[8], scale[8], add[4][8];
#pragma unroll
          for (int e = 0; e < 8 && kEp; ++e) {
            bias[e] = p.ep.bias && e < left ? __ldg(p.ep.bias + n + e) : 0.f;
            scale[e] = p.ep.add_scale && e < left ? __ldg(p.ep.add_scale + n + e) : 1.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) add[i][e] = p.ep.add && e < left && m0 + 8 * i < p.M ? __ldg(p.ep.add + (m0 + 8 * i) * p.ep.ld_add + n + e) : 0.f;
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float x[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              x[e] = copy[(c * 4 + i) * 8 + e];
              if (kEp) x[e] = fmaf(add[i][e], scale[e], x[e] + bias[e]);
            }
            store8(dst + (m0 + 8 * i) * p.ldc + n, m0 + 8 * i < p.M ? left : 0, p.c_vec, x);
          }
        }
      }
    }
  } else if (warp < kMmaWarp) {
    // ------------------------------------------------------------ producers
    fewer_registers<L::kRegsProducer>();
    // A warp converts 16 rows, in blocks of 8 rows x 32 k; a lane owns 8 consecutive k of a row, eight consecutive lanes eight rows
    // (no bank conflicts on either side: the float32 tile is swizzled).
    const int pw = warp - kEpilogueWarps, r0 = pw * 16 + (lane & 7);
    int stage = 0, raw = 0;
    uint32_t parity = 1, raw_parity = 0;   // a fresh barrier's previous phase counts as complete
    Walk at(first_tile, tile_step, nt, mt);
    for (int tile = first_tile; tile < tiles; tile += tile_step, at.next(nt, mt)) {
      const int k_len = k_length(at);
#pragma unroll 1
      for (int seg = 0; seg < k_len; seg += kBK) {
        float x[2][2][8];
        if (kWide) wait(&raw_full[raw], raw_parity);
        const uint8_t* const src = smem + L::kRawAt + raw * L::kRaw + r0 * 128;
        const int m = at.m * kTileM + rank * kBM + r0, k = at.sp * p.k_split + seg + (lane >> 3) * 8;
        uint32_t seen = 0;
#pragma unroll
        for (int g = 0; g < 2; ++g)
#pragma unroll
          for (int b = 0; b < 2; ++b) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              if (!kWide) {
                const float* const from = p.a + (m + 8 * g) * p.lda + k + 32 * b + 4 * h;
#pragma unroll
                for (int e = 0; e < 4; ++e) x[g][b][4 * h + e] = m + 8 * g < p.M && k + 32 * b + 4 * h + e < p.K ? __ldg(from + e) : 0.f;
                continue;
              }
              read_once(src + b * (L::kRaw / 2) + g * 1024 + (((lane >> 3) * 2 + h) ^ (lane & 7)) * 16, x[g][b] + 4 * h);
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) seen |= __float_as_uint(x[g][b][e]);
          }
        if (kWide) {   // the tile may be overwritten once every lane has its values: the vote takes all of them, and the arrival the vote
          const int off = __any_sync(0xffffffffu, seen == 1u) ? p.zero : 0;
          if (lane == 0) arrive(&raw_empty[raw] + off);
          if (++raw == L::kRaws) { raw = 0; raw_parity ^= 1; }
        }
        wait(&empty[stage], parity);
        uint8_t* const base = smem + stage * L::kStage + ((lane >> 3) * kBM + r0) * 16;
#pragma unroll
        for (int g = 0; g < 2; ++g)
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            uint4 hi, mid, lo;
            split8(x[g][b], hi, mid, lo);
            uint8_t* const dst = base + (b * 4 * kBM + g * 8) * 16;
            *reinterpret_cast<uint4*>(dst) = hi;
            *reinterpret_cast<uint4*>(dst + L::kPlaneA) = mid;
            *reinterpret_cast<uint4*>(dst + 2 * L::kPlaneA) = lo;
          }
        fence_smem_to_async();
        __syncwarp();
        if (lane == 0) {
          if (kPair) arrive_written(&full[stage]);
          else arrive(&full[stage]);
        }
        if (++stage == kStages) { stage = 0; parity ^= 1; }
      }
    }
  } else {
    fewer_registers<L::kRegsMma>();   // (a whole warpgroup's)
    if (warp == kMmaWarp) {
      // ---------------------------------------------------------- tensor core
      const bool leader = elect_one();
      const uint32_t idesc = idesc_bf16(kTileM, BN, false, false);
      int slot = 0, main_turn = 0, low_turn = 0;
      uint32_t parity = 0;
      const auto done = [&](uint64_t* bar) {
        if (leader) (kPair ? commit_pair : commit)(bar);
      };
      Walk at(first_tile, tile_step, nt, mt);
      for (int tile = first_tile; tile < tiles; tile += tile_step, at.next(nt, mt)) {
        const int k_len = k_length(at), stages = (k_len + kBK - 1) / kBK;
        int run = 0;   // stages in the hi*hi accumulator
        for (int stage = 0; stage < stages; ++stage) {
          wait(&full[slot], parity);
          if (kPair && rank != 0) {   // the other CTA issues
            if (leader) arrive_written(&peer_full[slot]);
            __syncwarp();
            if (++slot == kStages) { slot = 0; parity ^= 1; }
            continue;
          }
          if (kPair) wait(&peer_full[slot], parity);
          const uint32_t sa = smem_u32(smem + slot * L::kStage), sb = sa + 3 * L::kPlaneA;
          const auto a = [&](int i) { return Operand{sa + i * L::kPlaneA, kBM, false}; };   // hi, mid, lo
          const auto b = [&](int i) { return Operand{sb + i * L::kPlaneB, kRowsB, false}; };
          const int steps = min(kBK, k_len - stage * kBK + 15) / 16;   // of 16 k
          const auto product = [&](uint32_t d, const Operand& x, const Operand& y, bool accumulate) {
            const uint64_t dx = x.desc(0), dy = y.desc(0);
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k)
              if (leader && k < steps)
                (kPair ? mma_bf16_pair : mma_bf16)(d, dx + static_cast<uint64_t>(k * x.advance()), dy + static_cast<uint64_t>(k * y.advance()), idesc,
                                                  (accumulate || k > 0) ? 1u : 0u);
          };
          const int set = main_turn % kSets, low_set = low_turn % kSets;
          const uint32_t acc = tmem + set * 2 * BN, low = tmem + low_set * 2 * BN + BN;
          if (run == 0) wait(&main_empty[set], ((main_turn / kSets) & 1) ^ 1);
          fence_after_sync();
          product(acc, a(0), b(0), run > 0);
          const bool last = stage + 1 == stages;
          if (++run == (stage < kFirstRun ? kFirstRun : p.run) || last) {
            done(&main_full[set]);
            ++main_turn;
            run = 0;
          }
          const bool fresh = stage % kLowRun == 0;
          if (fresh) {
            wait(&low_empty[low_set], ((low_turn / kSets) & 1) ^ 1);
            fence_after_sync();
          }
          product(low, a(2), b(0), !fresh);
          product(low, a(0), b(2), true);
          product(low, a(1), b(1), true);
          product(low, a(1), b(0), true);
          product(low, a(0), b(1), true);
          done(&empty[slot]);
          if ((stage + 1) % kLowRun == 0 || last) {
            done(&low_full[low_set]);
            ++low_turn;
          }
          if (++slot == kStages) { slot = 0; parity ^= 1; }
        }
      }
      // the last commits may still be on their way to barriers in this CTA's shared memory
      for (int s = 0; s < kStages; ++s) {
        wait(&empty[slot], parity ^ 1);
        if (++slot == kStages) { slot = 0; parity ^= 1; }
      }
    } else if (warp == L::kImageWarp && lane == 0) {
      // ---------------------------------------------------------- the weight's image
      const int k_images = (p.K + kBK - 1) / kBK;
      int stage = 0;
      uint32_t parity = 1;
      Walk at(first_tile, tile_step, nt, mt);
      for (int tile = first_tile; tile < tiles; tile += tile_step, at.next(nt, mt)) {
        const int n0 = at.n * BN + rank * kRowsB, k0 = at.sp * p.k_split, k_len = k_length(at);
        const uint8_t* image = p.image + (static_cast<size_t>(n0 / kRowsB) * k_images + k0 / kBK) * (3 * L::kPlaneB);
        for (int seg = 0; seg < k_len; seg += kBK, image += 3 * L::kPlaneB) {
          wait(&empty[stage], parity);
          tma::expect_bytes(&full[stage], 3 * L::kPlaneB);
          tma::load_bulk(smem + stage * L::kStage + 3 * L::kPlaneA, image, 3 * L::kPlaneB, &full[stage]);
          if (++stage == kStages) { stage = 0; parity ^= 1; }
        }
      }
    } else if (kWide && warp == L::kRawWarp && lane == 0) {
      // ---------------------------------------------------------- float32 tiles of A
      int raw = 0;
      uint32_t parity = 1;
      Walk at(first_tile, tile_step, nt, mt);
      for (int tile = first_tile; tile < tiles; tile += tile_step, at.next(nt, mt)) {
        const int m0 = at.m * kTileM + rank * kBM, k0 = at.sp * p.k_split, k_len = k_length(at);
        for (int seg = 0; seg < k_len; seg += kBK) {
          wait(&raw_empty[raw], parity);
          uint8_t* const dst = smem + L::kRawAt + raw * L::kRaw;
          tma::expect_bytes(&raw_full[raw], L::kRaw);
          load_box(dst, &p.map_a, &raw_full[raw], k0 + seg, m0);   // zeros past the matrix
          load_box(dst + L::kRaw / 2, &p.map_a, &raw_full[raw], k0 + seg + 32, m0);
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

template <int BN, bool kWide, bool kEp>
int launch(const Params& p, long long ctas, cudaStream_t stream) {
  using L = Config<BN>;
  if (const int st = allow_smem<gemm32_long_kernel<BN, kWide, kEp>, L::kBytes>(); st != MXK_OK) return st;
  mxk::launch_kernel_clusters(gemm32_long_kernel<BN, kWide, kEp>, L::kPair ? 2 : 1, static_cast<unsigned>(std::min(ctas, static_cast<long long>(kNumSMs))),
                              L::kThreads, L::kBytes, stream, p);
  return launch_status();
}
template <int BN>
int launch(const Params& p, bool wide, long long ctas, cudaStream_t stream) {
  if (!wide) return launch<BN, false, true>(p, ctas, stream);   // (rare enough to do without a form of its own for no addition)
  return p.ep.bias || p.ep.add ? launch<BN, true, true>(p, ctas, stream) : launch<BN, true, false>(p, ctas, stream);
}

}  // namespace

// 256 x 256 on a pair of SMs reads the least shared memory per product, 256 x 128 where that leaves SMs without a tile or N is
// small, 128 x 64 on one SM where that one does, too.  A contraction is split when even the narrowest tiles leave SMs idle and
// each part still has enough stages to fill the pipeline (four).
Plan plan(int M, int N, int K) {
  Plan pl{256, 1, 0};
  const auto ctas = [&] { return static_cast<long long>((M + tile_m(pl.bn) - 1) / tile_m(pl.bn)) * ((N + pl.bn - 1) / pl.bn) * tile_ctas(pl.bn); };
  const int kblocks = (K + kBK - 1) / kBK, most = std::max(1, kblocks / 4);
  if (N <= 64 || M <= 128) pl.bn = 64;
  else if (N <= 128) pl.bn = 128;
  // without enough k to split, narrower tiles are the only way to occupy more SMs
  while (pl.bn > 64 && ctas() * most < kNumSMs) pl.bn /= 2;
  if (ctas() < kNumSMs && most > 1) pl.splits = static_cast<int>(std::min(static_cast<long long>(most), kNumSMs / ctas()));
  const int per = (kblocks + pl.splits - 1) / pl.splits;
  pl.k_split = per * kBK;
  pl.splits = (kblocks + per - 1) / per;
  return pl;
}

int launch_weights(const Plan& pl, const float* a, long long lda, const void* image, float* c, long long ldc, int M, int N, int K, const Epilogue& ep,
                   float* partial, int* status, cudaStream_t stream) {
  Params p{};
  p.a = a; p.lda = lda;
  p.image = static_cast<const uint8_t*>(image);
  p.c = pl.splits > 1 ? partial : c;
  p.ldc = pl.splits > 1 ? N : ldc;
  p.M = M; p.N = N; p.K = K;
  p.k_split = pl.k_split; p.splits = pl.splits;
  p.run = K < kLongRuns ? 1 : 2;
  if (pl.splits == 1) p.ep = ep;
  p.status = status;
  p.c_vec = vec_of(p.c, p.ldc);
  p.vectors = p.c_vec == 8 && (!p.ep.add || vec_of(p.ep.add, p.ep.ld_add) >= 4);
  const bool wide = vec_of(a, lda) >= 4;
  if (wide) {
    tma::EncodeTiledFn enc = tma::encode_tiled_fn();
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(M)}, strides[1] = {static_cast<cuuint64_t>(lda) * 4};
    const cuuint32_t box[2] = {32, kBM}, elem[2] = {1, 1};
    if (!enc || enc(&p.map_a, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(a), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return MXK_ERR_UNSUPPORTED;
  }
  const long long ctas = static_cast<long long>((M + tile_m(pl.bn) - 1) / tile_m(pl.bn)) * ((N + pl.bn - 1) / pl.bn) * pl.splits * tile_ctas(pl.bn);
  return pl.bn == 256 ? launch<256>(p, wide, ctas, stream) : pl.bn == 128 ? launch<128>(p, wide, ctas, stream) : launch<64>(p, wide, ctas, stream);
}

}  // namespace longk
}  // namespace gemm32
}  // namespace mxk
