// The Mamba layer between its Dense layers (mamba.py:100-135): causal convolution, SiLU, step sizes and decays, the
// selective scan and its read-out, RMSNorm and gate -- forward and backward -- without the (B, T, H, 16, 16) elements or
// states in memory.
//
// A block owns one (sequence, head) and walks time in stretches of 64 steps: the stretch's 48 channels are convolved into
// shared memory, its four quarters are scanned by four warps from a zero state, the quarters' end states are chained, and
// each warp replays its quarter from the right incoming state (a lane owns 8 of the 256 states; a step is 16 multiply-adds
// for the update and 8 for the read-out).  Bound by dependent steps and barriers (instructions issue in 40 % of the cycles)
// and by the chain of stretches when there are few sequences; the materialised form moved 2 KB per token and head and ran
// about thirty elementwise launches each way.  Outside the scans a thread keeps one channel and slides the taps over its
// rows (with the channel of every element found from its index, and a load per tap, those passes were 40 % of the
// instructions).  128 x 64 steps x 8 heads: 28 -> 17 us; 128 x 250 x 8: 94 -> 58; 1 x 2048 x 8: 425 -> 271.
//
// The backward pass starts every stretch from its saved state and needs sums that are each cheap in one lane layout only,
// so three groups of four warps run side by side: C's cotangent from the states (lane = n), x's (lane = p) and B's
// (lane = n) from the cotangent of the states.  The first group leaves every h_{t-1} in shared memory for the third,
// which has the decay's cotangent <dh_t, h_{t-1}> as a plain dot product (as a difference of larger sums it lost two
// digits).  Sums over lanes are taken for four steps together, 9 shuffles instead of 24.  128 x 64 x 8: 81 -> 59 us,
// 128 x 250 x 8: 321 -> 240, 1 x 2048 x 8: 635 -> 450.
#include "layers.cuh"
#include "mxk_common.cuh"

namespace mxk {
namespace layers {
namespace {

constexpr int kN = 16, kP = 16, kStates = kN * kP;   // per head
constexpr int kQuarter = 16;                         // steps per warp
constexpr int kTaps = 4, kHalo = kTaps - 1;
constexpr int kCh = 3 * 16;                          // channels of a head: x | B | C

__device__ __forceinline__ float sigmoid(float x) { return 1.f / (1.f + __expf(-x)); }
__device__ __forceinline__ float softplus(float x) { return x > 20.f ? x : log1pf(expf(x)); }

// Column of `proj` and channel of the convolution for channel c of head h.
__device__ __forceinline__ int proj_col(int c, int h, int hid) {
  return (c < 16 ? 0 : (c < 32 ? 2 * hid : 3 * hid)) + h * 16 + (c & 15);
}
__device__ __forceinline__ int conv_channel(int c, int h, int hid) { return (c >> 4) * hid + h * 16 + (c & 15); }

// conv_w | conv_b | a_log | dt_bias | d of every head
__host__ __device__ constexpr int partial_floats(int H) { return 48 * H * (kTaps + 1) + 3 * H; }

template <int kLen>
struct Stretch {            // of one head
  float raw[kLen + kHalo][kCh];   // projections, three steps of the past in front
  float act[kLen][kCh];     // silu(conv): x | B | C
  float dt[kLen], decay[kLen], kept[kLen];   // kept: decay, or 0 where a sequence begins
  unsigned char reset[kLen];
};

// The taps of one channel.
struct Taps {
  float w[kTaps], bias;
  __device__ __forceinline__ Taps(const MambaParams& p, int chn) : bias(__ldg(p.conv_b + chn)) {
#pragma unroll
    for (int k = 0; k < kTaps; ++k) w[k] = __ldg(p.conv_w + chn * kTaps + k);
  }
  // of four rows in a row, the oldest first
  __device__ __forceinline__ float operator()(const float* v) const {
    float u = bias;
#pragma unroll
    for (int k = 0; k < kTaps; ++k) u = fmaf(w[k], v[k], u);
    return u;
  }
};

// Convolves and activates the stretch at t0.  A thread has one channel and every row / kGroups of it: its taps and columns are found once, and
// a window slides over its rows.  Threads beyond kGroups x 48 only help with the steps.  Ends with a barrier.
template <int kGroups, int kLen>
__device__ __forceinline__ void load_stretch(Stretch<kLen>& s, const MambaParams& w, const float* __restrict__ proj, long long ld,
                                             const uint8_t* drow, int b, int h, int H, int T, int t0, int tid, int pc, int pg) {
  const int hid = H * 16;
  constexpr int kRows = kLen / kGroups;
  if (pg < kGroups) {
    const float* const col = proj + static_cast<long long>(b) * T * ld + proj_col(pc, h, hid);
#pragma unroll 8
    for (int i = 0; i < kRows; ++i) {
      const int r = i * kGroups + pg, t = t0 + r;
      s.raw[r + kHalo][pc] = t < T ? __ldg(col + t * ld) : 0.f;
    }
    for (int r = pg; r < kHalo; r += kGroups) {
      const int t = t0 + r - kHalo;
      s.raw[r][pc] = (t >= 0 && t < T) ? __ldg(col + t * ld) : 0.f;
    }
  }
  if (tid < kLen) {
    const int t = t0 + tid;
    float dt = 0.f, decay = 1.f;
    if (t < T) {
      dt = softplus(__ldg(proj + (static_cast<long long>(b) * T + t) * ld + 4 * hid + h) + w.dt_bias[h]);
      decay = expf(dt * -expf(w.a_log[h]));
    }
    s.dt[tid] = dt;        // past the end: nothing enters, nothing decays
    s.decay[tid] = decay;
    const unsigned char reset = (t < T && drow) ? drow[t] : 0;
    s.reset[tid] = reset;
    s.kept[tid] = reset ? 0.f : decay;
  }
  __syncthreads();
  if (pg < kGroups) {
    const Taps taps(w, conv_channel(pc, h, hid));
    float v[kTaps];
#pragma unroll
    for (int k = 0; k < kHalo; ++k) v[k + 1] = s.raw[pg * kRows + k][pc];
#pragma unroll 8
    for (int i = 0; i < kRows; ++i) {
      const int r = pg * kRows + i;
#pragma unroll
      for (int k = 0; k < kHalo; ++k) v[k] = v[k + 1];
      v[kHalo] = s.raw[r + kHalo][pc];
      const float u = taps(v);
      s.act[r][pc] = u * sigmoid(u);
    }
  }
  __syncthreads();
}

__device__ __forceinline__ void load8(const float* p, float* v) {   // 16-byte aligned shared memory
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

// kParts: warps, and parts of a stretch.
template <int kParts>
struct FwdSmem {
  Stretch<kParts * kQuarter> s;
  float end[kParts][8][32];           // [part][state of a lane][lane]
  float prod[kParts], dec[kParts];    // product of the decays (0 with a reset), and since the last reset
  int had[kParts];
  float carry[8][32];
  float carry_a;
};

// lane = p + 16 * (n >= 8): states n = 8 * (lane / 16) + j
template <int kParts>
__global__ void __launch_bounds__(kParts * 32) mamba_scan_fwd_kernel(MambaParams w, const float* __restrict__ proj, long long ld,
                                                             const float* __restrict__ h0, const float* __restrict__ a0,
                                                             const uint8_t* __restrict__ done, float* __restrict__ y_pre,
                                                             float* __restrict__ h_last, float* __restrict__ a_last,
                                                             float* __restrict__ states, int T, int H) {
  enter_kernel();
  constexpr int kLen = kParts * kQuarter;
  __shared__ __align__(16) FwdSmem<kParts> sm;
  const int tid = threadIdx.x, lane = tid & 31, q = tid >> 5;
  const int b = blockIdx.x / H, h = blockIdx.x % H, hid = H * 16;
  const int p = lane & 15, n0 = (lane >> 4) * 8;
  const uint8_t* drow = done ? done + static_cast<size_t>(b) * T : nullptr;
  const float skip = w.d[h];
  const int stretches = (T + kLen - 1) / kLen;
  if (q == 0) {
#pragma unroll
    for (int j = 0; j < 8; ++j)
      sm.carry[j][lane] = h0 ? h0[static_cast<size_t>(blockIdx.x) * kStates + (n0 + j) * kP + p] : 0.f;
    if (lane == 0) sm.carry_a = a0 ? a0[blockIdx.x] : 1.f;
  }
  for (int c = 0; c < stretches; ++c) {
    const int t0 = c * kLen;
    load_stretch<kParts / 2>(sm.s, w, proj, ld, drow, b, h, H, T, t0, tid, tid % kCh, tid / kCh);
    float st[8], v8[8];
    // ---- from a zero state: where the quarter ends
    {
#pragma unroll
      for (int j = 0; j < 8; ++j) st[j] = 0.f;
#pragma unroll 4
      for (int i = 0; i < kQuarter; ++i) {
        const int t = q * kQuarter + i;
        const float d = sm.s.kept[t];
        const float xd = sm.s.act[t][p] * sm.s.dt[t];
        load8(&sm.s.act[t][16 + n0], v8);
#pragma unroll
        for (int j = 0; j < 8; ++j) st[j] = fmaf(d, st[j], v8[j] * xd);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) sm.end[q][j][lane] = st[j];
      // the quarter's decays, a lane a step: of all of them, and of those from the last reset on
      const int t = q * kQuarter + p;
      const unsigned resets = __ballot_sync(0xffffffffu, sm.s.reset[t] != 0) & 0xffffu;
      float prod = sm.s.kept[t], dec = p >= 31 - __clz(resets) ? sm.s.decay[t] : 1.f;
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        prod *= __shfl_xor_sync(0xffffffffu, prod, o);
        dec *= __shfl_xor_sync(0xffffffffu, dec, o);
      }
      if (lane == 0) { sm.prod[q] = prod; sm.dec[q] = dec; sm.had[q] = resets != 0; }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 8; ++j) st[j] = sm.carry[j][lane];
    if (q == 0 && states) {
#pragma unroll
      for (int j = 0; j < 8; ++j) states[(static_cast<size_t>(blockIdx.x) * stretches + c) * kStates + (n0 + j) * kP + p] = st[j];
    }
    for (int s2 = 0; s2 < q; ++s2) {
      const float d = sm.prod[s2];
#pragma unroll
      for (int j = 0; j < 8; ++j) st[j] = fmaf(d, st[j], sm.end[s2][j][lane]);
    }
    // ---- replay with the read-out
#pragma unroll 4
    for (int i = 0; i < kQuarter; ++i) {
      const int t = q * kQuarter + i;
      const float d = sm.s.kept[t];
      const float x = sm.s.act[t][p], xd = x * sm.s.dt[t];
      load8(&sm.s.act[t][16 + n0], v8);
#pragma unroll
      for (int j = 0; j < 8; ++j) st[j] = fmaf(d, st[j], v8[j] * xd);
      load8(&sm.s.act[t][32 + n0], v8);
      float y = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) y = fmaf(v8[j], st[j], y);
      y += __shfl_xor_sync(0xffffffffu, y, 16);
      if (lane < 16 && t0 + t < T) y_pre[(static_cast<size_t>(b) * T + t0 + t) * hid + h * 16 + p] = fmaf(skip, x, y);
    }
    __syncthreads();   // carry and summaries have been read
    if (q == kParts - 1) {
#pragma unroll
      for (int j = 0; j < 8; ++j) sm.carry[j][lane] = st[j];
      if (lane == 0) {
        float a = sm.carry_a;
        for (int s2 = 0; s2 < kParts; ++s2) a = sm.had[s2] ? sm.dec[s2] : a * sm.dec[s2];
        sm.carry_a = a;
      }
    }
  }
  if (q == kParts - 1) {
#pragma unroll
    for (int j = 0; j < 8; ++j) h_last[static_cast<size_t>(blockIdx.x) * kStates + (n0 + j) * kP + p] = sm.carry[j][lane];
    if (lane == 0) a_last[blockIdx.x] = sm.carry_a;
  }
}

// ------------------------------------------------------------------------------------------------------ backward
// kParts: warps of a group, and parts of a stretch.
template <int kParts>
struct BwdSmem {
  static constexpr int kLen = kParts * kQuarter;
  Stretch<kLen> s;
  float g[kLen + kHalo][kCh];        // cotangents of the activations, then of the convolution's output; three steps of
                                     // the future behind
  float gy[kLen][16];
  union {
    float end[3][kParts][8][32];     // [task][part]...: where a part ends from nothing
    float4 prev[kLen][2][32];        // h_{t-1}, eight states per lane
    struct {
      float of_group[kTaps + 1][kParts * 96], of_warp[3][kParts * 3];
    } sums;
  };
  float prod[kParts];
  float carry[2][8][32];             // decay-weighted cotangent of the state entering the stretch from the right
  float e[kLen], u0[kLen];           // <dh_t, h_{t-1}>, <dh_t, B_t x_t>
};
constexpr int bwd_blocks(int parts) { return parts == 1 ? 7 : 8 / parts; }   // per SM
template <int kParts> constexpr bool fits = bwd_blocks(kParts) * (sizeof(BwdSmem<kParts>) + 1024) <= 228 * 1024;
static_assert(fits<1> && fits<2> && fits<4>, "blocks per SM");

// Sums over the two halves of a warp: of a in the lower one, of b in the upper one.
__device__ __forceinline__ float halves(float a, float b, int lane) {
  const bool up = lane & 16;
  return (up ? b : a) + __shfl_xor_sync(0xffffffffu, up ? a : b, 16);
}

template <int kParts>
__global__ void __launch_bounds__(kParts * 96, bwd_blocks(kParts)) mamba_scan_bwd_kernel(MambaParams w, const float* __restrict__ proj, long long ld,
                                                                const uint8_t* __restrict__ done,
                                                                const float* __restrict__ states,
                                                                const float* __restrict__ gy_pre,
                                                                const float* __restrict__ gh_last, float* __restrict__ gproj,
                                                                float* __restrict__ gh0, float* __restrict__ partial, int T, int H) {
  enter_kernel();
  extern __shared__ __align__(16) uint8_t raw_smem[];
  BwdSmem<kParts>& sm = *reinterpret_cast<BwdSmem<kParts>*>(raw_smem);
  constexpr int kLen = kParts * kQuarter, kThreads = kParts * 96, kGroups = kThreads / kCh, kRows = kLen / kGroups;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int task = warp / kParts, q = warp % kParts;   // task 0: C (lane = n), 1: x (lane = p), 2: B (lane = n)
  const int b = blockIdx.x / H, h = blockIdx.x % H, hid = H * 16;
  const int l16 = lane & 15, o8 = (lane >> 4) * 8;   // own index, and the first of the eight contracted ones
  const uint8_t* drow = done ? done + static_cast<size_t>(b) * T : nullptr;
  const float skip = w.d[h], neg_a = -expf(w.a_log[h]);
  const int stretches = (T + kLen - 1) / kLen;
  const size_t base = static_cast<size_t>(blockIdx.x) * kStates;
  // state (n, p) of slot j of this lane in this task's layout
  const auto state_at = [&](int j) { return task == 1 ? (o8 + j) * kP + l16 : l16 * kP + o8 + j; };

  if (q == 0 && task > 0) {
#pragma unroll
    for (int j = 0; j < 8; ++j) sm.carry[task - 1][j][lane] = gh_last ? gh_last[base + state_at(j)] : 0.f;
  }
  for (int i = tid; i < kHalo * kCh; i += kThreads) sm.g[kLen + i / kCh][i % kCh] = 0.f;
  const int pc = tid % kCh, pg = tid / kCh;   // outside the scans: thread = channel x kGroups groups of kRows steps
  const int chn = conv_channel(pc, h, hid);
  float gw[kTaps] = {0.f, 0.f, 0.f, 0.f}, gbias = 0.f, ga = 0.f, gdtb = 0.f, gd = 0.f;

  for (int c = stretches - 1; c >= 0; --c) {
    const int t0 = c * kLen;
    for (int i = tid; i < kLen * 16; i += kThreads) {
      const int r = i >> 4, p = i & 15;
      sm.gy[r][p] = t0 + r < T ? __ldg(gy_pre + (static_cast<size_t>(b) * T + t0 + r) * hid + h * 16 + p) : 0.f;
    }
    load_stretch<kGroups>(sm.s, w, proj, ld, drow, b, h, H, T, t0, tid, pc, pg);
    float st[8], a8[8];
    // ---- each quarter from nothing: states forward in time (task 0), their cotangents backward (tasks 1, 2)
#pragma unroll
    for (int j = 0; j < 8; ++j) st[j] = 0.f;
    float prod = 1.f;
#pragma unroll 4
    for (int i = 0; i < kQuarter; ++i) {
      const int t = q * kQuarter + (task == 0 ? i : kQuarter - 1 - i);
      const float d = sm.s.kept[t];
      if (task == 0) {
        const float bd = sm.s.act[t][16 + l16] * sm.s.dt[t];
        load8(&sm.s.act[t][o8], a8);
#pragma unroll
        for (int j = 0; j < 8; ++j) st[j] = fmaf(d, st[j], a8[j] * bd);
      } else {
        const float own = task == 1 ? sm.gy[t][l16] : sm.s.act[t][32 + l16];
        load8(task == 1 ? &sm.s.act[t][32 + o8] : &sm.gy[t][o8], a8);
#pragma unroll
        for (int j = 0; j < 8; ++j) st[j] = d * fmaf(a8[j], own, st[j]);
      }
      prod *= d;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) sm.end[task][q][j][lane] = st[j];
    if (task == 0 && lane == 0) sm.prod[q] = prod;
    __syncthreads();
    // ---- chain
    if (task == 0) {
#pragma unroll
      for (int j = 0; j < 8; ++j) st[j] = states[(static_cast<size_t>(blockIdx.x) * stretches + c) * kStates + state_at(j)];
      for (int s2 = 0; s2 < q; ++s2) {
        const float d = sm.prod[s2];
#pragma unroll
        for (int j = 0; j < 8; ++j) st[j] = fmaf(d, st[j], sm.end[0][s2][j][lane]);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) st[j] = sm.carry[task - 1][j][lane];
      for (int s2 = kParts - 1; s2 > q; --s2) {
        const float d = sm.prod[s2];
#pragma unroll
        for (int j = 0; j < 8; ++j) st[j] = fmaf(d, st[j], sm.end[task][s2][j][lane]);
      }
    }
    __syncthreads();   // summaries and carries have been read; the summaries' memory takes the states
    // ---- replay
    if (task == 0) {
#pragma unroll 2
      for (int i = 0; i < kQuarter; i += 2) {
        float v[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int t = q * kQuarter + i + u;
          const float d = sm.s.kept[t], bd = sm.s.act[t][16 + l16] * sm.s.dt[t];
          sm.prev[t][0][lane] = make_float4(st[0], st[1], st[2], st[3]);
          sm.prev[t][1][lane] = make_float4(st[4], st[5], st[6], st[7]);
          load8(&sm.s.act[t][o8], a8);
#pragma unroll
          for (int j = 0; j < 8; ++j) st[j] = fmaf(d, st[j], a8[j] * bd);
          load8(&sm.gy[t][o8], a8);
          v[u] = 0.f;
#pragma unroll
          for (int j = 0; j < 8; ++j) v[u] = fmaf(a8[j], st[j], v[u]);
        }
        sm.g[q * kQuarter + i + (lane >> 4)][32 + l16] = halves(v[0], v[1], lane);
      }
      asm volatile("bar.arrive %0, 64;" ::"r"(q + 1) : "memory");   // this quarter's states are there
    } else {
      if (task == 2) asm volatile("bar.sync %0, 64;" ::"r"(q + 1) : "memory");
      for (int i = kQuarter - 4; i >= 0; i -= 4) {
        float v[4], e[4];
#pragma unroll
        for (int u = 3; u >= 0; --u) {
          const int t = q * kQuarter + i + u;
          const float d = sm.s.kept[t];
          const float own = task == 1 ? sm.gy[t][l16] : sm.s.act[t][32 + l16];
          load8(task == 1 ? &sm.s.act[t][32 + o8] : &sm.gy[t][o8], a8);
          float x8[8];
          load8(task == 1 ? &sm.s.act[t][16 + o8] : &sm.s.act[t][o8], x8);
          v[u] = 0.f;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            a8[j] = fmaf(a8[j], own, st[j]);   // dh_t
            v[u] = fmaf(x8[j], a8[j], v[u]);
            st[j] = d * a8[j];
          }
          if (task == 2) {
            const float4 p0 = sm.prev[t][0][lane], p1 = sm.prev[t][1][lane];
            e[u] = a8[0] * p0.x + a8[1] * p0.y + a8[2] * p0.z + a8[3] * p0.w;
            e[u] += a8[4] * p1.x + a8[5] * p1.y + a8[6] * p1.z + a8[7] * p1.w;
          }
        }
        float both[4];   // of task 2: e of two steps, and B . (cotangent of B)
#pragma unroll
        for (int u = 0; u < 4; u += 2) {   // a half of the warp per step
          const int t = q * kQuarter + i + u + (lane >> 4);
          const float sum = halves(v[u], v[u + 1], lane);
          if (task == 1) {
            sm.g[t][l16] = fmaf(sm.s.dt[t], sum, skip * sm.gy[t][l16]);
          } else {
            sm.g[t][16 + l16] = sm.s.dt[t] * sum;
            both[u] = halves(e[u], e[u + 1], lane);
            both[u + 1] = sum * sm.s.act[t][16 + l16];
          }
        }
        if (task == 2) {   // four sums over 16 lanes; lane 4 m of a half ends with the one of `both` at m
          const bool b3 = lane & 8, b2 = lane & 4;
          const float r0 = (b3 ? both[2] : both[0]) + __shfl_xor_sync(0xffffffffu, b3 ? both[0] : both[2], 8);
          const float r1 = (b3 ? both[3] : both[1]) + __shfl_xor_sync(0xffffffffu, b3 ? both[1] : both[3], 8);
          float r = (b2 ? r1 : r0) + __shfl_xor_sync(0xffffffffu, b2 ? r0 : r1, 4);
          r += __shfl_xor_sync(0xffffffffu, r, 2);
          r += __shfl_xor_sync(0xffffffffu, r, 1);
          if ((lane & 3) == 0) (b2 ? sm.u0 : sm.e)[q * kQuarter + i + (b3 ? 2 : 0) + (lane >> 4)] = r;
        }
      }
      if (q == 0) {
#pragma unroll
        for (int j = 0; j < 8; ++j) sm.carry[task - 1][j][lane] = st[j];
      }
    }
    __syncthreads();
    // ---- step size and decay
    if (tid < kLen && t0 + tid < T) {
      const long long tok = static_cast<long long>(b) * T + t0 + tid;
      const float gl = sm.s.reset[tid] ? 0.f : sm.s.decay[tid] * sm.e[tid];   // cotangent of the log decay dt * neg_a
      const float logit = __ldg(proj + tok * ld + 4 * hid + h) + w.dt_bias[h];
      const float gdt = (sm.u0[tid] + gl * neg_a) * sigmoid(logit);
      gproj[tok * ld + 4 * hid + h] = gdt;
      gdtb += gdt;
      ga += gl * sm.s.dt[tid] * neg_a;
    }
    // ---- through SiLU; the convolution's weights and bias
    {
      const Taps taps(w, chn);
      float v[kTaps];
#pragma unroll
      for (int k = 0; k < kHalo; ++k) v[k + 1] = sm.s.raw[pg * kRows + k][pc];
#pragma unroll
      for (int i = 0; i < kRows; ++i) {
        const int r = pg * kRows + i;
#pragma unroll
        for (int k = 0; k < kHalo; ++k) v[k] = v[k + 1];
        v[kHalo] = sm.s.raw[r + kHalo][pc];
        const float u = taps(v), sg = sigmoid(u);
        if (pc < 16) gd = fmaf(sm.gy[r][pc], u * sg, gd);
        const float g = t0 + r < T ? sm.g[r][pc] * sg * (1.f + u * (1.f - sg)) : 0.f;
        sm.g[r][pc] = g;
        gbias += g;
#pragma unroll
        for (int k = 0; k < kTaps; ++k) gw[k] = fmaf(g, v[k], gw[k]);
      }
    }
    __syncthreads();
    // ---- through the convolution: inputs
    {
      const Taps taps(w, chn);
      float* const to = gproj + (static_cast<long long>(b) * T + t0 + pg * kRows) * ld + proj_col(pc, h, hid);
      float v[kTaps];   // v[k]: row r + k
#pragma unroll
      for (int k = 0; k < kHalo; ++k) v[k + 1] = sm.g[pg * kRows + k][pc];
#pragma unroll
      for (int i = 0; i < kRows; ++i) {
        const int r = pg * kRows + i;
#pragma unroll
        for (int k = 0; k < kHalo; ++k) v[k] = v[k + 1];
        v[kHalo] = sm.g[r + kHalo][pc];
        float u = 0.f;
#pragma unroll
        for (int k = 0; k < kTaps; ++k) u = fmaf(taps.w[k], v[kHalo - k], u);
        if (t0 + r < T) to[i * ld] = u;
      }
    }
    __syncthreads();
    for (int i = tid; i < kHalo * kCh; i += kThreads) sm.g[kLen + i / kCh][i % kCh] = sm.g[i / kCh][i % kCh];
    __syncthreads();
  }
  if (gh0 && task == 1 && q == 0) {
#pragma unroll
    for (int j = 0; j < 8; ++j) gh0[base + state_at(j)] = sm.carry[0][j][lane];
  }
  // ---- parameter gradients of this (sequence, head)
  float* const row = partial + static_cast<size_t>(b) * partial_floats(H);
  const int channels = 3 * hid;
#pragma unroll
  for (int k = 0; k < kTaps; ++k) sm.sums.of_group[k][tid] = gw[k];
  sm.sums.of_group[kTaps][tid] = gbias;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ga += __shfl_xor_sync(0xffffffffu, ga, o);
    gdtb += __shfl_xor_sync(0xffffffffu, gdtb, o);
    gd += __shfl_xor_sync(0xffffffffu, gd, o);
  }
  if (lane == 0) { sm.sums.of_warp[0][warp] = ga; sm.sums.of_warp[1][warp] = gdtb; sm.sums.of_warp[2][warp] = gd; }
  __syncthreads();
  for (int i = tid; i < (kTaps + 1) * kCh; i += kThreads) {
    const int k = i / kCh, ch = i % kCh, to = conv_channel(ch, h, hid);
    float v = 0.f;
#pragma unroll
    for (int j = 0; j < kGroups; ++j) v += sm.sums.of_group[k][j * kCh + ch];
    row[k < kTaps ? to * kTaps + k : channels * kTaps + to] = v;
  }
  if (tid < 3) {
    float v = 0.f;
#pragma unroll
    for (int i = 0; i < kThreads / 32; ++i) v += sm.sums.of_warp[tid][i];
    row[channels * (kTaps + 1) + tid * H + h] = v;
  }
}

// ----------------------------------------------------------------------------------------------- RMSNorm and gate
constexpr int kGateBlocks = 4 * kNumSMs;

// One warp per token.  kVals: a row of at most 32 x kVals channels is held in registers, all of it on its way at once (0: any row, read
// twice).  65536 tokens of 128: 31 us, 19 now (HBM 16); backward, with the next token's rows ahead and the weight's gradient in registers
// instead of shared memory, 68 and 32 (HBM 26).
template <int kVals>
__global__ void __launch_bounds__(256) mamba_gate_fwd_kernel(MambaParams w, const float* __restrict__ proj, long long ld,
                                                             const float* __restrict__ y_pre, float* __restrict__ z,
                                                             long long tokens, int hid) {
  enter_kernel();
  const int lane = threadIdx.x & 31;
  const long long tok = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  if (tok >= tokens) return;
  const float *y = y_pre + tok * hid, *gate = proj + tok * ld + hid;
  float ss = 0.f;
  if constexpr (kVals > 0) {
    float yv[kVals], gv[kVals], wv[kVals];
#pragma unroll
    for (int v = 0; v < kVals; ++v) {
      const int c = lane + 32 * v;
      yv[v] = c < hid ? y[c] : 0.f;
      gv[v] = c < hid ? __ldg(gate + c) : 0.f;
      wv[v] = c < hid ? __ldg(w.norm_w + c) : 0.f;
    }
#pragma unroll
    for (int v = 0; v < kVals; ++v) ss = fmaf(yv[v], yv[v], ss);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float rstd = rsqrtf(ss / hid + w.eps);
#pragma unroll
    for (int v = 0; v < kVals; ++v)
      if (lane + 32 * v < hid) z[tok * hid + lane + 32 * v] = yv[v] * rstd * wv[v] * (gv[v] * sigmoid(gv[v]));
    return;
  }
  for (int c = lane; c < hid; c += 32) ss = fmaf(y[c], y[c], ss);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  const float rstd = rsqrtf(ss / hid + w.eps);
  for (int c = lane; c < hid; c += 32) {
    const float g = __ldg(gate + c);
    z[tok * hid + c] = y[c] * rstd * w.norm_w[c] * (g * sigmoid(g));
  }
}

template <int kVals>
__global__ void __launch_bounds__(256) mamba_gate_bwd_kernel(MambaParams w, const float* __restrict__ proj, long long ld,
                                                             const float* __restrict__ y_pre, const float* __restrict__ gz,
                                                             float* __restrict__ gy_pre, float* __restrict__ gproj,
                                                             float* __restrict__ norm_partial, long long tokens, int hid) {
  enter_kernel();
  extern __shared__ float acc[];   // [8 warps][hid]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long first = static_cast<long long>(blockIdx.x) * 8 + warp, step = static_cast<long long>(gridDim.x) * 8;
  if constexpr (kVals > 0) {
    float wv[kVals], sum[kVals], yv[kVals], gv[kVals], gz_v[kVals];
    const auto fetch = [&](long long tok) {
#pragma unroll
      for (int v = 0; v < kVals; ++v) {
        const int c = lane + 32 * v;
        const bool in = tok < tokens && c < hid;
        yv[v] = in ? __ldg(y_pre + tok * hid + c) : 0.f;
        gv[v] = in ? __ldg(proj + tok * ld + hid + c) : 0.f;
        gz_v[v] = in ? __ldg(gz + tok * hid + c) : 0.f;
      }
    };
#pragma unroll
    for (int v = 0; v < kVals; ++v) {
      wv[v] = lane + 32 * v < hid ? __ldg(w.norm_w + lane + 32 * v) : 0.f;
      sum[v] = 0.f;
    }
    fetch(first);
    for (long long tok = first; tok < tokens; tok += step) {
      float y[kVals], gt[kVals], g[kVals], sg[kVals], ss = 0.f, dot = 0.f;
#pragma unroll
      for (int v = 0; v < kVals; ++v) {
        y[v] = yv[v];
        gt[v] = gv[v];
        g[v] = gz_v[v];
      }
      fetch(tok + step);
#pragma unroll
      for (int v = 0; v < kVals; ++v) {
        sg[v] = sigmoid(gt[v]);
        ss = fmaf(y[v], y[v], ss);
        dot = fmaf(g[v] * gt[v] * sg[v] * wv[v], y[v], dot);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        ss += __shfl_xor_sync(0xffffffffu, ss, o);
        dot += __shfl_xor_sync(0xffffffffu, dot, o);
      }
      const float rstd = rsqrtf(ss / hid + w.eps);
      const float mean = dot * rstd * rstd / hid;
#pragma unroll
      for (int v = 0; v < kVals; ++v) {
        const int c = lane + 32 * v;
        const float yn = y[v] * rstd, gs = g[v] * gt[v] * sg[v];
        if (c < hid) {
          gy_pre[tok * hid + c] = rstd * gs * wv[v] - mean * yn;
          gproj[tok * ld + hid + c] = g[v] * yn * wv[v] * sg[v] * (1.f + gt[v] * (1.f - sg[v]));
        }
        sum[v] = fmaf(gs, yn, sum[v]);
      }
    }
#pragma unroll
    for (int v = 0; v < kVals; ++v)
      if (lane + 32 * v < hid) acc[warp * hid + lane + 32 * v] = sum[v];
  } else {
    for (int i = threadIdx.x; i < 8 * hid; i += 256) acc[i] = 0.f;
    __syncthreads();
  }
  for (long long tok = first; kVals == 0 && tok < tokens; tok += step) {
    const float *y = y_pre + tok * hid, *gate = proj + tok * ld + hid, *g = gz + tok * hid;
    float ss = 0.f, dot = 0.f;
    for (int c = lane; c < hid; c += 32) {
      const float gt = __ldg(gate + c), gn = g[c] * gt * sigmoid(gt) * w.norm_w[c];
      ss = fmaf(y[c], y[c], ss);
      dot = fmaf(gn, y[c], dot);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ss += __shfl_xor_sync(0xffffffffu, ss, o);
      dot += __shfl_xor_sync(0xffffffffu, dot, o);
    }
    const float rstd = rsqrtf(ss / hid + w.eps);
    const float mean = dot * rstd * rstd / hid;   // mean of (cotangent of the normalised row) * (normalised row), times rstd
    for (int c = lane; c < hid; c += 32) {
      const float gt = __ldg(gate + c), sg = sigmoid(gt), yn = y[c] * rstd;
      const float gs = g[c] * gt * sg;             // cotangent of norm(y) * weight
      gy_pre[tok * hid + c] = rstd * gs * w.norm_w[c] - mean * yn;
      gproj[tok * ld + hid + c] = g[c] * yn * w.norm_w[c] * sg * (1.f + gt * (1.f - sg));
      acc[warp * hid + c] = fmaf(gs, yn, acc[warp * hid + c]);
    }
  }
  __syncthreads();
  for (int c = threadIdx.x; c < hid; c += 256) {
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) t += acc[i * hid + c];
    norm_partial[static_cast<size_t>(blockIdx.x) * hid + c] = t;
  }
}

// Parts of a stretch: a short sequence is one stretch without the steps that it does not have.  (us, forward / backward, with four parts and now:
// 512 x 20 steps x 8 heads 53 / 204 and 33 / 104; 1024 x 1 x 8 93 / 383 and 53 / 106.  At 64 steps and more two parts, four blocks an SM, were no
// faster: 128 x 64 x 8 backward 59 and 59.)
int parts_of(int T) { return T <= kQuarter ? 1 : T <= 2 * kQuarter ? 2 : 4; }

template <int kParts>
int launch_scan_bwd(const MambaParams& w, const float* proj, long long ld, const uint8_t* done, const float* states, const float* gy_pre,
                    const float* gh_last, float* gproj, float* gh0, float* partial, int B, int T, int H, cudaStream_t stream) {
  if (const int st = allow_smem<mamba_scan_bwd_kernel<kParts>, sizeof(BwdSmem<kParts>)>(); st != MXK_OK) return st;
  mxk::launch_kernel(mamba_scan_bwd_kernel<kParts>, B * H, kParts * 96, sizeof(BwdSmem<kParts>), stream, w, proj, ld, done, states, gy_pre, gh_last,
                     gproj, gh0, partial, T, H);
  return launch_status();
}

}  // namespace

size_t mamba_state_floats(int B, int T, int H) {
  const int len = parts_of(T) * kQuarter;
  return static_cast<size_t>(B) * H * ((T + len - 1) / len) * kStates;
}
int mamba_partial_floats(int H) { return partial_floats(H); }
int mamba_gate_blocks(long long tokens) {
  const long long need = (tokens + 7) / 8;
  return static_cast<int>(need < kGateBlocks ? need : kGateBlocks);
}

int mamba_scan_fwd(const MambaParams& w, const float* proj, long long ld, const float* h0, const float* a0, const uint8_t* done,
                   float* y_pre, float* h_last, float* a_last, float* states, int B, int T, int H, cudaStream_t stream) {
  if (B <= 0 || T <= 0 || H <= 0) return MXK_ERR_DIMS;
  const bool whole = parts_of(T) == 4;   // one warp has too few threads for the 48 channels
  mxk::launch_kernel(whole ? mamba_scan_fwd_kernel<4> : mamba_scan_fwd_kernel<2>, B * H, whole ? 128 : 64, 0, stream, w, proj, ld, h0, a0, done, y_pre,
                     h_last, a_last, states, T, H);
  return launch_status();
}

int mamba_scan_bwd(const MambaParams& w, const float* proj, long long ld, const uint8_t* done, const float* states,
                   const float* gy_pre, const float* gh_last, float* gproj, float* gh0,
                   float* partial, int B, int T, int H, cudaStream_t stream) {
  if (B <= 0 || T <= 0 || H <= 0) return MXK_ERR_DIMS;
  const auto launch = parts_of(T) == 1 ? launch_scan_bwd<1> : parts_of(T) == 2 ? launch_scan_bwd<2> : launch_scan_bwd<4>;
  return launch(w, proj, ld, done, states, gy_pre, gh_last, gproj, gh0, partial, B, T, H, stream);
}

int mamba_gate_fwd(const MambaParams& w, const float* proj, long long ld, const float* y_pre, float* z, long long tokens, int H,
                   cudaStream_t stream) {
  const auto kernel = H <= 8 ? mamba_gate_fwd_kernel<4> : H <= 16 ? mamba_gate_fwd_kernel<8> : mamba_gate_fwd_kernel<0>;
  mxk::launch_kernel(kernel, static_cast<unsigned>((tokens + 7) / 8), 256, 0, stream, w, proj, ld, y_pre, z, tokens, 16 * H);
  return launch_status();
}

int mamba_gate_bwd(const MambaParams& w, const float* proj, long long ld, const float* y_pre, const float* gz, float* gy_pre,
                   float* gproj, float* norm_partial, long long tokens, int H, cudaStream_t stream) {
  if (H > kMambaGradHeads) return MXK_ERR_UNSUPPORTED;
  const int hid = 16 * H, bytes = 8 * hid * static_cast<int>(sizeof(float));
  static_assert(8 * 16 * sizeof(float) * kMambaGradHeads <= kMaxSmem, "a row of sums per warp");
  if (bytes > 48 * 1024)
    if (const int st = allow_smem<mamba_gate_bwd_kernel<0>, kMaxSmem>(); st != MXK_OK) return st;
  const auto kernel = H <= 8 ? mamba_gate_bwd_kernel<4> : H <= 16 ? mamba_gate_bwd_kernel<8> : mamba_gate_bwd_kernel<0>;
  mxk::launch_kernel(kernel, mamba_gate_blocks(tokens), 256, bytes, stream, w, proj, ld, y_pre, gz, gy_pre, gproj, norm_partial, tokens, hid);
  return launch_status();
}

}  // namespace layers
}  // namespace mxk
