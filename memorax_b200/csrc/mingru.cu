// MinGRU's scan with its gate math fused in (min_gru.py:52-78 under the reset rule of memoroid.py:60-91): the two Dense
// pre-activations in, log-space states and read-out out, and the cotangents of the pre-activations back.
//
//   log_state = -softplus(-z) + log g(h~),  decay = -softplus(z),  x_t = logaddexp(decay_t + x_{t-1}, log_state_t)
//
// The states h = exp(x) obey h_t = sigmoid(-z) h_{t-1} + sigmoid(z) g(h~) with positive terms, so the linear form loses
// no relative precision and needs one logarithm per element instead of a logaddexp; where a pre-activation or the carry
// is so large that exp could leave float32's range (kSafe), the block takes the log form for that stretch of time.
//
// Bound: HBM (16 / 24 bytes per element; 30 / 45 us for 12.3 M elements) and about five special-function evaluations
// per element, which have to overlap: time is split over the warps of a block.  A block owns 32 channels of one
// sequence; every thread loads its stretch of at most kSteps steps, folds it into one affine map of the incoming value
// (forward: the state, backward: the carried cotangent; a reset cuts the map's slope), the maps are chained
// through shared memory, and the stretch is replayed from the right incoming value.  Longer sequences take several
// turns.  A stretch that a block takes whole, in the linear form and without a reset, runs through loops without their tests
// (a quarter fewer instructions).  96 x 250 x 512: 59 / 58 us (before, with those tests, one lane alone at a kink and blocks
// of sixteen warps: 96 / 68; one thread per channel walking all of T in log form: 116 / 136), 256 x 256 x 512: 137 / 147
// (206 / 176).  Left: the special functions and the dependent steps between two barriers of a turn.
#include <type_traits>

#include "layers.cuh"
#include "logspace.cuh"
#include "mxk_common.cuh"
#include "warp_tile.cuh"

namespace mxk {
namespace layers {
namespace {

constexpr int kSteps = 8;
// How a block took a turn, and left its states with `forms`.
constexpr uint8_t kLinear = 0, kLog = 1;

// d log g / dh~ jumps at h~ = 0 (from 1/2 to 2), so an element whose sign hangs on the rounding of its dot product is
// decided by the plain float32 sum in the order of k: the branch, and with it the gradient, does not depend on how the
// product was tiled.  Two such sums of terms with random signs differ by about 0.6 x 2^-24 |in| |w|; those below eight
// times 2^-24 |in| |w| are looked at (one in 100 000 at 512 terms), whatever the scale of the inputs and of the weights.
// A sum that is zero because its terms are needs no decision: a row or a channel of zeros has no such range, and where
// zeros of both meet (one-hot inputs, pruned weights) a stretch has several of them, which chance does not give without as
// many others in the range (an element in 4e7 is zero).  Without that distinction zeros cost 27 ms a pass at 96 x 250 x 512.
constexpr float kNearKink = 8.f / 16777216.f;
__device__ __noinline__ float dot_in_order(const float* __restrict__ in, const float* __restrict__ w, int F) {
  float acc = 0.f;
#pragma unroll 32
  for (int k = 0; k < F; ++k) acc = fmaf(in[k], w[k], acc);
  return acc;
}
// The same sum for one element, which is what a stretch mostly has if it has any: the warp brings the rows, every lane adds them up.
// (A lane alone with its loads held its block for 7 us at 512 terms, and the forward pass of 96 x 250 x 512 for 45 of 97.)
constexpr int kChunk = 128;
__device__ __noinline__ float dot_of_warp(const float* __restrict__ in, const float* __restrict__ w, int F, float (*buf)[kChunk], int lane) {
  float x[kChunk / 32], v[kChunk / 32], acc = 0.f;
  const auto load = [&](int k0) {
#pragma unroll
    for (int u = 0; u < kChunk / 32; ++u) {
      const int k = k0 + u * 32 + lane;
      x[u] = k < F ? __ldg(in + k) : 0.f;
      v[u] = k < F ? __ldg(w + k) : 0.f;
    }
  };
  load(0);
  for (int k0 = 0; k0 < F; k0 += kChunk) {
#pragma unroll
    for (int u = 0; u < kChunk / 32; ++u) {
      buf[0][u * 32 + lane] = x[u];
      buf[1][u * 32 + lane] = v[u];
    }
    __syncwarp();
    if (k0 + kChunk < F) load(k0 + kChunk);
    if (k0 + kChunk <= F) {
#pragma unroll 8
      for (int k = 0; k < kChunk; k += 4) {
        const float4 a = *reinterpret_cast<const float4*>(&buf[0][k]), b = *reinterpret_cast<const float4*>(&buf[1][k]);
        acc = fmaf(a.x, b.x, acc);
        acc = fmaf(a.y, b.y, acc);
        acc = fmaf(a.z, b.z, acc);
        acc = fmaf(a.w, b.w, acc);
      }
    } else {
      for (int k = 0; k < F - k0; ++k) acc = fmaf(buf[0][k], buf[1][k], acc);
    }
    __syncwarp();
  }
  return acc;
}
constexpr int kFewNear = 4;   // elements of a step up to which the warp takes them one by one

// Two-norms of the rows of a (rows_a, F), then of those of b (rows_b, F); a warp each.  0 where the squares leave float32's
// range: the gates are saturated there.  HBM-bound: one read of a.
__global__ void __launch_bounds__(256) row_norms_kernel(const float* __restrict__ a, long long rows_a, const float* __restrict__ b,
                                                        long long rows_b, int F, bool wide, float* __restrict__ out) {
  enter_kernel();
  const long long row = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= rows_a + rows_b) return;
  const float* const p = row < rows_a ? a + row * F : b + (row - rows_a) * F;
  float s[4] = {};
  if (wide) {
#pragma unroll 4
    for (int k = lane * 4; k < F; k += 128) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(p + k));
      s[0] = fmaf(v.x, v.x, s[0]); s[1] = fmaf(v.y, v.y, s[1]);
      s[2] = fmaf(v.z, v.z, s[2]); s[3] = fmaf(v.w, v.w, s[3]);
    }
  } else {
#pragma unroll 4
    for (int k = lane; k < F; k += 32) s[0] = fmaf(p[k], p[k], s[0]);
  }
  float sum = (s[0] + s[1]) + (s[2] + s[3]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (lane == 0) out[row] = sum < INFINITY ? sqrtf(sum) : 0.f;
}

// Largest |z|, |h~| and carried x for which the linear form stays inside float32: every state is at least e^-40, and what
// a product of decays below e^-87 would have contributed is below 1e-11 of it.
constexpr float kSafe = 20.f;

// exp, log and reciprocal inside that range (no denormals: the .ftz forms need no scaling around the special-function
// unit, which is most of what the general ones issue)
__device__ __forceinline__ float exp_safe(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x * 1.4426950408889634f));
  return y;
}
__device__ __forceinline__ float log_safe(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y * 0.6931471805599453f;
}
__device__ __forceinline__ float rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Reset bits of `count` (at most kSteps) steps from t_begin on; the warp's lanes read one byte each.
__device__ __forceinline__ unsigned reset_mask(const uint8_t* drow, int t_begin, int count, int lane) {
  const bool reset = drow && lane < count && drow[t_begin + lane] != 0;
  return __ballot_sync(0xffffffffu, reset);
}

// kSegs: warps of a block, and parts of a turn's time.
template <int kSegs>
__global__ void __launch_bounds__(32 * kSegs, 32 / kSegs)
mingru_fwd_kernel(const float* __restrict__ z, const float* ht, float* ht_kink, const float* __restrict__ dense_in,
                  const float* __restrict__ dense_w, const float* __restrict__ norms, int F, long long ld,
                  const float* __restrict__ x0, const float* __restrict__ a0, const uint8_t* __restrict__ done,
                  float* __restrict__ states, uint8_t* __restrict__ forms, float* __restrict__ y, float* __restrict__ x_last,
                  float* __restrict__ a_last, int B, int T, int D, int turn_len) {
  enter_kernel();
  __shared__ float sa[kSegs][32], sq[kSegs][32], sd[kSegs][32];
  __shared__ unsigned sr[kSegs];   // reset bits of a stretch
  __shared__ __align__(16) float rows[kSegs][2][kChunk];
  __shared__ float carry_x[32], carry_a[32];
  const int lane = threadIdx.x & 31, seg = threadIdx.x >> 5;
  const int groups = (D + 31) / 32;
  const int b = blockIdx.x / groups, d = (blockIdx.x % groups) * 32 + lane;
  const bool in = d < D;
  const uint8_t* drow = done ? done + static_cast<size_t>(b) * T : nullptr;
  const int len = (turn_len + kSegs - 1) / kSegs;
  if (seg == 0) {
    carry_x[lane] = (in && x0) ? x0[static_cast<size_t>(b) * D + d] : -INFINITY;
    carry_a[lane] = (in && a0) ? a0[static_cast<size_t>(b) * D + d] : 0.f;
  }
  const auto form_at = [&](int turn_no) { return static_cast<size_t>(blockIdx.x) * ((T + turn_len - 1) / turn_len) + turn_no; };
  const int step = static_cast<int>(ld);
  const float range = (ht_kink && in) ? kNearKink * __ldg(norms + static_cast<long long>(B) * T + d) : 0.f;
  for (int turn = 0; turn < T; turn += turn_len) {
    const int t_begin = turn + seg * len, t_end = min(min(T, turn + turn_len), t_begin + len);
    const int count = t_end - t_begin;   // steps of this warp (may be negative)
    // (nearly every warp's stretch is whole and without a reset: its loops are kept free of what the others ask step by step)
    const bool whole = __all_sync(0xffffffffu, in && count == kSteps);
    float lv[kSteps], dv[kSteps];
    {
      const long long token = static_cast<long long>(b) * T + t_begin;
      const float *pz = z + token * ld + d, *ph = ht + token * ld + d;
      if (whole) {
#pragma unroll
        for (int i = 0; i < kSteps; ++i) {
          lv[i] = ld_stream(pz + i * step);
          dv[i] = ld_stream(ph + i * step);
        }
      } else {
#pragma unroll
        for (int i = 0; i < kSteps; ++i) {
          const bool on = in && i < count;
          lv[i] = on ? ld_stream(pz + i * step) : 0.f;
          dv[i] = on ? ld_stream(ph + i * step) : 1.f;
        }
      }
    }
    const unsigned resets = reset_mask(drow, t_begin, count, lane);
    const bool plain = whole && resets == 0;
    float most = 0.f;
#pragma unroll
    for (int i = 0; i < kSteps; ++i) most = fmaxf(most, fmaxf(fabsf(lv[i]), fabsf(dv[i])));
    if (ht_kink) {
      const long long token0 = static_cast<long long>(b) * T + t_begin;
      const float norm = lane < count ? __ldg(norms + token0 + lane) : 0.f;
      unsigned near = 0, zero = 0;
#pragma unroll
      for (int i = 0; i < kSteps; ++i) {
        if (fabsf(dv[i]) < range * __shfl_sync(0xffffffffu, norm, i)) near |= 1u << i;
        if (dv[i] == 0.f) zero |= 1u << i;
      }
      if (__any_sync(0xffffffffu, near != 0)) {
        if (__reduce_add_sync(0xffffffffu, __popc(near & zero) - __popc(near & ~zero)) > 1) near &= ~zero;
#pragma unroll
        for (int i = 0; i < kSteps; ++i) {
          unsigned lanes = __ballot_sync(0xffffffffu, near >> i & 1u);
          if (lanes == 0) continue;
          const float* const row = dense_in + (token0 + i) * F;
          if (__popc(lanes) <= kFewNear) {
            for (; lanes; lanes &= lanes - 1) {
              const int l = __ffs(lanes) - 1;
              const float v = dot_of_warp(row, dense_w + static_cast<long long>(d - lane + l) * F, F, rows[seg], lane);
              if (lane == l) dv[i] = v;
            }
          } else if (near >> i & 1u) {
            dv[i] = dot_in_order(row, dense_w + static_cast<long long>(d) * F, F);
          }
          if (near >> i & 1u) ht_kink[(token0 + i) * ld + d] = dv[i];
        }
      }
    }
    const bool linear = !__syncthreads_or(!(most <= kSafe) || (seg == 0 && !(carry_x[lane] <= kSafe)));
    const size_t out0 = (static_cast<size_t>(b) * T + t_begin) * D + d;
    if (forms && threadIdx.x == 0) forms[form_at(turn / turn_len)] = linear ? kLinear : kLog;
    if (linear) {
      // h -> A h + Q; dec: decays since the last reset
      float A = 1.f, Q = 0.f, dec = 0.f, prod = 1.f;
#pragma unroll
      for (int i = 0; i < kSteps; ++i) {
        const float zi = lv[i], hi = dv[i];
        const float e = exp_safe(-fabsf(zi)), r = rcp(1.f + e), er = e * r;   // sigmoid(|z|), sigmoid(-|z|)
        const float sh = rcp(1.f + exp_safe(-hi)), g = hi >= 0.f ? hi + 0.5f : sh;
        lv[i] = (zi >= 0.f ? r : er) * g;
        dv[i] = zi >= 0.f ? er : r;
      }
      const auto fold = [&](auto asked) {   // four decays are at least e^-80
#pragma unroll
        for (int i = 0; i < kSteps; ++i) {
          if (!asked.value || i < count) {
            if (asked.value && (resets >> i & 1u)) { A = 0.f; Q = lv[i]; dec = 0.f; prod = dv[i]; }
            else { A *= dv[i]; Q = fmaf(dv[i], Q, lv[i]); prod *= dv[i]; }
          }
          if (i % 4 == 3) { dec += log_safe(prod); prod = 1.f; }
        }
      };
      if (plain) fold(std::false_type());
      else fold(std::true_type());
      sa[seg][lane] = A;
      sq[seg][lane] = Q;
      sd[seg][lane] = dec;
      if (lane == 0) sr[seg] = resets;
      float cur = exp_ls(carry_x[lane]);
      __syncthreads();
      // (a stretch with a reset forgets what comes in, finite or not)
      for (int s2 = 0; s2 < seg; ++s2) cur = sr[s2] ? sq[s2][lane] : fmaf(sa[s2][lane], cur, sq[s2][lane]);
      float *const ps = states + out0, *const py = y + out0;
      if (plain && states && forms && y) {
#pragma unroll
        for (int i = 0; i < kSteps; ++i) {
          cur = fmaf(dv[i], cur, lv[i]);
          st_stream(ps + i * D, cur);
          st_stream(py + i * D, cur);
        }
      } else {
#pragma unroll
        for (int i = 0; i < kSteps; ++i) {
          if (i < count) {
            cur = (resets >> i & 1u) ? lv[i] : fmaf(dv[i], cur, lv[i]);
            if (in) {
              if (states) st_stream(ps + i * D, forms ? cur : log_safe(cur));
              if (y) st_stream(py + i * D, cur);
            }
          }
        }
      }
      if (t_begin < t_end && t_end == min(T, turn + turn_len)) {
        // the thread that holds the turn's last step: the carry of the next turn
        float acc = carry_a[lane];
        for (int s2 = 0; s2 < kSegs; ++s2) acc = sr[s2] ? sd[s2][lane] : acc + sd[s2][lane];
        carry_a[lane] = acc;
        carry_x[lane] = log_safe(cur);
      }
      __syncthreads();
      continue;
    }
    // log form: x -> logaddexp(A + x, Q)
    float A = 0.f, Q = -INFINITY, dec = 0.f;
#pragma unroll
    for (int i = 0; i < kSteps; ++i) {
      if (i < count) {
        const float zi = lv[i], hi = dv[i];
        const float lz = log1p_ls(exp_ls(-fabsf(zi)));   // shared by softplus(z) and softplus(-z)
        lv[i] = log_g(hi) - (fmaxf(-zi, 0.f) + lz);
        dv[i] = -(fmaxf(zi, 0.f) + lz);
        if (resets >> i & 1u) { A = -INFINITY; Q = lv[i]; dec = dv[i]; }
        else { A += dv[i]; Q = log_add_exp(dv[i] + Q, lv[i]); dec += dv[i]; }
      }
    }
    sa[seg][lane] = A;
    sq[seg][lane] = Q;
    sd[seg][lane] = dec;
    if (lane == 0) sr[seg] = resets;
    __syncthreads();
    float cur = carry_x[lane];
    for (int s2 = 0; s2 < seg; ++s2) cur = sr[s2] ? sq[s2][lane] : log_add_exp(sa[s2][lane] + cur, sq[s2][lane]);
    __syncthreads();   // every segment has read the carry
#pragma unroll
    for (int i = 0; i < kSteps; ++i) {
      if (i < count) {
        cur = (resets >> i & 1u) ? lv[i] : log_add_exp(dv[i] + cur, lv[i]);
        if (in) {
          if (states) st_stream(states + out0 + static_cast<size_t>(i) * D, cur);
          if (y) st_stream(y + out0 + static_cast<size_t>(i) * D, exp_ls(cur));
        }
      }
    }
    if (t_begin < t_end && t_end == min(T, turn + turn_len)) {
      float acc = carry_a[lane];
      for (int s2 = 0; s2 < kSegs; ++s2) acc = sr[s2] ? sd[s2][lane] : acc + sd[s2][lane];
      carry_a[lane] = acc;
      carry_x[lane] = cur;
    }
    __syncthreads();
  }
  if (seg == 0 && in) {
    if (x_last) x_last[static_cast<size_t>(b) * D + d] = carry_x[lane];
    if (a_last) a_last[static_cast<size_t>(b) * D + d] = carry_a[lane];
  }
}

// states, forms: as the forward kernel left them (without forms: log states)
template <int kSegs>
__global__ void __launch_bounds__(32 * kSegs, 32 / kSegs)
mingru_bwd_kernel(const float* __restrict__ z, const float* __restrict__ ht, long long ld, const float* __restrict__ states,
                  const uint8_t* __restrict__ forms, const float* __restrict__ x0, const uint8_t* __restrict__ done,
                  const float* __restrict__ gx, const float* __restrict__ gy, const float* __restrict__ gx_last,
                  float* __restrict__ gz, float* __restrict__ gh, float* __restrict__ gx0, int B, int T, int D, int turn_len) {
  enter_kernel();
  __shared__ float sp[kSegs][32], sq[kSegs][32];
  __shared__ float carry[32];
  const int lane = threadIdx.x & 31, seg = threadIdx.x >> 5;
  const int groups = (D + 31) / 32;
  const int b = blockIdx.x / groups, d = (blockIdx.x % groups) * 32 + lane;
  const bool in = d < D;
  const uint8_t* drow = done ? done + static_cast<size_t>(b) * T : nullptr;
  const int len = (turn_len + kSegs - 1) / kSegs;
  const int step = static_cast<int>(ld);
  if (seg == 0) carry[lane] = (in && gx_last) ? gx_last[static_cast<size_t>(b) * D + d] : 0.f;
  for (int turn = (T - 1) / turn_len * turn_len; turn >= 0; turn -= turn_len) {
    const int t_begin = turn + seg * len, t_end = min(min(T, turn + turn_len), t_begin + len);
    const int count = t_end - t_begin;   // steps of this warp (may be negative)
    const size_t at0 = (static_cast<size_t>(b) * T + t_begin) * D + d;
    const long long io0 = (static_cast<long long>(b) * T + t_begin) * ld + d;
    // how this turn's states are stored, and the one in front of this warp's first step
    const auto stored = [&](int turn_no) { return forms ? forms[static_cast<size_t>(blockIdx.x) * ((T + turn_len - 1) / turn_len) + turn_no] : kLog; };
    const bool logs = stored(turn / turn_len) == kLog;
    const bool prev_log = t_begin == 0 || (t_begin > turn ? logs : stored(turn / turn_len - 1) == kLog);
    float zv[kSteps], hv[kSteps], sv[kSteps], e[kSteps], w[kSteps], prev = 0.f;
    const bool whole = __all_sync(0xffffffffu, in && count == kSteps);
    {
      const float *const pz = z + io0, *const ph = ht + io0, *const ps = states + at0, *const pg = gy + at0;
      if (in && count > 0) prev = t_begin > 0 ? ps[-D] : (x0 ? x0[static_cast<size_t>(b) * D + d] : -INFINITY);
      if (whole && gy) {
#pragma unroll
        for (int i = 0; i < kSteps; ++i) {
          zv[i] = ld_stream(pz + i * step);
          hv[i] = ld_stream(ph + i * step);
          sv[i] = ld_stream(ps + i * D);
          e[i] = ld_stream(pg + i * D);
        }
      } else {
#pragma unroll
        for (int i = 0; i < kSteps; ++i) {
          const bool on = in && i < count;
          zv[i] = on ? ld_stream(pz + i * step) : 0.f;
          hv[i] = on ? ld_stream(ph + i * step) : 0.f;
          sv[i] = on ? ld_stream(ps + i * D) : (logs ? 0.f : 1.f);
          e[i] = (on && gy) ? ld_stream(pg + i * D) : 0.f;
        }
      }
    }
    const unsigned resets = reset_mask(drow, t_begin, count, lane);
    const bool plain = whole && resets == 0;
    bool linear = !logs;
    if (!forms) {
      float most = (t_begin == 0 && x0) ? fmaxf(prev, 0.f) : 0.f;
#pragma unroll
      for (int i = 0; i < kSteps; ++i) most = fmaxf(most, fmaxf(fabsf(zv[i]), fabsf(hv[i])));
      linear = !__syncthreads_or(!(most <= kSafe));
    }
    // w_t = share of the incoming state in x_t; carry' = w (e + carry), right to left
    float P = 1.f, Q = 0.f;
    if (linear) {
      if (logs) {
#pragma unroll
        for (int i = 0; i < kSteps; ++i) sv[i] = exp_ls(sv[i]);
      }
      if (prev_log) prev = exp_ls(prev);
      if (gx && in) {
#pragma unroll
        for (int i = 0; i < kSteps; ++i) e[i] = i < count ? fmaf(e[i], sv[i], gx[at0 + static_cast<size_t>(i) * D]) : 0.f;
      } else {
#pragma unroll
        for (int i = 0; i < kSteps; ++i) e[i] *= sv[i];
      }
      const auto fold = [&](auto asked) {
#pragma unroll
        for (int i = kSteps - 1; i >= 0; --i) {
          const float ez = exp_safe(-fabsf(zv[i])), r = rcp(1.f + ez), er = ez * r;
          const float share = (zv[i] >= 0.f ? er : r) * (i > 0 ? sv[i > 0 ? i - 1 : 0] : prev) * rcp(sv[i]);
          w[i] = asked.value && (resets >> i & 1u) ? 0.f : share;
          zv[i] = zv[i] >= 0.f ? r : er;   // sigmoid(z)
          if (!asked.value || i < count) {
            Q = w[i] * (e[i] + Q);
            P *= w[i];
          }
        }
      };
      if (plain) fold(std::false_type());
      else fold(std::true_type());
    } else {
      // log form, from the log states
      if (!prev_log) prev = logf(prev);
#pragma unroll
      for (int i = kSteps - 1; i >= 0; --i) {
        w[i] = 0.f;
        if (i < count) {
          e[i] = e[i] != 0.f ? e[i] * exp_ls(sv[i]) : 0.f;
          if (gx && in) e[i] += gx[at0 + static_cast<size_t>(i) * D];
          const float ez = exp_ls(-fabsf(zv[i]));
          if (!(resets >> i & 1u)) {
            const float p = -(fmaxf(zv[i], 0.f) + log1p_ls(ez)) + (i > 0 ? sv[i > 0 ? i - 1 : 0] : prev);
            w[i] = p == -INFINITY ? 0.f : exp_ls(p - sv[i]);
          }
          zv[i] = (zv[i] >= 0.f ? 1.f : ez) / (1.f + ez);
          Q = w[i] * (e[i] + Q);
          P *= w[i];
        }
      }
    }
    sp[seg][lane] = P;
    sq[seg][lane] = Q;
    __syncthreads();
    float c = carry[lane];
    for (int s2 = kSegs - 1; s2 > seg; --s2) c = fmaf(sp[s2][lane], c, sq[s2][lane]);
    __syncthreads();   // every segment has read the carry
    float *const oz = gz + io0, *const oh = gh + io0;
    const auto replay = [&](auto asked) {
#pragma unroll
      for (int i = kSteps - 1; i >= 0; --i) {
        if (!asked.value || i < count) {
          const float g = e[i] + c, g_d = w[i] * g, g_ls = (1.f - w[i]) * g;
          c = g_d;
          // d(-softplus(-z))/dz = 1 - sigmoid(z), d(-softplus(z))/dz = -sigmoid(z)
          const float dg = rcp(hv[i] >= 0.f ? hv[i] + 0.5f : 1.f + exp_safe(hv[i]));
          if (!asked.value || in) {
            st_stream(oz + i * step, fmaf(-zv[i], g, g_ls));
            st_stream(oh + i * step, g_ls * dg);
          }
        }
      }
    };
    if (plain) replay(std::false_type());
    else replay(std::true_type());
    if (seg == 0) carry[lane] = c;
  }
  if (seg == 0 && in && gx0) gx0[static_cast<size_t>(b) * D + d] = carry[lane];
}

template <int kSplit>
__global__ void __launch_bounds__(128)
mingru_step_kernel(const float* __restrict__ in, const float* __restrict__ w_z, const float* __restrict__ w_h,
                   const float* __restrict__ x0, const float* __restrict__ a0, const uint8_t* __restrict__ done,
                   float* __restrict__ x, float* __restrict__ y, float* __restrict__ a_last, int B, int F, int D) {
  enter_kernel();
  const TilePlace<kSplit> at_tile;
  const int lane = at_tile.lane;
  const int units = (D + 1) / 2;
  const int d0 = (at_tile.tile % units) * 2, m0 = (at_tile.tile / units) * 8;
  if (m0 >= B) return;
  const size_t r0 = static_cast<size_t>(d0) * F, r1 = static_cast<size_t>(min(d0 + 1, D - 1)) * F;
  const float* rows[4] = {w_z + r0, w_h + r0, w_z + r1, w_h + r1};
  WarpTile acc;
  acc.accumulate(in + static_cast<size_t>(m0) * F, F, min(8, B - m0), rows, F, at_tile.first, at_tile.step);
  float v = acc.reduce(lane);
  if (!join_warps<kSplit>(v, lane)) return;
  const float other = __shfl_xor_sync(0xffffffffu, v, 1);
  const int m = m0 + (lane >> 2), d = d0 + ((lane >> 1) & 1);
  if ((lane & 1) || m >= B || d >= D) return;   // even lanes hold z, their neighbours h~
  const float lz = log1p_ls(exp_ls(-fabsf(v)));
  const float ls = log_g(other) - (fmaxf(-v, 0.f) + lz), dec = -(fmaxf(v, 0.f) + lz);
  const size_t at = static_cast<size_t>(m) * D + d;
  const bool reset = done && done[m] != 0;
  const float cur = reset ? ls : log_add_exp(dec + (x0 ? x0[at] : -INFINITY), ls);
  x[at] = cur;
  y[at] = exp_ls(cur);
  if (a_last) a_last[at] = reset ? dec : dec + (a0 ? a0[at] : 0.f);
}

unsigned blocks_of(int B, int D) { return static_cast<unsigned>(static_cast<long long>(B) * ((D + 31) / 32)); }
// Warps of a block.  Two blocks of sixteen fit an SM: as long as the grid fits so, they halve the turns (us, forward / backward: 1 x 1000 x 64
// 29 / 22 with sixteen, 42 / 34 with eight; 8 x 250 x 512 28 / 8 and 35 / 12).  Above, four blocks of eight keep an SM at it while one of
// them waits at its barriers, and a grid up to twice that size is one wave instead of two (19 x 250 x 512: 32 / 18 and 20 / 16;
// 96 x 250 x 512 backward: 60 and 55).
int segments(int B, int D) { return blocks_of(B, D) > 2 * kNumSMs ? 8 : 16; }
// Steps a block takes per turn: as evenly divided as the stretches allow (T = 250 is two turns of 125, not 128 + 122).
int turn_length(int B, int T, int D) {
  const int most = segments(B, D) * kSteps, turns = (T + most - 1) / most;
  return (T + turns - 1) / turns;
}
int check_dims(int B, int T, int D) {
  return (B <= 0 || T <= 0 || D <= 0 || static_cast<long long>(B) * ((D + 31) / 32) > 0x7fffffffLL) ? MXK_ERR_DIMS : MXK_OK;
}

}  // namespace

int row_norms(const float* a, long long rows_a, const float* b, long long rows_b, int F, float* out, cudaStream_t stream) {
  const bool wide = F % 4 == 0 && aligned16(a) && aligned16(b);
  mxk::launch_kernel(row_norms_kernel, static_cast<unsigned>((rows_a + rows_b + 7) / 8), 256, 0, stream, a, rows_a, b, rows_b, F, wide, out);
  return launch_status();
}

int mingru_fwd(const float* z, const float* h_tilde, const NearKink& kink, long long ld, const float* x0, const float* a0,
               const uint8_t* done, float* states, uint8_t* forms, float* y, float* x_last, float* a_last, int B, int T, int D,
               cudaStream_t stream) {
  if (const int st = check_dims(B, T, D)) return st;
  const int segs = segments(B, D);
  mxk::launch_kernel(segs == 8 ? mingru_fwd_kernel<8> : mingru_fwd_kernel<16>, blocks_of(B, D), 32 * segs, 0, stream, z, h_tilde, kink.h, kink.in, kink.w,
                     kink.norms, kink.F, ld, x0, a0, done, states, forms, y, x_last, a_last, B, T, D, turn_length(B, T, D));
  return launch_status();
}

size_t mingru_forms(int B, int T, int D) { return static_cast<size_t>(blocks_of(B, D)) * ((T + turn_length(B, T, D) - 1) / turn_length(B, T, D)); }

int mingru_bwd(const float* z, const float* h_tilde, long long ld, const float* states, const uint8_t* forms, const float* x0, const uint8_t* done,
               const float* gx, const float* gy, const float* gx_last, float* gz, float* gh, float* gx0, int B, int T, int D,
               cudaStream_t stream) {
  if (const int st = check_dims(B, T, D)) return st;
  const int segs = segments(B, D);
  mxk::launch_kernel(segs == 8 ? mingru_bwd_kernel<8> : mingru_bwd_kernel<16>, blocks_of(B, D), 32 * segs, 0, stream, z, h_tilde, ld, states, forms, x0, done, gx,
                     gy, gx_last, gz, gh, gx0, B, T, D, turn_length(B, T, D));
  return launch_status();
}

int mingru_step(const float* in, const float* w_z, const float* w_h, const float* x0, const float* a0, const uint8_t* done,
                float* x, float* y, float* a_last, int B, int F, int D, cudaStream_t stream) {
  if (B <= 0 || F <= 0 || D <= 0) return MXK_ERR_DIMS;
  const long long tiles = static_cast<long long>((B + 7) / 8) * ((D + 1) / 2);
  mxk::launch_kernel(few_tiles(tiles) ? mingru_step_kernel<4> : mingru_step_kernel<1>, tile_blocks(tiles), 128, 0, stream, in, w_z, w_h, x0, a0, done,
                     x, y, a_last, B, F, D);
  return launch_status();
}

}  // namespace layers
}  // namespace mxk
