// The LRU layer's own kernels: a fused single time step (acting), and the gradients of its parameters from those of the
// real projection matrices.
#include <cuda_bf16.h>

#include <type_traits>

#include "layers.cuh"
#include "mxk_common.cuh"
#include "warp_tile.cuh"

namespace mxk {
namespace layers {
namespace {

// One time step of a few sequences is two matrix-vector-like products over weights that fit L2: launch latency and the
// depth of the memory pipeline are what counts, so every warp computes eight sequences x four outputs with its lanes
// across the contraction (the 12 loads of an iteration are independent), and nothing but the state makes a round trip
// through memory between the two launches.  (16 sequences, F = 128, N = 256: 25 launches, 250 us on the host -> 2.)
template <int kSplit>
__global__ void __launch_bounds__(128) lru_step_state_kernel(LruWeights w, const float* __restrict__ x,
                                                             const float* __restrict__ h0, const float* __restrict__ a0,
                                                             const uint8_t* __restrict__ done, float* __restrict__ h,
                                                             float* __restrict__ a_last, int B, int F, int N) {
  enter_kernel();
  const TilePlace<kSplit> at_tile;
  const int lane = at_tile.lane;
  const int units = (N + 1) / 2;
  const int n0 = (at_tile.tile % units) * 2, m0 = (at_tile.tile / units) * 8;
  if (m0 >= B) return;
  WarpTile acc;
  const float* rows[4] = {w.b_re + static_cast<size_t>(n0) * F, w.b_im + static_cast<size_t>(n0) * F,
                          w.b_re + static_cast<size_t>(min(n0 + 1, N - 1)) * F, w.b_im + static_cast<size_t>(min(n0 + 1, N - 1)) * F};
  acc.accumulate(x + static_cast<size_t>(m0) * F, F, min(8, B - m0), rows, F, at_tile.first, at_tile.step);
  float v = acc.reduce(lane);
  if (!join_warps<kSplit>(v, lane)) return;
  // this lane: sequence m, component j & 1 of unit n
  const int m = m0 + (lane >> 2), n = n0 + ((lane >> 1) & 1), im = lane & 1;
  if (m >= B || n >= N) return;
  const float bu = v * expf(w.gamma_log[n]);
  const float r = expf(-expf(w.nu_log[n]));
  float s, c;
  sincosf(expf(w.theta_log[n]), &s, &c);
  const float lre = r * c, lim = r * s;
  const bool reset = done && done[m] != 0;
  const size_t at = static_cast<size_t>(m) * N + n;
  const float2 hp = h0 ? reinterpret_cast<const float2*>(h0)[at] : make_float2(0.f, 0.f);
  // (the terms of a complex product in the recurrence kernels' order)
  float out = im ? fmaf(lre, hp.y, fmaf(lim, hp.x, bu)) : fmaf(lre, hp.x, fmaf(-lim, hp.y, bu));
  if (reset) out = bu;
  h[2 * at + im] = out;
  if (a_last) {
    const float2 ap = (a0 && !reset) ? reinterpret_cast<const float2*>(a0)[at] : make_float2(1.f, 0.f);
    a_last[2 * at + im] = im ? lre * ap.y + lim * ap.x : lre * ap.x - lim * ap.y;
  }
}

template <int kSplit>
__global__ void __launch_bounds__(128) lru_step_read_kernel(LruWeights w, const float* __restrict__ x,
                                                            const float* __restrict__ h, float* __restrict__ y, int B,
                                                            int F, int N) {
  enter_kernel();
  const TilePlace<kSplit> at_tile;
  const int lane = at_tile.lane;
  const int units = (F + 3) / 4;
  const int f0 = (at_tile.tile % units) * 4, m0 = (at_tile.tile / units) * 8;
  if (m0 >= B) return;
  const int mv = min(8, B - m0);
  WarpTile acc;
#pragma unroll 2
  for (int n = at_tile.first; n < N; n += at_tile.step) {
    float2 hv[8];
    float cr[4], ci[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const size_t row = static_cast<size_t>(min(f0 + j, F - 1)) * N + n;
      cr[j] = __ldg(w.c_re + row);
      ci[j] = __ldg(w.c_im + row);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
      hv[i] = reinterpret_cast<const float2*>(h)[static_cast<size_t>(m0 + min(i, mv - 1)) * N + n];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc.v[i * 4 + j] = fmaf(hv[i].x, cr[j], fmaf(-hv[i].y, ci[j], acc.v[i * 4 + j]));
  }
  float v = acc.reduce(lane);
  if (!join_warps<kSplit>(v, lane)) return;
  const int m = m0 + (lane >> 2), f = f0 + (lane & 3);
  if (m >= B || f >= F) return;
  const size_t at = static_cast<size_t>(m) * F + f;
  y[at] = fmaf(x[at], w.d[f], v);
}

constexpr int kSkipBlocks = 4 * kNumSMs;

// HBM-bound: one read of both operands; a block takes every gridDim.x-th group of rows, its threads the columns, kVec of them each.
// Four blocks an SM with four rows of both operands as 16-byte vectors under way per thread are 128 KiB, the last rows among them
// (65536 x 256: 25 us; eight rows of single elements and the remainder one by one: 42).
template <int kVec>
__global__ void __launch_bounds__(256) skip_grad_kernel(const float* __restrict__ gy, const float* __restrict__ x,
                                                        float* __restrict__ partial, long long rows, int F) {
  enter_kernel();
  constexpr int kRows = kVec == 4 ? 4 : 8;
  __shared__ float sums[256][kVec];
  const int vectors = F / kVec, width = min(vectors, 256);
  const int per = 256 / width;   // rows side by side in a block
  const int ro = threadIdx.x / width, ct = threadIdx.x % width;
  const auto load = [](const float* p, float* v) {
    if constexpr (kVec == 4) {
      const float4 u = ld_stream(reinterpret_cast<const float4*>(p));
      v[0] = u.x; v[1] = u.y; v[2] = u.z; v[3] = u.w;
    } else {
      v[0] = ld_stream(p);
    }
  };
  for (int c0 = 0; c0 < vectors; c0 += 256) {
    const int c = (c0 + ct) * kVec;
    float s[2][kVec] = {};
    if (ro < per && c0 + ct < vectors) {
      const long long step = static_cast<long long>(gridDim.x) * per;
      long long r = static_cast<long long>(blockIdx.x) * per + ro;
      const float *pg = gy + r * F + c, *px = x ? x + r * F + c : nullptr;
      for (; r < rows; r += kRows * step, pg += kRows * step * F) {
        float a[kRows][kVec], b[kRows][kVec];
#pragma unroll
        for (int u = 0; u < kRows; ++u) {
          const bool in = r + u * step < rows;
#pragma unroll
          for (int e = 0; e < kVec; ++e) {
            a[u][e] = 0.f;
            b[u][e] = 1.f;
          }
          if (in) load(pg + u * step * F, a[u]);
          if (in && px) load(px + u * step * F, b[u]);
        }
        if (px) px += kRows * step * F;
#pragma unroll
        for (int u = 0; u < kRows; ++u)
#pragma unroll
          for (int e = 0; e < kVec; ++e) s[u & 1][e] = fmaf(a[u][e], b[u][e], s[u & 1][e]);
      }
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < kVec; ++e) sums[threadIdx.x][e] = s[0][e] + s[1][e];
    __syncthreads();
    if (ro == 0 && c0 + ct < vectors) {
#pragma unroll
      for (int e = 0; e < kVec; ++e) {
        float v = 0.f;
        for (int i = 0; i < per; ++i) v += sums[i * width + ct][e];
        partial[static_cast<size_t>(blockIdx.x) * F + c + e] = v;
      }
    }
  }
}

// Blocks 0..N-1: hidden unit n (its rows of the input projection, and lambda); N..N+F-1: feature f (its row of the
// read-out and its skip weight).  Sums over splits run in a fixed order.
__global__ void __launch_bounds__(128) lru_param_grads_kernel(LruWeights w, LruGrads g, int F, int N) {
  enter_kernel();
  __shared__ float red[128];
  const int tid = threadIdx.x;
  const auto block_sum = [&](float v) {
    red[tid] = v;
    __syncthreads();
    for (int o = 64; o > 0; o >>= 1) {
      if (tid < o) red[tid] += red[tid + o];
      __syncthreads();
    }
    return red[0];
  };
  if (static_cast<int>(blockIdx.x) < N) {
    const int n = blockIdx.x;
    const float scale = expf(w.gamma_log[n]);
    const size_t plane = static_cast<size_t>(2) * N * F;
    float dot = 0.f;
    for (int f = tid; f < F; f += 128) {
      float re = 0.f, im = 0.f;
      const float* p = g.in_partial + static_cast<size_t>(2) * n * F + f;
#pragma unroll 6
      for (int s = 0; s < g.in_splits; ++s) { re += p[s * plane]; im += p[s * plane + F]; }
      re *= scale;
      im *= scale;
      const size_t at = static_cast<size_t>(n) * F + f;
      g.g_b_re[at] = re;
      g.g_b_im[at] = im;
      dot += re * w.b_re[at] + im * w.b_im[at];
    }
    dot = block_sum(dot);
    if (tid == 0) {
      g.g_gamma[n] = dot;
      // lambda = exp(-e^nu + i e^theta); with cotangent G (torch's convention): dL = Re(conj(G) dlambda)
      const float2 l = reinterpret_cast<const float2*>(g.lambda)[n], gl = reinterpret_cast<const float2*>(g.g_lambda)[n];
      g.g_nu[n] = -expf(w.nu_log[n]) * (gl.x * l.x + gl.y * l.y);
      g.g_theta[n] = expf(w.theta_log[n]) * (gl.y * l.x - gl.x * l.y);
    }
  } else {
    const int f = blockIdx.x - N;
    const size_t plane = static_cast<size_t>(2) * N * F;
    for (int n = tid; n < N; n += 128) {
      float re = 0.f, im = 0.f;
      const float2* p = reinterpret_cast<const float2*>(g.out_partial + static_cast<size_t>(f) * 2 * N) + n;
#pragma unroll 6
      for (int s = 0; s < g.out_splits; ++s) { const float2 v = p[s * (plane / 2)]; re += v.x; im += v.y; }
      const size_t at = static_cast<size_t>(f) * N + n;
      g.g_c_re[at] = re;
      g.g_c_im[at] = -im;
    }
    float s = 0.f;
    for (int b = tid; b < g.skip_blocks; b += 128) s += g.skip_partial[static_cast<size_t>(b) * F + f];
    s = block_sum(s);
    if (tid == 0) g.g_d[f] = s;
  }
}

// ------------------------------------------------------------------------------------------------ sensitivities
// Every leaf obeys S_t = done_t ? J_t : lambda S_{t-1} + J_t with local Jacobians that are never formed here:
//   nu, theta  J = -e^nu q, i e^theta q with q_t = lambda h_{t-1} (zero where step t resets)
//   gamma      J = B u: the recurrence of the states themselves from another start, S_T = h_T + P (S_0 - h_0)
//   B          J = gamma_n u_f and i gamma_n u_f: S_T = P S_0 + gamma_n W, W[n][f] = sum over t >= r of lambda_n^(T-1-t) u_t[f]
// with r the last reset of the segment and P = lambda^T without one, else 0.

__device__ __forceinline__ int last_reset(const uint8_t* drow, int T) {   // -1 without one; whole block
  __shared__ int found;
  if (threadIdx.x == 0) found = -1;
  __syncthreads();
  if (drow) {
    int r = -1;
    for (int t = threadIdx.x; t < T; t += blockDim.x)
      if (drow[t]) r = t;
    if (r >= 0) atomicMax(&found, r);
  }
  __syncthreads();
  return found;
}

// lambda^k of the float32 lambda, multiplied up in double
__device__ __forceinline__ float2 power(float2 l, int k) {
  double br = l.x, bi = l.y, r = 1.0, i = 0.0;
  for (; k > 0; k >>= 1) {
    if (k & 1) {
      const double t = r * br - i * bi;
      i = r * bi + i * br;
      r = t;
    }
    const double t = br * br - bi * bi;
    bi = 2.0 * br * bi;
    br = t;
  }
  return make_float2(static_cast<float>(r), static_cast<float>(i));
}
__device__ __forceinline__ float2 cmul(float2 a, float2 b) { return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ float2 cmul_add(float2 a, float2 b, float2 c) {
  return make_float2(fmaf(a.x, b.x, fmaf(-a.y, b.y, c.x)), fmaf(a.x, b.y, fmaf(a.y, b.x, c.y)));
}

// nu, theta, gamma of 32 units: with s0 the first step after the last reset (0 without one, and then the carried state is
// "step -1"), the sum over s >= s0 of lambda^(T-1-s) h_s is cut into eight stretches of time, one per warp, each by Horner's
// rule with eight states in flight (one thread per unit walking all of T was a chain of L2 round trips: 20 us at T = 64).
__device__ __forceinline__ void unit_sensitivities(const LruWeights& w, const float* __restrict__ lambda, const float* __restrict__ h,
                                                   const float* __restrict__ h0, const LruSensitivities& s, int b, int n0, int r,
                                                   int T, int N) {
  __shared__ float2 part[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = n0 + lane;
  const bool in = n < N;
  const size_t at = static_cast<size_t>(b) * N + (in ? n : 0);
  const float2 l = reinterpret_cast<const float2*>(lambda)[in ? n : 0];
  const float2* hs = reinterpret_cast<const float2*>(h) + static_cast<size_t>(b) * T * N + (in ? n : 0);
  const int s0 = max(r, 0), len = (T - 1 - s0 + 7) / 8;
  const int from = min(T - 1, s0 + warp * len), to = min(T - 1, from + len);
  float2 acc = make_float2(0.f, 0.f);
  constexpr int kDeep = 8;
  for (int t = from; t < to; t += kDeep) {
    float2 v[kDeep];
#pragma unroll
    for (int u = 0; u < kDeep; ++u)
      if (t + u < to) v[u] = __ldg(hs + static_cast<size_t>(t + u) * N);
#pragma unroll
    for (int u = 0; u < kDeep; ++u)
      if (t + u < to) acc = cmul(l, make_float2(acc.x + v[u].x, acc.y + v[u].y));
  }
  part[warp][lane] = cmul(power(l, T - 1 - to), acc);
  __syncthreads();
  if (warp > 0 || !in) return;
  // (what a reset cuts off does not enter, finite or not)
  const bool kept = r < 0;
  const float2 none = make_float2(0.f, 0.f);
  const float2 start = h0 && kept ? reinterpret_cast<const float2*>(h0)[at] : none;
  const float2 p = kept ? power(l, T) : none;
  acc = cmul(p, start);
#pragma unroll
  for (int i = 0; i < 8; ++i) { acc.x += part[i][lane].x; acc.y += part[i][lane].y; }
  const float en = expf(w.nu_log[n]), et = expf(w.theta_log[n]);
  const auto old = [&](const float* q) { return kept ? reinterpret_cast<const float2*>(q)[at] : none; };
  const float2 last = hs[static_cast<size_t>(T - 1) * N], g0 = old(s.gamma);
  reinterpret_cast<float2*>(s.nu_out)[at] = cmul_add(p, old(s.nu), make_float2(-en * acc.x, -en * acc.y));
  reinterpret_cast<float2*>(s.theta_out)[at] = cmul_add(p, old(s.theta), make_float2(-et * acc.y, et * acc.x));
  reinterpret_cast<float2*>(s.gamma_out)[at] = cmul_add(p, make_float2(g0.x - start.x, g0.y - start.y), last);
}

// B: a block owns one sequence, 256 / kLanes units and 4 kLanes features; kLanes lanes share a unit, four features each.
// The powers of lambda are made once per block, so a step costs one packed multiply-add per entry, and only the old and the
// new sensitivities touch memory: HBM-bound at large N F, else bound by the multiply-adds.  The blocks behind them take the
// other leaves.  (64 sequences x 64 steps, 64 features, 128 units: the materialised Jacobians took 490 us of kernels in 76
// launches.)
// kWide: sixteen-byte accesses to the sensitivities of B (known when compiled, the old ones' loads stay in front of the sums:
// 3 us of 44 for the whole segment).
constexpr int kSensSteps = 64;
template <int kLanes, bool kWide>
__global__ void __launch_bounds__(256) lru_sensitivities_kernel(LruWeights w, const float* __restrict__ lambda,
                                                                const float* __restrict__ h, const float* __restrict__ h0,
                                                                const float* __restrict__ u, const uint8_t* __restrict__ done,
                                                                LruSensitivities s, int T, int F, int N, int input_blocks) {
  enter_kernel();
  constexpr int kUnits = 256 / kLanes, kFeatures = 4 * kLanes;
  __shared__ __align__(16) float us[kSensSteps][kFeatures];
  __shared__ float2 pw[kUnits][kSensSteps + 1];
  const int b = blockIdx.y;
  const uint8_t* drow = done ? done + static_cast<size_t>(b) * T : nullptr;
  if (static_cast<int>(blockIdx.x) >= input_blocks) {
    unit_sensitivities(w, lambda, h, h0, s, b, (blockIdx.x - input_blocks) * 32, last_reset(drow, T), T, N);
    return;
  }
  const int unit_groups = (N + kUnits - 1) / kUnits;
  const int n0 = (blockIdx.x % unit_groups) * kUnits, f0 = (blockIdx.x / unit_groups) * kFeatures;
  const int un = threadIdx.x / kLanes, lf = threadIdx.x % kLanes;
  const int n = n0 + un, f = f0 + lf * 4;
  const bool in = n < N && f < F;
  const size_t at = (static_cast<size_t>(b) * N + (in ? n : 0)) * F + (in ? f : 0);
  float4 ore[2] = {}, oim[2] = {};   // old sensitivities, on their way while the sums are formed
  if (kWide && in) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      ore[e] = ld_stream(reinterpret_cast<const float4*>(s.b_re + 2 * at) + e);
      oim[e] = ld_stream(reinterpret_cast<const float4*>(s.b_im + 2 * at) + e);
    }
  }
  const int r = last_reset(drow, T);
  const int first = max(r, 0);
  for (int i = threadIdx.x; i < kUnits * (kSensSteps + 1); i += 256) {
    const int ui = i / (kSensSteps + 1), k = i % (kSensSteps + 1);
    if (n0 + ui < N) pw[ui][k] = power(reinterpret_cast<const float2*>(lambda)[n0 + ui], k);
  }
  float2 acc[4] = {};
  const float* ub = u + static_cast<size_t>(b) * T * F;
  for (int t0 = first; t0 < T; t0 += kSensSteps) {
    const int len = min(kSensSteps, T - t0);
    __syncthreads();
    for (int i = threadIdx.x; i < len * kFeatures; i += 256) {
      const int t = i / kFeatures, c = i % kFeatures;
      us[t][c] = f0 + c < F ? __ldg(ub + static_cast<size_t>(t0 + t) * F + f0 + c) : 0.f;
    }
    __syncthreads();
    const float2 shift = pw[un][len];   // what earlier steps have decayed by at the end of this stretch
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[e] = cmul(shift, acc[e]);
#pragma unroll 8
    for (int t = 0; t < len; ++t) {
      const float4 x = *reinterpret_cast<const float4*>(&us[t][lf * 4]);
      const float2 p = pw[un][len - 1 - t];
      acc[0] = __ffma2_rn(p, make_float2(x.x, x.x), acc[0]);
      acc[1] = __ffma2_rn(p, make_float2(x.y, x.y), acc[1]);
      acc[2] = __ffma2_rn(p, make_float2(x.z, x.z), acc[2]);
      acc[3] = __ffma2_rn(p, make_float2(x.w, x.w), acc[3]);
    }
  }
  if (!in) return;
  const float gamma = expf(w.gamma_log[n]);
  const float2 p = r < 0 ? power(reinterpret_cast<const float2*>(lambda)[n], T) : make_float2(0.f, 0.f);
  const auto add_old = [&](float2 o, float2 v) { return r < 0 ? cmul_add(p, o, v) : v; };
  const auto re = [&](float2 o, int e) { return add_old(o, make_float2(gamma * acc[e].x, gamma * acc[e].y)); };
  const auto im = [&](float2 o, int e) { return add_old(o, make_float2(-gamma * acc[e].y, gamma * acc[e].x)); };
  if (kWide) {   // two complex entries each
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float2 v0 = re({ore[e].x, ore[e].y}, 2 * e), v1 = re({ore[e].z, ore[e].w}, 2 * e + 1);
      const float2 y0 = im({oim[e].x, oim[e].y}, 2 * e), y1 = im({oim[e].z, oim[e].w}, 2 * e + 1);
      reinterpret_cast<float4*>(s.b_re_out + 2 * at)[e] = make_float4(v0.x, v0.y, v1.x, v1.y);
      reinterpret_cast<float4*>(s.b_im_out + 2 * at)[e] = make_float4(y0.x, y0.y, y1.x, y1.y);
    }
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (f + e >= F) break;
      reinterpret_cast<float2*>(s.b_re_out)[at + e] = re(reinterpret_cast<const float2*>(s.b_re)[at + e], e);
      reinterpret_cast<float2*>(s.b_im_out)[at + e] = im(reinterpret_cast<const float2*>(s.b_im)[at + e], e);
    }
  }
}

struct ColumnSums {
  ColumnSum job[4];
  int first_block[5];
};
// 32 columns per block; 32 groups of rows (few rows per thread: latency-bound), added in order
__global__ void __launch_bounds__(1024) column_sums_kernel(const __grid_constant__ ColumnSums p) {
  enter_kernel();
  __shared__ float part[32][33];
  int j = 0;
  while (static_cast<int>(blockIdx.x) >= p.first_block[j + 1]) ++j;
  const ColumnSum& jb = p.job[j];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int col = (blockIdx.x - p.first_block[j]) * 32 + tx;
  float s = 0.f;
  if (col < jb.cols)
#pragma unroll 4
    for (int r = ty; r < jb.rows; r += 32) s += jb.src[static_cast<size_t>(r) * jb.cols + col];
  part[ty][tx] = s;
  __syncthreads();
  if (ty == 0 && col < jb.cols) {
    float t = part[0][tx];
#pragma unroll
    for (int i = 1; i < 32; ++i) t += part[i][tx];
    if (jb.dst16) static_cast<__nv_bfloat16*>(jb.dst16)[col] = __float2bfloat16(t);
    else jb.dst[col] = t;
  }
}

}  // namespace

int column_sums(const ColumnSum* jobs, int count, cudaStream_t stream) {
  if (count < 1 || count > 4) return MXK_ERR_DIMS;
  ColumnSums p{};
  for (int j = 0; j < count; ++j) {
    p.job[j] = jobs[j];
    p.first_block[j + 1] = p.first_block[j] + (jobs[j].cols + 31) / 32;
  }
  for (int j = count; j < 4; ++j) p.first_block[j + 1] = 0x7fffffff;
  mxk::launch_kernel(column_sums_kernel, p.first_block[count], 1024, 0, stream, p);
  return launch_status();
}

int lru_step(const LruWeights& w, const float* x, const float* h0, const float* a0, const uint8_t* done, float* h,
             float* a_last, float* y, int B, int F, int N, cudaStream_t stream) {
  if (B <= 0 || F <= 0 || N <= 0) return MXK_ERR_DIMS;
  const long long groups = (B + 7) / 8;
  const long long tiles_h = groups * ((N + 1) / 2), tiles_y = groups * ((F + 3) / 4);
  const auto state = few_tiles(tiles_h) ? lru_step_state_kernel<4> : lru_step_state_kernel<1>;
  const auto read = few_tiles(tiles_y) ? lru_step_read_kernel<4> : lru_step_read_kernel<1>;
  mxk::launch_kernel(state, tile_blocks(tiles_h), 128, 0, stream, w, x, h0, a0, done, h, a_last, B, F, N);
  mxk::launch_kernel(read, tile_blocks(tiles_y), 128, 0, stream, w, x, h, y, B, F, N);
  return launch_status();
}

int skip_grad_blocks(long long rows) { return static_cast<int>(rows < kSkipBlocks ? rows : kSkipBlocks); }

int skip_grad(const float* gy, const float* x, float* partial, long long rows, int F, cudaStream_t stream) {
  const bool vectors = F % 4 == 0 && aligned16(gy) && (!x || aligned16(x));
  mxk::launch_kernel(vectors ? skip_grad_kernel<4> : skip_grad_kernel<1>, skip_grad_blocks(rows), 256, 0, stream, gy, x, partial, rows, F);
  return launch_status();
}

int lru_param_grads(const LruWeights& w, const LruGrads& g, int F, int N, cudaStream_t stream) {
  mxk::launch_kernel(lru_param_grads_kernel, N + F, 128, 0, stream, w, g, F, N);
  return launch_status();
}

int lru_sensitivities(const LruWeights& w, const float* lambda, const float* h, const float* h0, const float* u,
                      const uint8_t* done, const LruSensitivities& s, int B, int T, int F, int N, cudaStream_t stream) {
  if (B <= 0 || T <= 0 || F <= 0 || N <= 0 || B > 65535) return MXK_ERR_DIMS;
  // whole vectors per unit, from where they may start
  bool wide = F % 4 == 0;
  for (const float* p : {s.b_re, s.b_im, static_cast<const float*>(s.b_re_out), static_cast<const float*>(s.b_im_out)}) wide = wide && aligned16(p);
  // lanes per unit: as many as four features each need, so that narrow inputs leave none idle
  const auto go = [&](auto lanes_c) {
    constexpr int lanes = decltype(lanes_c)::value, units = 256 / lanes;
    const int inputs = ((N + units - 1) / units) * ((F + 4 * lanes - 1) / (4 * lanes));
    mxk::launch_kernel(wide ? lru_sensitivities_kernel<lanes, true> : lru_sensitivities_kernel<lanes, false>, dim3(inputs + (N + 31) / 32, B), 256, 0,
                       stream, w, lambda, h, h0, u, done, s, T, F, N, inputs);
    return launch_status();
  };
  if (F <= 32) return go(std::integral_constant<int, 8>{});
  if (F <= 64) return go(std::integral_constant<int, 16>{});
  return go(std::integral_constant<int, 32>{});
}

}  // namespace layers
}  // namespace mxk
