// The elementwise work around the mLSTM layer's products and chunk kernels (mlstm.py:129-229), bf16 in and out, float32
// arithmetic: causal convolution + SiLU, gates and key scaling, head-wise LayerNorm + skip + output gate, and their
// gradients.  Bound by HBM, one read and one write of each operand; a thread owns eight or four channels and walks
// tokens, so that the convolution's window and the parameter gradients stay in registers.  (As separate torch calls they
// were about sixty launches of a layer step.)
#include <cuda_bf16.h>

#include <algorithm>

#include "layers.cuh"
#include "mxk_common.cuh"
#include "umma.cuh"

namespace mxk {
namespace layers {
namespace {

using umma::pack8_bf16;
using umma::pack_bf16;
using umma::unpack8_bf16;
using bf16 = __nv_bfloat16;

constexpr int kTaps = 4;

__device__ __forceinline__ float sigmoid(float x) { return 1.f / (1.f + __expf(-x)); }
__device__ __forceinline__ float softplus(float x) { return x > 20.f ? x : log1pf(__expf(x)); }
// a value that the bf16 layer holds in memory
__device__ __forceinline__ float held(float x) { return __bfloat162float(__float2bfloat16(x)); }
// The same for two and for eight: a conversion of a pair costs what one of a single value does, and the gate has eight to an element.
__device__ __forceinline__ float2 held(float2 x) {
  const uint32_t p = pack_bf16(x.x, x.y);
  return make_float2(__uint_as_float(p << 16), __uint_as_float(p & 0xffff0000u));
}
__device__ __forceinline__ void hold8(float* x) { unpack8_bf16(pack8_bf16(x), x); }
__device__ __forceinline__ void load8(const bf16* p, float* x) { unpack8_bf16(*reinterpret_cast<const uint4*>(p), x); }
__device__ __forceinline__ void unpack4(uint2 v, float2* x) {
  x[0] = make_float2(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u));
  x[1] = make_float2(__uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
}
__device__ __forceinline__ void store8(bf16* p, const float* x) { *reinterpret_cast<uint4*>(p) = pack8_bf16(x); }

// The taps of four channels, in pairs.
struct Taps {
  float2 w[kTaps][2], b[2];
  __device__ __forceinline__ Taps(const bf16* conv_w, const bf16* conv_b, int c) {
    float raw[4 * kTaps];
    load8(conv_w + c * kTaps, raw);
    load8(conv_w + c * kTaps + 8, raw + 8);
#pragma unroll
    for (int k = 0; k < kTaps; ++k) {
      w[k][0] = make_float2(raw[k], raw[kTaps + k]);
      w[k][1] = make_float2(raw[2 * kTaps + k], raw[3 * kTaps + k]);
    }
    unpack4(*reinterpret_cast<const uint2*>(conv_b + c), b);
  }
};

// A thread walks a run of four channels; inputs are a ring of four steps, the loop's unrolling, loads as far ahead.  65536 x 512:
// 49 us (eight channels and moved windows 68); bound by instructions, the sigmoids' divisions among them (HBM 21).
template <int kRun>   // tokens per thread
__global__ void __launch_bounds__(256) conv_fwd_kernel(const bf16* __restrict__ up, long long ld, const bf16* __restrict__ conv_w,
                                                       const bf16* __restrict__ conv_b, bf16* __restrict__ u, int B, int T, int hid,
                                                       int runs) {
  enter_kernel();
  const int groups = hid / 4;
  const long long id = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x;
  const int c = static_cast<int>(id % groups) * 4;
  const long long seq_run = id / groups;
  if (seq_run >= static_cast<long long>(B) * runs) return;
  const int b = static_cast<int>(seq_run / runs), t0 = static_cast<int>(seq_run % runs) * kRun;
  const long long tok0 = static_cast<long long>(b) * T + t0;
  const bf16* const src = up + tok0 * ld + c;
  bf16* const dst = u + tok0 * hid + c;
  const auto at = [](const bf16* from) { return *reinterpret_cast<const uint2*>(from); };
  uint2 next[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (t0 + i < T) next[i] = at(src + i * ld);
  float2 win[kTaps][2];   // step t0 + i in slot i & 3
#pragma unroll
  for (int i = 1; i < 4; ++i) {
    win[i][0] = win[i][1] = make_float2(0.f, 0.f);
    if (t0 + i - 4 >= 0) unpack4(at(src + (i - 4) * ld), win[i]);
  }
  const Taps taps(conv_w, conv_b, c);
#pragma unroll 1
  for (int i0 = 0; i0 < kRun; i0 += 4)
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int i = i0 + s;
      if (t0 + i >= T) break;
      unpack4(next[s], win[s]);
      if (i + 4 < kRun && t0 + i + 4 < T) next[s] = at(src + (i + 4) * ld);
      float2 v[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float2 a = taps.b[h];
#pragma unroll
        for (int k = 0; k < kTaps; ++k) a = __ffma2_rn(taps.w[k][h], win[(s + 1 + k) & 3][h], a);
        a = held(a);
        v[h] = make_float2(a.x * sigmoid(a.x), a.y * sigmoid(a.y));
      }
      *reinterpret_cast<uint2*>(dst + i * hid) = make_uint2(pack_bf16(v[0].x, v[0].y), pack_bf16(v[1].x, v[1].y));
    }
}

// A thread walks runs of four channels, and the three steps after each: the convolution's output is recomputed, its cotangent
// g_t = gu_t silu'(.) meets the four inputs it came from.  Inputs and their cotangents are rings of four steps, the loop's unrolling.
// Bound: the instructions of an element (about 25, in pairs), at two blocks an SM beside HBM (8 bytes an element).  65536 x 512: 145 us;
// eight channels a thread, one block of 223 registers an SM, windows moved along by copies and loads two steps ahead: 257.  6016 x 256: 14.5 (31.5).
template <int kRun>
__global__ void __launch_bounds__(256, 2) conv_bwd_kernel(const bf16* __restrict__ up, long long ld, const bf16* __restrict__ conv_w,
                                                          const bf16* __restrict__ conv_b, const bf16* __restrict__ gu,
                                                          const bf16* __restrict__ gx, bf16* __restrict__ gup,
                                                          float* __restrict__ partial, int B, int T, int hid, int runs, int lanes) {
  enter_kernel();
  extern __shared__ float red[];   // [channel][taps + bias] sums of the block's runs, one run group at a time
  // a block: `lanes` groups of four channels (a divisor of both 256 and of all of them) x 256 / lanes runs
  const int l = threadIdx.x % lanes, rg = threadIdx.x / lanes, c = (blockIdx.y * lanes + l) * 4;
  const Taps taps(conv_w, conv_b, c);
  float2 gw[kTaps][2], gb[2];
  const float2 zero = make_float2(0.f, 0.f);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    gb[h] = zero;
#pragma unroll
    for (int k = 0; k < kTaps; ++k) gw[k][h] = zero;
  }
  const long long all = static_cast<long long>(B) * runs;
  for (long long run = static_cast<long long>(blockIdx.x) * (256 / lanes) + rg; run < all; run += static_cast<long long>(gridDim.x) * (256 / lanes)) {
    const int b = static_cast<int>(run / runs), t0 = static_cast<int>(run % runs) * kRun;
    const long long tok0 = static_cast<long long>(b) * T + t0;
    const bf16* const pu = up + tok0 * ld + c;
    const bf16* const pg = gu + tok0 * hid + c;
    const bf16* const px = gx + tok0 * hid + c;
    bf16* const po = gup + tok0 * ld + c;
    const auto at = [](const bf16* from) { return *reinterpret_cast<const uint2*>(from); };
    uint2 nu[4], ng[4], nx[4];   // four steps, already on their way
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (t0 + i < T) {
        nu[i] = at(pu + i * ld);
        ng[i] = at(pg + i * hid);
        nx[i] = at(px + i * hid);
      }
    float2 win[4][2], acc[4][2];   // step t0 + i in slot i & 3
#pragma unroll
    for (int i = 1; i < 4; ++i) {
      win[i][0] = win[i][1] = zero;
      if (t0 + i - 4 >= 0) unpack4(at(pu + (i - 4) * ld), win[i]);
      acc[i][0] = acc[i][1] = zero;
    }
#pragma unroll 1
    for (int i0 = 0; i0 < kRun + 4; i0 += 4) {
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const int i = i0 + s, t = t0 + i;
        const uint2 x_done = nx[(s + 1) & 3];   // of step t - 3
        acc[s][0] = acc[s][1] = zero;
        if (t < T && i < kRun + kTaps - 1) {
          const bool own = i < kRun;
          float2 g[2];
          unpack4(nu[s], win[s]);
          unpack4(ng[s], g);
          if (t + 4 < T && i + 4 < kRun + kTaps - 1) {
            nu[s] = at(pu + (i + 4) * ld);
            ng[s] = at(pg + (i + 4) * hid);
          }
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float2 a = taps.b[h];
#pragma unroll
            for (int k = 0; k < kTaps; ++k) a = __ffma2_rn(taps.w[k][h], win[(s + 1 + k) & 3][h], a);
            a = held(a);
            const float sx = sigmoid(a.x), sy = sigmoid(a.y);
            g[h].x *= sx * (1.f + a.x * (1.f - sx));
            g[h].y *= sy * (1.f + a.y * (1.f - sy));
#pragma unroll
            for (int k = 0; k < kTaps; ++k) acc[(s + 1 + k) & 3][h] = __ffma2_rn(taps.w[k][h], g[h], acc[(s + 1 + k) & 3][h]);
            if (own) {
              gb[h].x += g[h].x;
              gb[h].y += g[h].y;
#pragma unroll
              for (int k = 0; k < kTaps; ++k) gw[k][h] = __ffma2_rn(g[h], win[(s + 1 + k) & 3][h], gw[k][h]);
            }
          }
        }
        // input t - 3 has met every output it reaches
        const int done = i - (kTaps - 1);
        if (done >= 0 && done < kRun && t0 + done < T) {
          float2 x[2];
          unpack4(x_done, x);
          if (done + 4 < kRun && t0 + done + 4 < T) nx[(s + 1) & 3] = at(px + (done + 4) * hid);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            x[h].x += acc[(s + 1) & 3][h].x;
            x[h].y += acc[(s + 1) & 3][h].y;
          }
          *reinterpret_cast<uint2*>(po + done * ld) = make_uint2(pack_bf16(x[0].x, x[0].y), pack_bf16(x[1].x, x[1].y));
        }
      }
    }
  }
  // block sums, run groups added in order
  for (int r = 0; r < 256 / lanes; ++r) {
    __syncthreads();
    if (rg == r) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float* const row = red + (l * 4 + e) * (kTaps + 1);
#pragma unroll
        for (int k = 0; k < kTaps; ++k) row[k] = (r ? row[k] : 0.f) + (e & 1 ? gw[k][e >> 1].y : gw[k][e >> 1].x);
        row[kTaps] = (r ? row[kTaps] : 0.f) + (e & 1 ? gb[e >> 1].y : gb[e >> 1].x);
      }
    }
  }
  __syncthreads();
  float* const out = partial + static_cast<size_t>(blockIdx.x) * hid * (kTaps + 1);
  for (int i = threadIdx.x; i < lanes * 4 * (kTaps + 1); i += 256) {
    const int ch = blockIdx.y * lanes * 4 + i / (kTaps + 1), k = i % (kTaps + 1);
    out[k < kTaps ? ch * kTaps + k : hid * kTaps + ch] = red[i];
  }
}

__global__ void __launch_bounds__(256) weights_kernel(const uint4* __restrict__ q, const uint4* __restrict__ k, const uint4* __restrict__ i_w,
                                                      const uint4* __restrict__ f_w, const bf16* __restrict__ i_b,
                                                      const bf16* __restrict__ f_b, uint4* __restrict__ qk_w, uint4* __restrict__ gate_w,
                                                      bf16* __restrict__ gate_b, int H, int head8, int gate8) {
  enter_kernel();
  const int heads = H * head8;
  int i = blockIdx.x * 256 + threadIdx.x;
  if (i < 2 * H) gate_b[i] = i < H ? i_b[i] : f_b[i - H];
  if (i < 2 * heads) {
    const bool is_k = i >= heads;
    if (is_k) i -= heads;
    qk_w[(2 * (i / head8) + is_k) * head8 + i % head8] = (is_k ? k : q)[i];
  } else if (i - 2 * heads < 2 * gate8) {
    i -= 2 * heads;
    gate_w[i] = i < gate8 ? i_w[i] : f_w[i - gate8];
  }
}

__global__ void __launch_bounds__(256) gates_fwd_kernel(const bf16* __restrict__ logits, const bf16* __restrict__ k, long long ld,
                                                        float scale, float* __restrict__ log_i, float* __restrict__ log_f,
                                                        bf16* __restrict__ ks, long long tokens, int H, int hid8, int hp, unsigned vec_blocks) {
  enter_kernel();
  if (blockIdx.x < vec_blocks) {
    const long long i = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x;
    const long long tok = i / hid8;
    const int c = static_cast<int>(i % hid8) * 8;
    if (tok >= tokens) return;
    const int d = hid8 * 8 / H;
    float x[8];
    load8(k + tok * ld + c / d * hp + c % d, x);
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] *= scale;
    store8(ks + tok * hid8 * 8 + c, x);
    return;
  }
  const long long i = static_cast<long long>(blockIdx.x - vec_blocks) * 256 + threadIdx.x;
  if (i >= tokens * H) return;
  const long long tok = i / H;
  const int h = static_cast<int>(i % H);
  log_i[i] = __bfloat162float(logits[tok * 2 * H + h]);
  log_f[i] = -held(softplus(-__bfloat162float(logits[tok * 2 * H + H + h])));
}

constexpr int kGateBlocks = 2 * kNumSMs;

__global__ void __launch_bounds__(256) gates_bwd_kernel(const bf16* __restrict__ logits, const float* __restrict__ glog_i,
                                                        const float* __restrict__ glog_f,
                                                        const bf16* __restrict__ gks, float scale, bf16* __restrict__ gk, long long ld,
                                                        bf16* __restrict__ glogits, float* __restrict__ partial, long long tokens,
                                                        int H, int hid8, int hp, unsigned vec_blocks) {
  enter_kernel();
  __shared__ float red[256];
  if (blockIdx.x < vec_blocks) {
    const long long i = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x;
    const long long tok = i / hid8;
    const int c = static_cast<int>(i % hid8) * 8;
    if (tok >= tokens) return;
    float x[8];
    load8(gks + tok * hid8 * 8 + c, x);
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] *= scale;
    const int d = hid8 * 8 / H;
    store8(gk + tok * ld + c / d * hp + c % d, x);
    return;
  }
  const int cols = 2 * H, per = 256 / cols;
  const int c = threadIdx.x % cols, ro = threadIdx.x / cols;
  const unsigned blocks = gridDim.x - vec_blocks, blk = blockIdx.x - vec_blocks;
  float sum = 0.f;
  if (ro < per)
    for (long long tok = static_cast<long long>(blk) * per + ro; tok < tokens; tok += static_cast<long long>(blocks) * per) {
      float v;
      if (c < H) v = held(glog_i[tok * H + c]);
      else v = held(held(glog_f[tok * H + c - H]) * sigmoid(-__bfloat162float(logits[tok * cols + c])));
      glogits[tok * cols + c] = __float2bfloat16(v);
      sum += v;
    }
  red[threadIdx.x] = sum;
  __syncthreads();
  if (threadIdx.x < cols) {
    float v = 0.f;
    for (int i = 0; i < per; ++i) v += red[i * cols + threadIdx.x];
    partial[blk * cols + threadIdx.x] = v;
  }
}

// Statistics of a head vector held by d / 8 neighbouring lanes (a power of two, or the loop below takes shared turns).
template <int LPH>
__device__ __forceinline__ float head_sum(float v) {
#pragma unroll
  for (int o = 1; o < LPH; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Bound by instructions: about eight roundings to bf16 and a sigmoid an element (HBM 42 us at 65536 x 512).  77 us with all loads before
// the sums and roundings in pairs; 96 with u's and z's after them and single roundings.
template <int LPH>
__global__ void __launch_bounds__(256) out_fwd_kernel(const bf16* __restrict__ h, const bf16* __restrict__ u, const bf16* __restrict__ z,
                                                      long long ld, const bf16* __restrict__ norm_w, const bf16* __restrict__ skip,
                                                      bf16* __restrict__ g, long long tokens, int hid8) {
  enter_kernel();
  const long long i = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x;
  const long long tok = i / hid8;
  const int c = static_cast<int>(i % hid8) * 8;
  const bool in = tok < tokens;
  uint4 raw[5] = {};   // all on their way before the sums of a head
  if (in) {
    raw[0] = *reinterpret_cast<const uint4*>(h + tok * hid8 * 8 + c);
    raw[1] = *reinterpret_cast<const uint4*>(u + tok * hid8 * 8 + c);
    raw[2] = *reinterpret_cast<const uint4*>(z + tok * ld + c);
    raw[3] = *reinterpret_cast<const uint4*>(norm_w + c);
    raw[4] = *reinterpret_cast<const uint4*>(skip + c);
  }
  float x[8];
  unpack8_bf16(raw[0], x);
  float s = 0.f, q = 0.f;
#pragma unroll
  for (int e = 0; e < 8; ++e) s += x[e];
  const float mean = head_sum<LPH>(s) * (1.f / (8 * LPH));
#pragma unroll
  for (int e = 0; e < 8; ++e) q = fmaf(x[e] - mean, x[e] - mean, q);
  const float rstd = rsqrtf(head_sum<LPH>(q) * (1.f / (8 * LPH)) + 1e-5f);
  if (!in) return;
  float w[8], sk[8], uu[8], zz[8];
  unpack8_bf16(raw[1], uu);
  unpack8_bf16(raw[2], zz);
  unpack8_bf16(raw[3], w);
  unpack8_bf16(raw[4], sk);
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    x[e] = (x[e] - mean) * rstd;
    w[e] += 1.f;
    uu[e] *= sk[e];
    zz[e] *= sigmoid(zz[e]);
  }
  hold8(x);
  hold8(w);
  hold8(uu);
  hold8(zz);
#pragma unroll
  for (int e = 0; e < 8; ++e) x[e] *= w[e];
  hold8(x);
#pragma unroll
  for (int e = 0; e < 8; ++e) x[e] += uu[e];
  hold8(x);
#pragma unroll
  for (int e = 0; e < 8; ++e) x[e] *= zz[e];
  store8(g + tok * hid8 * 8 + c, x);
}

// A thread keeps its eight channels over all its tokens (256 / hid8 tokens side by side in a block), the next one's rows on their
// way.  65536 x 512: 104 us (HBM 73); 150 with loads where they are used and single roundings.
template <int LPH>
__global__ void __launch_bounds__(256, 2) out_bwd_kernel(const bf16* __restrict__ gg, const bf16* __restrict__ h, const bf16* __restrict__ u,
                                                      const bf16* __restrict__ z, long long ld, const bf16* __restrict__ norm_w,
                                                      const bf16* __restrict__ skip, bf16* __restrict__ gh, bf16* __restrict__ gz,
                                                      long long ld_gz, bf16* __restrict__ gu, float* __restrict__ partial,
                                                      long long tokens, int hid8) {
  enter_kernel();
  __shared__ float red[256 * 16];
  const int per = 256 / hid8;
  const int c = (threadIdx.x % hid8) * 8, ro = threadIdx.x / hid8;
  float w[8], sk[8], gw[8], gs[8];
  load8(norm_w + c, w);
  load8(skip + c, sk);
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    gw[e] = gs[e] = 0.f;
    w[e] += 1.f;
  }
  hold8(w);
  const long long step = static_cast<long long>(gridDim.x) * per;
  uint4 raw[4];
  const auto fetch = [&](long long tok) {
    const bool in = tok < tokens;
    const uint4 none = make_uint4(0, 0, 0, 0);
    raw[0] = in ? *reinterpret_cast<const uint4*>(h + tok * hid8 * 8 + c) : none;
    raw[1] = in ? *reinterpret_cast<const uint4*>(gg + tok * hid8 * 8 + c) : none;
    raw[2] = in ? *reinterpret_cast<const uint4*>(u + tok * hid8 * 8 + c) : none;
    raw[3] = in ? *reinterpret_cast<const uint4*>(z + tok * ld + c) : none;
  };
  fetch(static_cast<long long>(blockIdx.x) * per + ro);
  for (long long t0 = static_cast<long long>(blockIdx.x) * per; t0 < tokens; t0 += step) {   // all lanes stay for the shuffles
    const long long tok = t0 + ro;
    const bool in = tok < tokens;
    float x[8], g[8], uu[8], zz[8];
    unpack8_bf16(raw[0], x);
    unpack8_bf16(raw[1], g);
    unpack8_bf16(raw[2], uu);
    unpack8_bf16(raw[3], zz);
    fetch(tok + step);
    float s = 0.f, q = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) s += x[e];
    const float mean = head_sum<LPH>(s) * (1.f / (8 * LPH));
#pragma unroll
    for (int e = 0; e < 8; ++e) q = fmaf(x[e] - mean, x[e] - mean, q);
    const float rstd = rsqrtf(head_sum<LPH>(q) * (1.f / (8 * LPH)) + 1e-5f);
    float s1 = 0.f, s2 = 0.f;
    // in the order of the layer: normed, scaled, skip and sum before the output gate; then their cotangents
    float n[8], y[8], t[8], sg[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) n[e] = x[e] = (x[e] - mean) * rstd;
    hold8(n);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      y[e] = n[e] * w[e];
      t[e] = sk[e] * uu[e];
    }
    hold8(y);
    hold8(t);
#pragma unroll
    for (int e = 0; e < 8; ++e) y[e] += t[e];
    hold8(y);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      sg[e] = sigmoid(zz[e]);
      t[e] = zz[e] * sg[e];
      y[e] *= g[e];
    }
    hold8(t);
    hold8(y);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      zz[e] = y[e] * sg[e] * (1.f + zz[e] * (1.f - sg[e]));
      g[e] *= t[e];
    }
    hold8(g);   // cotangent of the sum
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      n[e] *= g[e];
      t[e] = g[e] * uu[e];
      uu[e] = g[e] * sk[e];
      g[e] *= w[e];
    }
    hold8(n);
    hold8(t);
    hold8(g);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      gw[e] += n[e];
      gs[e] += t[e];
      s1 += g[e];
      s2 = fmaf(g[e], x[e], s2);
    }
    s1 = head_sum<LPH>(s1) * (1.f / (8 * LPH));
    s2 = head_sum<LPH>(s2) * (1.f / (8 * LPH));
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] = rstd * (g[e] - s1 - x[e] * s2);
    if (in) {
      store8(gh + tok * hid8 * 8 + c, x);
      store8(gz + tok * ld_gz + c, zz);
      store8(gu + tok * hid8 * 8 + c, uu);
    }
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    red[threadIdx.x * 16 + e] = gw[e];
    red[threadIdx.x * 16 + 8 + e] = gs[e];
  }
  __syncthreads();
  const int hid = hid8 * 8;
  for (int i = threadIdx.x; i < 2 * hid; i += 256) {
    const int ch = i % hid, at = (ch / 8) * 16 + (i < hid ? 0 : 8) + ch % 8;
    float v = 0.f;
    for (int r = 0; r < per; ++r) v += red[r * hid8 * 16 + at];
    partial[static_cast<size_t>(blockIdx.x) * 2 * hid + i] = v;
  }
}

// Tokens per thread of the convolution: sixteen reuse the window best; four where the machine would not be full (a thread
// walks them one after the other)
int run_of(int B, int T, int hid) { return static_cast<long long>(B) * T * (hid / 8) >= 16LL * 512 * kNumSMs ? 16 : 4; }
int runs_of(int T, int run) { return (T + run - 1) / run; }
// groups of four channels side by side in a block of the convolution's backward pass: 32 or what divides
int conv_lanes(int hid) {
  int l = 32;
  while ((hid / 4) % l) l /= 2;
  return l;
}

}  // namespace

int mlstm_conv_fwd(const void* up, long long ld, const void* conv_w, const void* conv_b, void* u, int B, int T, int hid,
                   cudaStream_t stream) {
  const int run = run_of(B, T, hid), runs = runs_of(T, run);
  const long long threads = static_cast<long long>(B) * runs * (hid / 4);
  const auto go = [&](auto kernel) {
    mxk::launch_kernel(kernel, static_cast<unsigned>((threads + 255) / 256), 256, 0, stream, static_cast<const bf16*>(up), ld, static_cast<const bf16*>(conv_w), static_cast<const bf16*>(conv_b), static_cast<bf16*>(u), B, T, hid, runs);
    return launch_status();
  };
  return run == 16 ? go(conv_fwd_kernel<16>) : go(conv_fwd_kernel<4>);
}

// of runs; a wave at most, since every one leaves a row of sums
int mlstm_conv_blocks(int B, int T, int hid) {
  const int lanes = conv_lanes(hid), per = 256 / lanes, most = std::max(1, 2 * kNumSMs / (hid / 4 / lanes));
  return static_cast<int>(std::min<long long>(most, (static_cast<long long>(B) * runs_of(T, run_of(B, T, hid)) + per - 1) / per));
}

int mlstm_conv_bwd(const void* up, long long ld, const void* conv_w, const void* conv_b, const void* gu, const void* gx, void* gup,
                   float* partial, int B, int T, int hid, cudaStream_t stream) {
  const int lanes = conv_lanes(hid), bytes = lanes * 4 * (kTaps + 1) * static_cast<int>(sizeof(float));
  const int run = run_of(B, T, hid), runs = runs_of(T, run);
  const auto go = [&](auto kernel) {
    mxk::launch_kernel(kernel, dim3(mlstm_conv_blocks(B, T, hid), hid / 4 / lanes), 256, bytes, stream, static_cast<const bf16*>(up), ld, static_cast<const bf16*>(conv_w), static_cast<const bf16*>(conv_b), static_cast<const bf16*>(gu),
        static_cast<const bf16*>(gx), static_cast<bf16*>(gup), partial, B, T, hid, runs, lanes);
    return launch_status();
  };
  return run == 16 ? go(conv_bwd_kernel<16>) : go(conv_bwd_kernel<4>);
}

int mlstm_weights(const void* q, const void* k, const void* i_w, const void* f_w, const void* i_b, const void* f_b, void* qk_w, void* gate_w,
                  void* gate_b, int H, int d, cudaStream_t stream) {
  const int head8 = d * d / 8, gate8 = H * 3 * H * d / 8, all = 2 * H * head8 + 2 * gate8;
  const auto vecs = [](const void* p) { return static_cast<const uint4*>(p); };
  mxk::launch_kernel(weights_kernel, (all + 255) / 256, 256, 0, stream, vecs(q), vecs(k), vecs(i_w), vecs(f_w), static_cast<const bf16*>(i_b),
                     static_cast<const bf16*>(f_b), static_cast<uint4*>(qk_w), static_cast<uint4*>(gate_w), static_cast<bf16*>(gate_b), H, head8, gate8);
  return launch_status();
}

int mlstm_gates_fwd(const void* logits, const void* k, long long ld, int hp, float scale,
                    float* log_i, float* log_f, void* k_scaled, long long tokens, int H, int d, cudaStream_t stream) {
  const int hid8 = H * d / 8;
  const unsigned vb = static_cast<unsigned>((tokens * hid8 + 255) / 256), gb = static_cast<unsigned>((tokens * H + 255) / 256);
  mxk::launch_kernel(gates_fwd_kernel, vb + gb, 256, 0, stream, static_cast<const bf16*>(logits), static_cast<const bf16*>(k), ld, scale, log_i, log_f, static_cast<bf16*>(k_scaled), tokens, H, hid8, hp, vb);
  return launch_status();
}

int mlstm_gate_blocks(long long tokens) {
  const long long need = (tokens + 63) / 64;
  return static_cast<int>(need < kGateBlocks ? need : kGateBlocks);
}

int mlstm_gates_bwd(const void* logits, const float* glog_i, const float* glog_f, const void* gk_scaled,
                    float scale, void* gk, long long ld, int hp, void* glogits, float* partial, long long tokens, int H, int d,
                    cudaStream_t stream) {
  if (H > 128) return MXK_ERR_UNSUPPORTED;
  const int hid8 = H * d / 8;
  const unsigned vb = static_cast<unsigned>((tokens * hid8 + 255) / 256), gb = static_cast<unsigned>(mlstm_gate_blocks(tokens));
  mxk::launch_kernel(gates_bwd_kernel, vb + gb, 256, 0, stream, static_cast<const bf16*>(logits), glog_i, glog_f,
                                                static_cast<const bf16*>(gk_scaled), scale, static_cast<bf16*>(gk), ld, static_cast<bf16*>(glogits),
                                                partial, tokens, H, hid8, hp, vb);
  return launch_status();
}

int mlstm_out_fwd(const void* h, const void* u, const void* z, long long ld, const void* norm_w, const void* skip, void* g,
                  long long tokens, int H, int d, cudaStream_t stream) {
  const int hid8 = H * d / 8;
  const unsigned blocks = static_cast<unsigned>((tokens * hid8 + 255) / 256);
  const auto go = [&](auto kernel) {
    mxk::launch_kernel(kernel, blocks, 256, 0, stream, static_cast<const bf16*>(h), static_cast<const bf16*>(u), static_cast<const bf16*>(z), ld,
                                       static_cast<const bf16*>(norm_w), static_cast<const bf16*>(skip), static_cast<bf16*>(g), tokens, hid8);
    return launch_status();
  };
  return d == 64 ? go(out_fwd_kernel<8>) : d == 32 ? go(out_fwd_kernel<4>) : d == 16 ? go(out_fwd_kernel<2>) : MXK_ERR_UNSUPPORTED;
}

int mlstm_out_blocks(long long tokens, int hid) {
  const long long per = 256 / (hid / 8), need = (tokens + per - 1) / per, most = 4 * kNumSMs;
  return static_cast<int>(need < most ? need : most);
}

int mlstm_out_bwd(const void* gg, const void* h, const void* u, const void* z, long long ld, const void* norm_w, const void* skip,
                  void* gh, void* gz, long long ld_gz, void* gu, float* partial, long long tokens, int H, int d, cudaStream_t stream) {
  const int hid8 = H * d / 8;
  if (hid8 > 256 || 256 % hid8) return MXK_ERR_UNSUPPORTED;
  const auto go = [&](auto kernel) {
    mxk::launch_kernel(kernel, mlstm_out_blocks(tokens, hid8 * 8), 256, 0, stream, static_cast<const bf16*>(gg), static_cast<const bf16*>(h), static_cast<const bf16*>(u), static_cast<const bf16*>(z), ld,
        static_cast<const bf16*>(norm_w), static_cast<const bf16*>(skip), static_cast<bf16*>(gh), static_cast<bf16*>(gz), ld_gz,
        static_cast<bf16*>(gu), partial, tokens, hid8);
    return launch_status();
  };
  return d == 64 ? go(out_bwd_kernel<8>) : d == 32 ? go(out_bwd_kernel<4>) : d == 16 ? go(out_bwd_kernel<2>) : MXK_ERR_UNSUPPORTED;
}

}  // namespace layers
}  // namespace mxk
