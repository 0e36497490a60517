// What the attention-style layers (linear attention, gated delta rule) do around their chunked kernels, in bf16: products
// of few rows, one-step forms of the mixers for acting, and the delta rule's input normalisation and gates.
#include <cuda_bf16.h>

#include "layers.cuh"
#include "linattn_common.cuh"
#include "mxk_common.cuh"
#include "umma.cuh"

namespace mxk {
namespace layers {
namespace {

using umma::pack8_bf16;
using umma::unpack8_bf16;

__device__ __forceinline__ float bf(const __nv_bfloat16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ float round_bf(float x) { return __bfloat162float(__float2bfloat16(x)); }
__device__ __forceinline__ float sigmoid(float x) { return 1.f / (1.f + __expf(-x)); }
__device__ __forceinline__ float softplus(float x) { return x > 20.f ? x : log1pf(__expf(x)); }

__global__ void __launch_bounds__(256) stack_rows_kernel(WeightRows w, uint4* __restrict__ dst, int padded, int k8) {
  enter_kernel();
  const long long i = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x;
  if (i >= static_cast<long long>(padded) * k8) return;
  int row = static_cast<int>(i / k8);
  const int c = static_cast<int>(i % k8);
  uint4 v = make_uint4(0, 0, 0, 0);
#pragma unroll
  for (int s = 0; s < kMaxWeights; ++s) {
    if (s >= w.count) break;
    if (row < w.rows[s]) {
      v = reinterpret_cast<const uint4*>(w.ptr[s])[static_cast<long long>(row) * k8 + c];
      break;
    }
    row -= w.rows[s];
  }
  dst[i] = v;
}

// Few rows (acting): too little work for 128-row tensor-memory tiles to spread over the SMs, so a block takes 16 x 32
// outputs and its four warps a quarter of the contraction each.  Latency-bound: operands come straight from L2 into
// mma.sync fragments, eight consecutive k per lane and load -- the order of k inside a product is free, so those eight
// serve two k16 steps -- and nothing waits before the last product but the loads themselves.
__global__ void __launch_bounds__(128) small_product_kernel(const __nv_bfloat16* __restrict__ x, WeightRows w,
                                                            const __nv_bfloat16* __restrict__ bias, int bias_from,
                                                            __nv_bfloat16* __restrict__ c, long long ldc, int M, int N, int K) {
  enter_kernel();
  __shared__ float part[4][16][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int m0 = blockIdx.y * 16, n0 = blockIdx.x * 32;
  const int steps = K / 32, per = (steps + 3) / 4;
  const int first = warp * per, last = min(steps, first + per);
  float acc[4][4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
  const __nv_bfloat16* a0 = x + static_cast<long long>(min(m0 + g, M - 1)) * K + t * 8;
  const __nv_bfloat16* a1 = x + static_cast<long long>(min(m0 + g + 8, M - 1)) * K + t * 8;
  const __nv_bfloat16* b[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    int row = min(n0 + j * 8 + g, N - 1), s = 0;
    while (row >= w.rows[s]) row -= w.rows[s++];
    b[j] = static_cast<const __nv_bfloat16*>(w.ptr[s]) + static_cast<long long>(row) * K + t * 8;
  }
#pragma unroll 2
  for (int i = first; i < last; ++i) {
    const uint4 u0 = *reinterpret_cast<const uint4*>(a0 + i * 32), u1 = *reinterpret_cast<const uint4*>(a1 + i * 32);
    uint4 v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = __ldg(reinterpret_cast<const uint4*>(b[j] + i * 32));
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                   : "+f"(acc[j][0]), "+f"(acc[j][1]), "+f"(acc[j][2]), "+f"(acc[j][3])
                   : "r"(u0.x), "r"(u1.x), "r"(u0.y), "r"(u1.y), "r"(v[j].x), "r"(v[j].y));
      asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                   : "+f"(acc[j][0]), "+f"(acc[j][1]), "+f"(acc[j][2]), "+f"(acc[j][3])
                   : "r"(u0.z), "r"(u1.z), "r"(u0.w), "r"(u1.w), "r"(v[j].z), "r"(v[j].w));
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    part[warp][g][j * 8 + 2 * t] = acc[j][0];
    part[warp][g][j * 8 + 2 * t + 1] = acc[j][1];
    part[warp][g + 8][j * 8 + 2 * t] = acc[j][2];
    part[warp][g + 8][j * 8 + 2 * t + 1] = acc[j][3];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 16 * 32; i += 128) {
    const int r = i >> 5, n = i & 31;
    if (m0 + r < M && n0 + n < N) {
      float v = (part[0][r][n] + part[1][r][n]) + (part[2][r][n] + part[3][r][n]);
      if (bias && n0 + n >= bias_from) v += bf(bias + n0 + n - bias_from);
      c[(m0 + r) * ldc + n0 + n] = __float2bfloat16(v);
    }
  }
}

// ------------------------------------------------------------------------------------------------ one time step
// HBM-bound on the state (read once, written once: 33.5 MB for 256 x 4 x 64 x 64, 5.2 us); one block per sequence, so that
// the RMSNorm over its heads needs no second pass.  LPR lanes share a state row, 16 bytes per lane and vector.
constexpr int kStepThreads = 512;

__device__ __forceinline__ float block_sum(float v, float* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.f;
#pragma unroll
  for (int i = 0; i < kStepThreads / 32; ++i) t += red[i];
  return t;
}

// o (already rounded to bf16) -> RMSNorm -> y
__device__ __forceinline__ void norm_row(const float* o, int hid, const __nv_bfloat16* norm_w, float norm_eps, __nv_bfloat16* y, float* red) {
  float ss = 0.f;
  for (int c = threadIdx.x; c < hid; c += kStepThreads) ss = fmaf(o[c], o[c], ss);
  const float rstd = rsqrtf(block_sum(ss, red) / hid + norm_eps);
  for (int c = threadIdx.x; c < hid; c += kStepThreads) y[c] = __float2bfloat16(o[c] * rstd * bf(norm_w + c));
}

template <int D>
__global__ void __launch_bounds__(kStepThreads) linattn_step_kernel(const __nv_bfloat16* __restrict__ qkv, long long ld,
                                                                    const float* __restrict__ s0, const float* __restrict__ z0,
                                                                    const uint8_t* __restrict__ done,
                                                                    const __nv_bfloat16* __restrict__ norm_w, float norm_eps,
                                                                    float eps, __nv_bfloat16* __restrict__ y,
                                                                    float* __restrict__ s_last, float* __restrict__ z_last, int H) {
  enter_kernel();
  extern __shared__ __align__(16) float sm[];   // q | k | v | o of all heads, then the denominators
  constexpr int kVecs = D / 32, kLanes = 8;     // 16-byte vectors per lane; lanes per row
  __shared__ float red[kStepThreads / 32];
  const int hid = H * D, tid = threadIdx.x, b = blockIdx.x;
  float *q = sm, *k = sm + hid, *v = sm + 2 * hid, *o = sm + 3 * hid, *den = sm + 4 * hid;
  const bool fresh = done && done[b] != 0;
  const bool keep_s = s0 && !fresh, keep_z = z0 && !fresh;
  for (int i = tid; i < 3 * hid / 8; i += kStepThreads) {
    uint4 raw = *reinterpret_cast<const uint4*>(qkv + b * ld + i * 8);
    if (i < 2 * hid / 8) raw = linattn::phi8(raw);
    unpack8_bf16(raw, sm + i * 8);
  }
  __syncthreads();
  const size_t zb = static_cast<size_t>(b) * hid;
  for (int h = tid >> 5; h < H; h += kStepThreads / 32) {
    float s = 0.f;
    for (int i = tid & 31; i < D; i += 32) {
      const float z = (keep_z ? z0[zb + h * D + i] : 0.f) + k[h * D + i];
      z_last[zb + h * D + i] = z;
      s = fmaf(z, q[h * D + i], s);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if ((tid & 31) == 0) den[h] = 1.f / fmaxf(s, eps);
  }
  const int l = tid % kLanes;
#pragma unroll 4
  for (int r = tid / kLanes; r < hid; r += kStepThreads / kLanes) {
    const int h = r / D;
    const size_t at = (zb + r) * D + l * 4;
    float4 st[kVecs];
#pragma unroll
    for (int i = 0; i < kVecs; ++i)
      st[i] = keep_s ? ld_stream(reinterpret_cast<const float4*>(s0 + at + i * 32)) : make_float4(0.f, 0.f, 0.f, 0.f);
    float num = 0.f;
#pragma unroll
    for (int i = 0; i < kVecs; ++i) {
      const float4 kk = *reinterpret_cast<const float4*>(k + h * D + l * 4 + i * 32), qq = *reinterpret_cast<const float4*>(q + h * D + l * 4 + i * 32);
      st[i].x = fmaf(v[r], kk.x, st[i].x); st[i].y = fmaf(v[r], kk.y, st[i].y);
      st[i].z = fmaf(v[r], kk.z, st[i].z); st[i].w = fmaf(v[r], kk.w, st[i].w);
      num = fmaf(st[i].x, qq.x, fmaf(st[i].y, qq.y, fmaf(st[i].z, qq.z, fmaf(st[i].w, qq.w, num))));
      st_stream(reinterpret_cast<float4*>(s_last + at + i * 32), st[i]);
    }
#pragma unroll
    for (int off = kLanes / 2; off > 0; off >>= 1) num += __shfl_xor_sync(0xffffffffu, num, off);
    if (l == 0) o[r] = num;
  }
  __syncthreads();
  for (int c = tid; c < hid; c += kStepThreads) o[c] = round_bf(o[c] * den[c / D]);
  __syncthreads();
  norm_row(o, hid, norm_w, norm_eps, y + zb, red);
}

template <int D>
__global__ void __launch_bounds__(kStepThreads) gdelta_step_kernel(const __nv_bfloat16* __restrict__ qkvg, long long ld,
                                                                   const float* __restrict__ s0, const uint8_t* __restrict__ done,
                                                                   const __nv_bfloat16* __restrict__ norm_w, float norm_eps,
                                                                   __nv_bfloat16* __restrict__ y, float* __restrict__ s_last, int H) {
  enter_kernel();
  extern __shared__ __align__(16) float sm[];   // q | k | v | o, then alpha | beta
  constexpr int kLanes = 16, kVecs = D / 64;
  __shared__ float red[kStepThreads / 32];
  const int hid = H * D, tid = threadIdx.x, b = blockIdx.x;
  float *q = sm, *k = sm + hid, *v = sm + 2 * hid, *o = sm + 3 * hid, *alpha = sm + 4 * hid, *beta = alpha + H;
  const bool keep = s0 && !(done && done[b] != 0);
  const __nv_bfloat16* row = qkvg + b * ld;
  for (int i = tid; i < 3 * hid / 8; i += kStepThreads) unpack8_bf16(*reinterpret_cast<const uint4*>(row + i * 8), sm + i * 8);
  for (int h = tid; h < H; h += kStepThreads) {
    beta[h] = sigmoid(bf(row + 3 * hid + h));
    alpha[h] = keep ? __expf(-softplus(bf(row + 3 * hid + H + h))) : 0.f;
  }
  __syncthreads();
  for (int i = tid >> 5; i < 2 * H; i += kStepThreads / 32) {   // a warp per head vector of q and k
    float* const x = sm + i * D;
    float ss = 0.f;
    for (int c = tid & 31; c < D; c += 32) ss = fmaf(x[c], x[c], ss);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
    const float inv = 1.f / fmaxf(sqrtf(ss), 1e-12f);
    for (int c = tid & 31; c < D; c += 32) x[c] = round_bf(x[c] * inv);
  }
  __syncthreads();
  const size_t base = static_cast<size_t>(b) * hid;
  const int l = tid % kLanes;
#pragma unroll 2
  for (int r = tid / kLanes; r < hid; r += kStepThreads / kLanes) {
    const int h = r / D;
    const size_t at = (base + r) * D + l * 4;
    float4 st[kVecs], kk[kVecs];
    float sk = 0.f;
    const float a = alpha[h];
#pragma unroll
    for (int i = 0; i < kVecs; ++i) {
      st[i] = keep ? ld_stream(reinterpret_cast<const float4*>(s0 + at + i * 64)) : make_float4(0.f, 0.f, 0.f, 0.f);
      kk[i] = *reinterpret_cast<const float4*>(k + h * D + l * 4 + i * 64);
    }
#pragma unroll
    for (int i = 0; i < kVecs; ++i) {
      st[i].x *= a; st[i].y *= a; st[i].z *= a; st[i].w *= a;
      sk = fmaf(st[i].x, kk[i].x, fmaf(st[i].y, kk[i].y, fmaf(st[i].z, kk[i].z, fmaf(st[i].w, kk[i].w, sk))));
    }
#pragma unroll
    for (int off = kLanes / 2; off > 0; off >>= 1) sk += __shfl_xor_sync(0xffffffffu, sk, off);
    const float u = beta[h] * (v[r] - sk);
    float num = 0.f;
#pragma unroll
    for (int i = 0; i < kVecs; ++i) {
      const float4 qq = *reinterpret_cast<const float4*>(q + h * D + l * 4 + i * 64);
      st[i].x = fmaf(u, kk[i].x, st[i].x); st[i].y = fmaf(u, kk[i].y, st[i].y);
      st[i].z = fmaf(u, kk[i].z, st[i].z); st[i].w = fmaf(u, kk[i].w, st[i].w);
      num = fmaf(st[i].x, qq.x, fmaf(st[i].y, qq.y, fmaf(st[i].z, qq.z, fmaf(st[i].w, qq.w, num))));
      st_stream(reinterpret_cast<float4*>(s_last + at + i * 64), st[i]);
    }
#pragma unroll
    for (int off = kLanes / 2; off > 0; off >>= 1) num += __shfl_xor_sync(0xffffffffu, num, off);
    if (l == 0) o[r] = round_bf(num);
  }
  __syncthreads();
  norm_row(o, hid, norm_w, norm_eps, y + base, red);
}

// ------------------------------------------------------------------------------------- delta rule: inputs, gates
// HBM-bound.  LPH lanes hold one head vector, 16 bytes each; the first blocks take the gates, whose loads are few and slow
// (after the vectors they were a tail of their own).  A thread walks over kWalk vectors at a time, all loaded before the
// first is used, and divides only once: a 64-bit division per vector took as long as its 16 bytes.
constexpr int kWalk = 4;
struct Walk {   // vector i of the q and k columns is (token, column) = (i / width, i % width)
  long long tok;
  int c, width, dtok, dc;
  __device__ __forceinline__ Walk(unsigned block, unsigned blocks, int w) : width(w) {
    const long long i = static_cast<long long>(block) * 256 + threadIdx.x, step = static_cast<long long>(blocks) * 256;
    tok = i / w;
    c = static_cast<int>(i % w);
    dtok = static_cast<int>(step / w);
    dc = static_cast<int>(step % w);
  }
  __device__ __forceinline__ void next() {
    tok += dtok;
    c += dc;
    if (c >= width) { c -= width; ++tok; }
  }
};

template <int LPH>
__global__ void __launch_bounds__(256) delta_inputs_kernel(const __nv_bfloat16* __restrict__ qkvg, long long ld,
                                                           uint4* __restrict__ q, uint4* __restrict__ k, float* __restrict__ alpha,
                                                           float* __restrict__ beta, long long tokens, int H, unsigned gate_blocks) {
  enter_kernel();
  const int hid8 = H * LPH;
  if (blockIdx.x >= gate_blocks) {
    Walk w(blockIdx.x - gate_blocks, gridDim.x - gate_blocks, 2 * hid8);
    // (of a warp's lanes the first is the last to run out)
    while (__shfl_sync(0xffffffffu, w.tok, 0) < tokens) {
      uint4 raw[kWalk];
      uint4* dst[kWalk];
#pragma unroll
      for (int u = 0; u < kWalk; ++u) {
        const bool in = w.tok < tokens;
        raw[u] = in ? ld_stream(reinterpret_cast<const uint4*>(qkvg + w.tok * ld + w.c * 8)) : make_uint4(0, 0, 0, 0);
        dst[u] = in ? (w.c < hid8 ? q : k) + w.tok * hid8 + (w.c < hid8 ? w.c : w.c - hid8) : nullptr;
        w.next();
      }
#pragma unroll
      for (int u = 0; u < kWalk; ++u) {
        float x[8], ss = 0.f;
        unpack8_bf16(raw[u], x);
#pragma unroll
        for (int e = 0; e < 8; ++e) ss = fmaf(x[e], x[e], ss);
#pragma unroll
        for (int off = 1; off < LPH; off <<= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
        const float inv = 1.f / fmaxf(sqrtf(ss), 1e-12f);
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] *= inv;
        if (dst[u]) *dst[u] = pack8_bf16(x);
      }
    }
  } else {
    const long long i = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x;
    if (i >= tokens * H) return;
    const long long tok = i / H;
    const int h = static_cast<int>(i % H);
    const __nv_bfloat16* g = qkvg + tok * ld + 3 * hid8 * 8;
    beta[i] = sigmoid(bf(g + h));
    alpha[i] = __expf(-softplus(bf(g + H + h)));
  }
}

template <int LPH>
__global__ void __launch_bounds__(256) delta_inputs_bwd_kernel(const __nv_bfloat16* __restrict__ qkvg, long long ld,
                                                               const uint4* __restrict__ dq, const uint4* __restrict__ dk,
                                                               const float* __restrict__ dalpha, const float* __restrict__ dbeta,
                                                               __nv_bfloat16* __restrict__ g, float* __restrict__ partial,
                                                               long long tokens, int H, unsigned gate_blocks) {
  enter_kernel();
  __shared__ float red[256];
  const int hid8 = H * LPH, hid = hid8 * 8;
  if (blockIdx.x >= gate_blocks) {
    Walk w(blockIdx.x - gate_blocks, gridDim.x - gate_blocks, 2 * hid8);
    while (__shfl_sync(0xffffffffu, w.tok, 0) < tokens) {
      uint4 xr[kWalk], dr[kWalk];
      uint4* dst[kWalk];
#pragma unroll
      for (int u = 0; u < kWalk; ++u) {
        const bool in = w.tok < tokens;
        const long long at = w.tok * ld + w.c * 8;
        xr[u] = in ? ld_stream(reinterpret_cast<const uint4*>(qkvg + at)) : make_uint4(0, 0, 0, 0);
        dr[u] = in ? ld_stream((w.c < hid8 ? dq : dk) + w.tok * hid8 + (w.c < hid8 ? w.c : w.c - hid8)) : make_uint4(0, 0, 0, 0);
        dst[u] = in ? reinterpret_cast<uint4*>(g + at) : nullptr;
        w.next();
      }
#pragma unroll
      for (int u = 0; u < kWalk; ++u) {
        float x[8], d[8], ss = 0.f, sd = 0.f;
        unpack8_bf16(xr[u], x);
        unpack8_bf16(dr[u], d);
#pragma unroll
        for (int e = 0; e < 8; ++e) { ss = fmaf(x[e], x[e], ss); sd = fmaf(x[e], d[e], sd); }
#pragma unroll
        for (int off = 1; off < LPH; off <<= 1) {
          ss += __shfl_xor_sync(0xffffffffu, ss, off);
          sd += __shfl_xor_sync(0xffffffffu, sd, off);
        }
        const float inv = 1.f / fmaxf(sqrtf(ss), 1e-12f), ydy = sd * inv;
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = inv * (d[e] - x[e] * inv * ydy);
        if (dst[u]) *dst[u] = pack8_bf16(x);
      }
    }
    return;
  }
  // gates: columns 0..H-1 beta, H..2H-1 decay, then the padding
  const int cols = static_cast<int>(ld) - 3 * hid, per = 256 / cols;
  const int c = threadIdx.x % cols, ro = threadIdx.x / cols;
  const unsigned blocks = gate_blocks, blk = blockIdx.x;
  float sum = 0.f;
  if (ro < per)
#pragma unroll 4
    for (long long tok = static_cast<long long>(blk) * per + ro; tok < tokens; tok += static_cast<long long>(blocks) * per) {
      float v = 0.f;
      if (c < 2 * H) {
        const float z = bf(qkvg + tok * ld + 3 * hid + c), s = sigmoid(z);
        v = round_bf(c < H ? dbeta[tok * H + c] * s * (1.f - s) : -dalpha[tok * H + c - H] * __expf(-softplus(z)) * s);
      }
      g[tok * ld + 3 * hid + c] = __float2bfloat16(v);
      sum += v;
    }
  red[threadIdx.x] = sum;
  __syncthreads();
  if (threadIdx.x < 2 * H) {
    float v = 0.f;
    for (int i = 0; i < per; ++i) v += red[i * cols + threadIdx.x];
    partial[blk * 2 * H + threadIdx.x] = v;
  }
}

constexpr int kGateBlocks = 2 * kNumSMs;
unsigned walk_blocks(long long vecs) {   // a wave of eight blocks an SM
  const long long need = (vecs + 256 * kWalk - 1) / (256 * kWalk);
  return static_cast<unsigned>(need < 8 * kNumSMs ? need : 8 * kNumSMs);
}

}  // namespace

int stack_rows(const WeightRows& w, void* dst, int padded, int K, cudaStream_t stream) {
  if (K % 8 || w.count < 1 || w.count > kMaxWeights) return MXK_ERR_UNSUPPORTED;
  const long long vecs = static_cast<long long>(padded) * (K / 8);
  mxk::launch_kernel(stack_rows_kernel, static_cast<unsigned>((vecs + 255) / 256), 256, 0, stream, w, static_cast<uint4*>(dst), padded, K / 8);
  return launch_status();
}

int small_product(const void* x, const WeightRows& w, const void* bias, int bias_from, void* c, long long ldc, int M, int K, cudaStream_t stream) {
  if (K % 32 || M <= 0 || w.count < 1 || w.count > kMaxWeights) return MXK_ERR_UNSUPPORTED;
  int N = 0;
  for (int i = 0; i < w.count; ++i) N += w.rows[i];
  mxk::launch_kernel(small_product_kernel, dim3((N + 31) / 32, (M + 15) / 16), 128, 0, stream, static_cast<const __nv_bfloat16*>(x), w, static_cast<const __nv_bfloat16*>(bias), bias_from, static_cast<__nv_bfloat16*>(c), ldc, M, N, K);
  return launch_status();
}

int linattn_step(const void* qkv, long long ld, const float* s0, const float* z0, const uint8_t* done, const void* norm_w,
                 float norm_eps, float eps, void* y, float* s_last, float* z_last, int B, int H, int d, cudaStream_t stream) {
  const int bytes = (4 * H * d + H) * static_cast<int>(sizeof(float));
  const auto* x = static_cast<const __nv_bfloat16*>(qkv);
  const auto* nw = static_cast<const __nv_bfloat16*>(norm_w);
  auto* out = static_cast<__nv_bfloat16*>(y);
  if (bytes > 48 * 1024) return MXK_ERR_UNSUPPORTED;
  if (d == 64) mxk::launch_kernel(linattn_step_kernel<64>, B, kStepThreads, bytes, stream, x, ld, s0, z0, done, nw, norm_eps, eps, out, s_last, z_last, H);
  else if (d == 32) mxk::launch_kernel(linattn_step_kernel<32>, B, kStepThreads, bytes, stream, x, ld, s0, z0, done, nw, norm_eps, eps, out, s_last, z_last, H);
  else return MXK_ERR_UNSUPPORTED;
  return launch_status();
}

int gdelta_step(const void* qkvg, long long ld, const float* s0, const uint8_t* done, const void* norm_w,
                float norm_eps, void* y, float* s_last, int B, int H, int d, cudaStream_t stream) {
  const int bytes = (4 * H * d + 2 * H) * static_cast<int>(sizeof(float));
  const auto* x = static_cast<const __nv_bfloat16*>(qkvg);
  const auto* nw = static_cast<const __nv_bfloat16*>(norm_w);
  auto* out = static_cast<__nv_bfloat16*>(y);
  if (bytes > 48 * 1024) return MXK_ERR_UNSUPPORTED;
  if (d == 128) mxk::launch_kernel(gdelta_step_kernel<128>, B, kStepThreads, bytes, stream, x, ld, s0, done, nw, norm_eps, out, s_last, H);
  else if (d == 64) mxk::launch_kernel(gdelta_step_kernel<64>, B, kStepThreads, bytes, stream, x, ld, s0, done, nw, norm_eps, out, s_last, H);
  else return MXK_ERR_UNSUPPORTED;
  return launch_status();
}

int delta_inputs(const void* qkvg, long long ld, void* q, void* k, float* alpha, float* beta,
                 long long tokens, int H, int d, cudaStream_t stream) {
  const long long vecs = tokens * 2 * H * (d / 8);
  const unsigned vb = walk_blocks(vecs), gb = static_cast<unsigned>((tokens * H + 255) / 256);
  const auto* x = static_cast<const __nv_bfloat16*>(qkvg);
  if (d == 64) mxk::launch_kernel(delta_inputs_kernel<8>, vb + gb, 256, 0, stream, x, ld, static_cast<uint4*>(q), static_cast<uint4*>(k), alpha, beta, tokens, H, gb);
  else if (d == 128) mxk::launch_kernel(delta_inputs_kernel<16>, vb + gb, 256, 0, stream, x, ld, static_cast<uint4*>(q), static_cast<uint4*>(k), alpha, beta, tokens, H, gb);
  else return MXK_ERR_UNSUPPORTED;
  return launch_status();
}

int delta_gate_blocks(long long tokens) {
  const long long need = (tokens + 63) / 64;
  return static_cast<int>(need < kGateBlocks ? need : kGateBlocks);
}

int delta_inputs_bwd(const void* qkvg, long long ld, const void* dq, const void* dk, const float* dalpha,
                     const float* dbeta, void* g, float* partial, long long tokens, int H, int d, cudaStream_t stream) {
  if (ld - 3 * H * d > 256 || ld - 3 * H * d < 2 * H) return MXK_ERR_UNSUPPORTED;
  const long long vecs = tokens * 2 * H * (d / 8);
  const unsigned vb = walk_blocks(vecs), gb = static_cast<unsigned>(delta_gate_blocks(tokens));
  const auto* x = static_cast<const __nv_bfloat16*>(qkvg);
  auto* out = static_cast<__nv_bfloat16*>(g);
  if (d == 64) mxk::launch_kernel(delta_inputs_bwd_kernel<8>, vb + gb, 256, 0, stream, x, ld, static_cast<const uint4*>(dq), static_cast<const uint4*>(dk), dalpha, dbeta, out, partial, tokens, H, gb);
  else if (d == 128) mxk::launch_kernel(delta_inputs_bwd_kernel<16>, vb + gb, 256, 0, stream, x, ld, static_cast<const uint4*>(dq), static_cast<const uint4*>(dk), dalpha, dbeta, out, partial, tokens, H, gb);
  else return MXK_ERR_UNSUPPORTED;
  return launch_status();
}

}  // namespace layers
}  // namespace mxk
