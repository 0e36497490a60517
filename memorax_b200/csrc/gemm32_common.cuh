// What the kernels of float32 products share (gemm32.cu, gemm32_long.cu, gemm32_long_outer.cu).
#pragma once

#include "gemm32.cuh"
#include "mxk_common.cuh"
#include "tma.cuh"
#include "umma.cuh"

namespace mxk {
namespace gemm32 {

__device__ __forceinline__ void load8(const float* p, int valid, int vec, float* x) {
  if (valid >= 8 && vec == 8) {
    asm volatile("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]), "=f"(x[4]), "=f"(x[5]), "=f"(x[6]), "=f"(x[7])
                 : "l"(p));
  } else if (valid >= 8 && vec == 4) {
    const float4 u = __ldg(reinterpret_cast<const float4*>(p)), v = __ldg(reinterpret_cast<const float4*>(p) + 1);
    x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w;
    x[4] = v.x; x[5] = v.y; x[6] = v.z; x[7] = v.w;
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] = e < valid ? __ldg(p + e) : 0.f;
  }
}

__device__ __forceinline__ void store8(float* p, int valid, int vec, const float* x) {
  if (valid >= 8 && vec == 8) {
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(x[0]), "f"(x[1]), "f"(x[2]),
                 "f"(x[3]), "f"(x[4]), "f"(x[5]), "f"(x[6]), "f"(x[7])
                 : "memory");
  } else if (valid >= 8 && vec == 4) {
    reinterpret_cast<float4*>(p)[0] = make_float4(x[0], x[1], x[2], x[3]);
    reinterpret_cast<float4*>(p)[1] = make_float4(x[4], x[5], x[6], x[7]);
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e)
      if (e < valid) p[e] = x[e];
  }
}

__device__ __forceinline__ void arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(umma::smem_u32(bar)) : "memory");
}

inline int vec_of(const void* p, long long ld) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(p);
  if (a % 32 == 0 && ld % 8 == 0) return 8;
  if (a % 16 == 0 && ld % 4 == 0) return 4;
  return 1;
}

// Two floats to bf16, to the nearest; what lies beyond bf16's largest number, the largest floats and infinity, becomes that
// number (an infinite plane times a zero one would be NaN).
__device__ __forceinline__ uint32_t pack_finite(float lo, float hi) {
  uint32_t v;
  asm("cvt.rn.satfinite.bf16x2.f32 %0, %1, %2;" : "=r"(v) : "f"(hi), "f"(lo));
  return v;
}

// hi / mid / lo bf16 planes of eight floats
__device__ __forceinline__ void split8(const float* x, uint4& hi, uint4& mid, uint4& lo) {
  uint32_t h[4], m[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float a = x[2 * i], b = x[2 * i + 1];
    h[i] = pack_finite(a, b);
    a -= __uint_as_float(h[i] << 16);
    b -= __uint_as_float(h[i] & 0xFFFF0000u);
    m[i] = pack_finite(a, b);
    a -= __uint_as_float(m[i] << 16);
    b -= __uint_as_float(m[i] & 0xFFFF0000u);
    l[i] = pack_finite(a, b);
  }
  hi = make_uint4(h[0], h[1], h[2], h[3]);
  mid = make_uint4(m[0], m[1], m[2], m[3]);
  lo = make_uint4(l[0], l[1], l[2], l[3]);
}

// Eight elements along k from k = 8 g on of W's row n, zero past the matrix.  (What kind of weight it is, is asked once, so that
// the eight loads are under way together.)
__device__ __forceinline__ void weight_vector(const WeightJob& jb, int n, int g, float* x) {
  const int k = g * 8, valid = n < jb.N ? jb.K - k : 0;
  const Weight& w = jb.w;
  const auto loads = [&](const float* p, long long step) {
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] = e < valid ? __ldg(p + e * step) : 0.f;
  };
  const auto pairs = [&](const float* p0, const float* p1, long long step) {   // even and odd elements
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] = e < valid ? __ldg((e & 1 ? p1 : p0) + (e >> 1) * step) : 0.f;
  };
  if (w.form == Form::kComplexRows) {
    if (!jb.transposed) {
      loads(w.ptr[n & 1] + static_cast<long long>(n >> 1) * w.ld + k, 1);
      const float s = w.log_scale && valid > 0 ? expf(__ldg(w.log_scale + (n >> 1))) : 1.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] *= s;
    } else {
      const long long at = static_cast<long long>(k >> 1) * w.ld + n;
      pairs(w.ptr[0] + at, w.ptr[1] + at, w.ld);
#pragma unroll
      for (int e = 0; e < 8; e += 2) {
        const float s = w.log_scale && e < valid ? expf(__ldg(w.log_scale + ((k + e) >> 1))) : 1.f;
        x[e] *= s;
        x[e + 1] *= s;
      }
    }
  } else if (w.form == Form::kComplexCols) {
    if (!jb.transposed) {
      const long long at = static_cast<long long>(n) * w.ld + (k >> 1);
      pairs(w.ptr[0] + at, w.ptr[1] + at, 1);
#pragma unroll
      for (int e = 1; e < 8; e += 2) x[e] = -x[e];
    } else {
      loads(w.ptr[n & 1] + static_cast<long long>(k) * w.ld + (n >> 1), w.ld);
      if (n & 1) {
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = -x[e];
      }
    }
  } else {
    const auto piece = [&](int row, int& start) {
      int s = 0;
      start = 0;
      for (; s < w.count - 1 && row >= w.row_end[s]; ++s) start = w.row_end[s];
      return s;
    };
    int start;
    if (!jb.transposed) {
      const int s = piece(n, start);
      loads(w.ptr[s] + static_cast<long long>(n - start) * w.ld + k, 1);
    } else {
      const int s = piece(k, start);
      if (s == w.count - 1 || k + 7 < w.row_end[s]) {
        loads(w.ptr[s] + static_cast<long long>(k - start) * w.ld + n, w.ld);
      } else {
#pragma unroll 1
        for (int e = 0; e < 8; ++e) {
          const int q = piece(k + e, start);
          const float v = e < valid ? __ldg(w.ptr[q] + static_cast<long long>(k + e - start) * w.ld + n) : 0.f;
#pragma unroll
          for (int i = 0; i < 8; ++i) x[i] = i == e ? v : x[i];
        }
      }
    }
  }
}

// ---- contractions of more than kShortK (gemm32_long.cu) ----
namespace longk {

constexpr int kBK = 64;

struct Plan {
  int bn, splits, k_split;
};
Plan plan(int M, int N, int K);
// Rows of a weight that one CTA of a tile's holds.
__host__ __device__ constexpr int rows_of(int bn) { return bn == 64 ? 64 : bn / 2; }
// C = A W^T; `partial` (splits x M x N) takes the parts of a split contraction.
int launch_weights(const Plan& pl, const float* a, long long lda, const void* image, float* c, long long ldc, int M, int N, int K, const Epilogue& ep,
                   float* partial, int* status, cudaStream_t stream);
// C = A^T B, both stored [K][..] (gemm32_long_outer.cu).
Plan plan_outer(int M, int N, int K);
int launch_outer(const Plan& pl, const float* a, long long lda, const float* b, long long ldb, float* c, long long ldc, int M, int N, int K, float* partial,
                 int* status, cudaStream_t stream);

// Column of a 32-column block in which W's row `n` of the block is placed, so that the eight values that a thread reads from a
// lane with tmem_ld_16x32 are consecutive columns of C and its stores fill whole lines.
__device__ __forceinline__ int placed(int n) { return 8 * ((n >> 1) & 3) + 2 * (n >> 3) + (n & 1); }

constexpr int kBM = 128;
template <int N> __device__ __forceinline__ void more_registers() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void fewer_registers() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

// Arrives on the barrier of this offset in the CTA of rank 0: tensor memory has been read (tcgen05 fences order that; a release
// at cluster scope would wait for every access to global memory under way, 1900 cycles).
__device__ __forceinline__ void arrive_read(uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %0, 0;\n\t"
      "mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [ra];\n\t}\n" ::"r"(umma::smem_u32(bar))
      : "memory");
}
// The same after writes to shared memory that the tensor core is to read.
__device__ __forceinline__ void arrive_written(uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %0, 0;\n\t"
      "mbarrier.arrive.shared::cluster.b64 _, [ra];\n\t}\n" ::"r"(umma::smem_u32(bar))
      : "memory");
}
// 16 TMEM lanes x 32 columns: r[4 j + 2 h + e] is lane (lane / 4) + 8 h, column 8 j + 2 (lane % 4) + e.
__device__ __forceinline__ void tmem_ld_16x32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// Four floats of shared memory, read here and nowhere else: a plain load may be repeated where its values are used, after the tile
// has been given back.
__device__ __forceinline__ void read_once(const void* p, float* x) {
  asm volatile("ld.volatile.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]) : "r"(umma::smem_u32(p)) : "memory");
}
__device__ __forceinline__ float read_once(const void* p) {
  float x;
  asm volatile("ld.volatile.shared.f32 %0, [%1];" : "=f"(x) : "r"(umma::smem_u32(p)) : "memory");
  return x;
}
__device__ __forceinline__ void load_box(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(umma::smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(umma::smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}

}  // namespace longk
}  // namespace gemm32
}  // namespace mxk
