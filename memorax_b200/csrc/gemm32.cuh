// float32 matrix products on the tensor cores: host-side interface.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "mxk.h"

namespace mxk {
namespace gemm32 {

constexpr int kMaxSegs = 6;
// Contractions of at most this many elements: gemm32.cu.  Longer ones: gemm32_long.cu, gemm32_long_outer.cu, which are the more precise form
// and, with a weight, the faster one (142 against 187 us at 65536 x 1024 x 256); three stages of theirs or fewer have not been measured.
constexpr int kShortK = 255;

// A row-major weight matrix.  kStacked: rows of up to kMaxSegs arrays on top of each other (the Dense layers that read
// the same input), array s holding rows [row_end[s-1], row_end[s]).  The two others are the complex-diagonal cells'
// projections as real matrices over interleaved (re, im) pairs:
//   kComplexRows: row 2n = re[n] exp(log_scale[n]), row 2n + 1 = im[n] exp(log_scale[n])   (re = ptr[0], im = ptr[1])
//   kComplexCols: column 2n = re[.][n], column 2n + 1 = -im[.][n]
enum class Form { kStacked, kComplexRows, kComplexCols };
struct Weight {
  Form form = Form::kStacked;
  const float* ptr[kMaxSegs] = {};
  int row_end[kMaxSegs] = {};
  int count = 0;
  long long ld = 0;
  const float* log_scale = nullptr;
};
inline Weight weight_of(const float* p, long long ld) {
  Weight w;
  w.ptr[0] = p;
  w.row_end[0] = 0x7fffffff;
  w.count = 1;
  w.ld = ld;
  return w;
}

// What is added to the product on its way out: c = acc + bias[n] + add[m][n] * add_scale[n] (each optional;
// add without add_scale is added as it is).
struct Epilogue {
  const float* bias = nullptr;
  const float* add = nullptr;
  long long ld_add = 0;
  const float* add_scale = nullptr;
};

// Weights in the form the kernel multiplies with: W [N][K] (or its transpose stored [K][N], `transposed`) as hi / mid /
// lo bf16 planes cut into the tiles and stages of the product C[M][N] = A[M][K] W^T, `image_bytes` long.
struct WeightJob {
  Weight w;
  bool transposed = false;
  int N = 0, K = 0;
  int bn = 0;            // tile width the image is cut for (tile_width)
  void* image = nullptr;
};
// lambda[n] = exp(-exp(nu_log[n]) + i exp(theta_log[n])), computed by the launch that splits the weights.
struct LambdaJob {
  const float* nu_log = nullptr;
  const float* theta_log = nullptr;
  float* lambda = nullptr;
  int N = 0;
};
int tile_width(int M, int N, int K);
size_t image_bytes(int M, int N, int K);
// Up to four images in one launch.
int split_weights(const WeightJob* jobs, int count, const LambdaJob& lambda, cudaStream_t stream);

// C[M][N] = A[M][K] W^T from an image made for this M, N, K.
int run_weights(const float* a, long long lda, const void* image, float* c, long long ldc, int M, int N, int K,
                const Epilogue& ep, float* ws, size_t ws_bytes, int* status, cudaStream_t stream);
// C[M][N] = A^T B with A stored [K][M] and B stored [K][N]: the gradient of a weight, contracted over the tokens.
// With `partials` the splits are left in `ws` ([splits][M][N], the count returned there) for the caller to add up.
int run_outer(const float* a, long long lda, const float* b, long long ldb, float* c, long long ldc, int M, int N, int K,
              float* ws, size_t ws_bytes, int* partials, int* status, cudaStream_t stream);
// Partial products of a split contraction (`ws` of either).
size_t workspace_bytes(int M, int N, int K);

}  // namespace gemm32
}  // namespace mxk
