// bf16 matrix products (float32 accumulation) on tcgen05: host-side interface (gemm16.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "mxk.h"

namespace mxk {
namespace gemm16 {

// A stored row-major matrix per batch: rows x cols elements, `ld` apart (a multiple of 8), batches `batch_stride` apart.
struct Matrix {
  const void* ptr;
  long long ld;
  long long batch_stride = 0;
};

// C[b][M][N] = op(A) op(B) (+ bias[N]) (+ C, when `accumulate`), bf16.
//   a_rows = false: A is stored [M][K]; true: [K][M].   b_rows = false: B is stored [N][K]; true: [K][N].
struct Job {
  Matrix a, b;
  const void* bias;
  void* c;
  long long ldc, c_batch_stride;
  bool accumulate;
  int batch, M, N, K;
};
// `ws` (workspace_bytes) holds the float32 partial products of a split contraction.
size_t workspace_bytes(int batch, int M, int N, int K);
int run(const Job& job, bool a_rows, bool b_rows, void* ws, size_t ws_bytes, int* status, cudaStream_t stream);
// Up to kMaxGroup products that do not depend on one another, in one launch and one for the sums of what was split.
constexpr int kMaxGroup = 6;
size_t group_workspace_bytes(const Job* jobs, int count);
int run_group(const Job* jobs, int count, bool a_rows, bool b_rows, void* ws, size_t ws_bytes, int* status, cudaStream_t stream);

}  // namespace gemm16
}  // namespace mxk
