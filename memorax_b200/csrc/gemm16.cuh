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
// `ws` (workspace_bytes) holds the float32 partial products of a split contraction.
size_t workspace_bytes(int batch, int M, int N, int K);
int run(const Matrix& a, bool a_rows, const Matrix& b, bool b_rows, const void* bias, void* c, long long ldc,
        long long c_batch_stride, bool accumulate, int batch, int M, int N, int K, void* ws, size_t ws_bytes, int* status,
        cudaStream_t stream);

}  // namespace gemm16
}  // namespace mxk
