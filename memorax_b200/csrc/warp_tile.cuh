// Small float32 products y[m][n] = sum_k x[m][k] w[n][k]: a warp computes 8 rows of x times 4 rows of w, its lanes
// spread over k.
#pragma once

namespace mxk {

struct WarpTile {
  float v[32];   // [m][n] partial sums of this lane
  __device__ __forceinline__ WarpTile() {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = 0.f;
  }
  // x: first of `rows` rows (1..8; the others repeat the last one), `ld` apart; w: the four weight rows
  __device__ __forceinline__ void accumulate(const float* __restrict__ x, long long ld, int rows, const float* const (&w)[4],
                                             int K, int lane) {
#pragma unroll 2
    for (int k = lane; k < K; k += 32) {
      float xv[8], wv[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) wv[j] = __ldg(w[j] + k);
#pragma unroll
      for (int i = 0; i < 8; ++i) xv[i] = x[min(i, rows - 1) * ld + k];
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) v[i * 4 + j] = fmaf(xv[i], wv[j], v[i * 4 + j]);
    }
  }
  // Sum over the lanes, scattered: lane l receives entry l = m * 4 + n (31 shuffles for the 32 sums).
  __device__ __forceinline__ float reduce(int lane) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const bool high = (lane & o) != 0;
#pragma unroll
      for (int i = 0; i < o; ++i) {
        const float keep = high ? v[i + o] : v[i], give = high ? v[i] : v[i + o];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
      }
    }
    return v[0];
  }
};

}  // namespace mxk
