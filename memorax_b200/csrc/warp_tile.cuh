// Small float32 products y[m][n] = sum_k x[m][k] w[n][k]: kSplit warps compute 8 rows of x times 4 rows of w, their lanes
// spread over k.  Blocks of four warps; four to a tile while there are few tiles (the loop over k is a chain of L2 round
// trips: 16 x 256 x 128 took 7.2 us with one warp per tile), one where the tiles fill the machine anyway.
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
                                             int K, int first, int step) {
#pragma unroll 2
    for (int k = first; k < K; k += step) {
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

// Where a thread of a block of four warps works: its tile, and its share of k.
template <int kSplit>
struct TilePlace {
  int tile, first, step, lane;
  __device__ __forceinline__ TilePlace() {
    const int warp = threadIdx.x >> 5;
    lane = threadIdx.x & 31;
    tile = kSplit == 4 ? static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x) * 4 + warp;
    first = kSplit == 4 ? warp * 32 + lane : lane;
    step = 32 * kSplit;
  }
};
// The sum of a tile's warps, in the first of them; the others are done.
template <int kSplit>
__device__ __forceinline__ bool join_warps(float& v, int lane) {
  if constexpr (kSplit == 4) {
    __shared__ float part[3][32];
    const int warp = threadIdx.x >> 5;
    if (warp > 0) part[warp - 1][lane] = v;
    __syncthreads();
    if (warp > 0) return false;
    v += (part[0][lane] + part[1][lane]) + part[2][lane];
  }
  return true;
}
inline bool few_tiles(long long tiles) { return tiles <= 8 * 148; }
inline unsigned tile_blocks(long long tiles) { return static_cast<unsigned>(few_tiles(tiles) ? tiles : (tiles + 3) / 4); }

}  // namespace mxk
