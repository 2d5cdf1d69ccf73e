// Sums of rows of f64 partials (a unit's energies and virial, a block's) in
// an order that does not depend on the launch: tiles of NB_SUM_TILE rows, a
// block each, whose sums replace the tile's first row, then the tiles in the
// last block to finish.  A tile past the rows sums nothing, so a buffer with
// more room gives the same bits.
//
// One block over all rows, a thread a row, took 1,025 µs for the 600,000
// units of the 1.07 M-atom box (39 MB) and 31 µs for 23,490 atoms.
#pragma once
#include "nb_common.cuh"

#define NB_SUM_TILE 2048

namespace {

// The sum of rows [tile NB_SUM_TILE, + NB_SUM_TILE) of `rows` (W doubles a row)
// into the tile's first row, by a block of 32 W threads: thread t takes
// column t % W of every 32nd row (whole lines at a time), then the 32
// threads of a column are added in order.
template <int W>
__device__ __forceinline__ void nb_tile_rows(double *__restrict__ p, int64_t rows, int tile, double *s) {
  const int64_t first = (int64_t)tile * NB_SUM_TILE;
  if (first >= rows) return;
  const int64_t last = min(rows, first + NB_SUM_TILE) * W;
  double v = 0.0;
#pragma unroll 8
  for (int64_t e = first * W + threadIdx.x; e < last; e += 32 * W) v += p[e];
  s[threadIdx.x] = v;
  __syncthreads();
  if (threadIdx.x < W) {
    double t = 0.0;
#pragma unroll
    for (int k = 0; k < 32; ++k) t += s[k * W + threadIdx.x];
    p[first * W + threadIdx.x] = t;
  }
  __syncthreads();
}

// True in the block that finishes last (every block calls it once); the
// counter is back at zero for the next launch.
__device__ __forceinline__ bool nb_last_block(unsigned int *done) {
  __shared__ unsigned s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    s_last = atomicAdd(done, 1u) == gridDim.x - 1 ? 1u : 0u;
    if (s_last) *done = 0u;
  }
  __syncthreads();
  __threadfence();
  return s_last != 0u;
}

// The sum of column t (threads t < W) over the tiles' first rows, in tile
// order within each of 32 shares; the same block size as nb_tile_rows.
template <int W>
__device__ __forceinline__ double nb_sum_tiles(const double *p, int64_t rows, double *s) {
  const int64_t tiles = (rows + NB_SUM_TILE - 1) / NB_SUM_TILE;
  double v = 0.0;
  const int col = threadIdx.x % W;
  for (int64_t t = threadIdx.x / W; t < tiles; t += 32) v += __ldcg(p + t * NB_SUM_TILE * W + col);
  s[threadIdx.x] = v;
  __syncthreads();
  double total = 0.0;
  if (threadIdx.x < W) {
#pragma unroll
    for (int k = 0; k < 32; ++k) total += s[k * W + threadIdx.x];
  }
  __syncthreads();
  return total;
}

}  // namespace
