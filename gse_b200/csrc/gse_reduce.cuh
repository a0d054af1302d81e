// gse_reduce.cuh -- deterministic block and grid reductions of doubles shared
// by the energy kernels (gse_kernels.cu, gse_fft.cu).
#pragma once

#include "gse_internal.cuh"

namespace gse {

// ---------------------------------------------------------------------------
// Block reduction of a double into *out, and into partials[blockIdx.x] (fixed order).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void block_sum_at(double v, double* out) {
  __shared__ double red[32];
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) red[w] = v;
  __syncthreads();
  if (w == 0) {
    double s = (lane < (int)(blockDim.x >> 5)) ? red[lane] : 0.0;
    s = warp_sum(s);
    if (lane == 0) *out = s;
  }
}
__device__ __forceinline__ void block_sum_to(double v, double* partials) {
  block_sum_at(v, partials + blockIdx.x);
}

// This thread's share (threadIdx.x, threadIdx.x + blockDim.x, ...) of the sum of
// p[0..n), written by other blocks: eight loads in flight at a time (one after the
// other they cost an L2 round trip each, 3 us for the 2368 blocks of k_green_apply).
__device__ __forceinline__ double partials_share(const double* p, unsigned n) {
  double t = 0.0;
  for (unsigned i = threadIdx.x; i < n; i += 8 * blockDim.x) {
    double v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = i + k * blockDim.x < n ? __ldcg(p + i + k * blockDim.x) : 0.0;
#pragma unroll
    for (int k = 0; k < 8; k++) t += v[k];
  }
  return t;
}

// After block_sum_to: the block that finishes last (a counter at `done`, zero
// between launches) adds the n partials in index order -- the result does not
// depend on which block ran when -- and writes factor * sum to out[0].
__device__ __forceinline__ void last_block_sum_n(double* partials, unsigned n, unsigned* done,
                                                 double factor, double* out) {
  __shared__ bool last;
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;  // uniform in the block
  __threadfence();
  __shared__ double red[32];
  const double t = warp_sum(partials_share(partials, n));
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) red[w] = t;
  __syncthreads();
  if (w == 0) {
    double u = (lane < (int)(blockDim.x >> 5)) ? red[lane] : 0.0;
    u = warp_sum(u);
    if (lane == 0) {
      out[0] = u * factor;
      *done = 0u;
    }
  }
}
// One partial per block.
__device__ __forceinline__ void last_block_sum_counter(double* partials, unsigned* done,
                                                       double factor, double* out) {
  last_block_sum_n(partials, gridDim.x, done, factor, out);
}

}  // namespace gse
