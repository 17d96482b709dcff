// The residual sums of a context that marches, as its one-step kernels add them
// (k_finish, k_finish32): the same additions in the same order as in a march.
#pragma once

#include <cuda_runtime.h>

#include "plfbs_internal.hpp"

namespace plfbs {
namespace {

// v[c] of thread b: tile b's sum over its warps' partial sums, in order (0 beyond
// the last tile). A thread per tile and component loads up to 16 of them at a time:
// bound by the latency of these loads, a thread per tile that loaded as it added
// took 8.2 us for 65,536 cells (6.2 so; 4.2 to 5.7 for the sums per block of a context
// that does not march).
// Every thread of the block must call this (it synchronises).
__device__ __forceinline__ void tile_sums(const KernelArgs& a, double v[4]) {
  static_assert(4 * kMaxTiles <= kFinishBlock, "a thread per tile and component");
  __shared__ double sum[4 * kMaxTiles];
  const int t = threadIdx.x, tile = t >> 2, c = t & 3;
  if (tile < a.tiles.n) {
    const int w0 = tile * a.red_warps, w1 = min(w0 + a.red_warps, (a.C + 31) / 32);
    double s = 0.0;
    for (int w = w0; w < w1; w += 16) {
      double x[16];
#pragma unroll
      for (int k = 0; k < 16; k++) x[k] = w + k < w1 ? __ldg(a.partial + 4 * (w + k) + c) : 0.0;
#pragma unroll
      for (int k = 0; k < 16; k++)
        if (w + k < w1) s += x[k];
    }
    sum[t] = s;
  }
  __syncthreads();
  if (t < a.tiles.n)
#pragma unroll
    for (int k = 0; k < 4; k++) v[k] = sum[4 * t + k];
}

}  // namespace
}  // namespace plfbs
