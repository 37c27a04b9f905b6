// Device helpers that several H.v kernel files share.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "kernels.cuh"

namespace qed {

// Inter-spin density-density terms of one state (see InterSpin). MASKED false: without
// mode 4, for kernels whose operator has it as mode 2.
template <bool MASKED = true>
__device__ __forceinline__ double inter_term(const InterSpin &it, uint32_t up, uint32_t dn) {
  if (it.mode == 1) return it.u * (double)__popc(up & dn);
  if (MASKED && it.mode == 4) return it.sum[__popc(up & dn & it.mask)];
  double s = 0.0;
  if (it.mode == 2) {
    uint32_t w = up & dn;
    while (w) {
      int r = __ffs(w) - 1;
      s += __ldg(it.v + r);
      w &= w - 1;
    }
  } else if (it.mode == 3) {
    uint32_t wd = dn;
    while (wd) {
      int r = __ffs(wd) - 1;
      uint32_t wu = up;
      while (wu) {
        int c = __ffs(wu) - 1;
        s += __ldg(it.v + r * it.n + c);
        wu &= wu - 1;
      }
      wd &= wd - 1;
    }
  }
  return s;
}

// The CTA's sums of NRED values per thread into its row of `partials`, in a
// fixed order.
template <int NRED>
__device__ __forceinline__ void block_reduce_store(double (&v)[NRED], double *partials, int nred) {
  __shared__ double sm[NRED > 0 ? NRED : 1][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int i = 0; i < NRED; ++i) {
    double x = v[i];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) sm[i][warp] = x;
  }
  __syncthreads();
  if (threadIdx.x < nred) {
    double s = 0.0;
    for (int w = 0; w < nw; ++w) s += sm[threadIdx.x][w];
    partials[(size_t)blockIdx.x * Reducer::kMaxRed + threadIdx.x] = s;
  }
}

}  // namespace qed
