// Fast reciprocal for elimination steps.
#pragma once
#include <cuda_runtime.h>

namespace qed {

// 1 / d for d > 0, within one unit in the last place of the division: the hardware's
// approximation (rcp.approx, at least 20 bits) and two Newton-Raphson steps
// r += r (1 - d r), each doubling the number of correct bits. A division instead costs
// a call with its checks per elimination step. Everything outside (1e-290, 1e290) takes
// the division: zero, subnormal and negative d, infinities, NaN.
__device__ __forceinline__ double reciprocal(double d) {
  if (!(d > 1e-290 && d < 1e290)) return 1.0 / d;
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
  r = fma(r, fma(-d, r, 1.0), r);
  return fma(r, fma(-d, r, 1.0), r);
}

}  // namespace qed
