// Exact scaling of matrices whose products would leave the range of double.
#pragma once

#include <cuda_runtime.h>

namespace tg {

// The high word of |x|: it orders like |x|, and from 0x7ff00000 on x is not finite.
__device__ __forceinline__ int magnitude(double x) { return __double2hiint(x) & 0x7fffffff; }
__device__ __forceinline__ int magnitude(double2 x) { return max(magnitude(x.x), magnitude(x.y)); }

// A power of two that takes a matrix with the largest magnitude `top` to
// entries of about 1, and its inverse.  1 between 2^-100 and 2^100, where the
// squares of inner products of its columns stay in range (so the scaling
// changes nothing there), and for a matrix of zeros or with values that are not
// finite.
__device__ __forceinline__ double range_scale(int top, double& inverse) {
  const int e = top >> 20;  // biased exponent
  inverse = 1.0;
  if (top == 0 || e == 0x7ff || (e >= 1023 - 100 && e <= 1023 + 100)) return 1.0;
  const int s = min(max(2046 - e, 1), 2045);
  inverse = __hiloint2double((2046 - s) << 20, 0);
  return __hiloint2double(s << 20, 0);
}

}  // namespace tg
