// The angle of a one-sided Jacobi rotation.
#pragma once

#include <cuda_runtime.h>

namespace tg {

// The rotation of columns with squared norms al, be and |inner product| g > 0:
// t = tan, the smaller root of t^2 + 2 zeta t = 1 with zeta = (be - al) / 2g,
// from single-precision arithmetic; c = 1 / sqrt(1 + t^2) and s = c t in double,
// so that the rotation is orthogonal to double precision whatever the error
// of t.  That error, 1e-7, leaves 1e-7 of the inner product, below the square
// of it that a sweep leaves anyway; in double precision the three square roots
// were the longest part of a rotation's chain.
__device__ __forceinline__ void rotation_angle(double al, double be, double g, double& t, double& c, double& s) {
  const double tau = be - al, g2 = 2.0 * g;
  // both scaled by the power of two that takes the larger one into [1, 2)
  const int ha = __double2hiint(fabs(tau)), hg = __double2hiint(g2);
  const int e = min((ha > hg ? ha : hg) & 0x7ff00000, 0x7fd00000);
  const double scale = __hiloint2double(0x7fe00000 - e, 0);
  const float a = __double2float_rn(fabs(tau) * scale), b = __double2float_rn(g2 * scale);
  const float w = fmaf(a, a, b * b);
  const float tf = __fdividef(b, a + w * rsqrtf(w));
  const float cf = rsqrtf(fmaf(tf, tf, 1.0f));
  // a rotation this small is g / tau to all digits; as a float it could vanish
  t = b < 1e-18f ? g / tau : copysign(static_cast<double>(tf), tau);
  const double c0 = static_cast<double>(cf), h = fma(t, t, 1.0) * c0;
  const double err = fma(-h, c0, 1.0);  // 1 - (1 + t^2) c0^2, about 1e-7
  c = fma(c0 * err, fma(err, 0.375, 0.5), c0);
  s = c * t;
}

}  // namespace tg
