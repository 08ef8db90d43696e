// FP64 roots and reciprocals from FP32 starts by Newton's method in its
// division-free forms, for the FP64 pipe of 2 operations a clock per SM: a
// division or root is some 20 operations there.  Within 3 units of 2^-53 of
// CUDA's results for the roots, 12 for beta (tests/roots_check.cu).
#pragma once
#include <cuda_runtime.h>

namespace tnfa {
namespace la {

// 1 / sqrt(x) to FP64 for x in [1, 2]: FP32 root, one third-order Newton step
// (y e (1/2 + 3/8 e), e = 1 - x y^2: the error term is e^3).
__device__ __forceinline__ double rsqrt_1_2(double x) {
  const double y = (double)rsqrtf((float)x);
  const double e = fma(-x * y, y, 1.0);
  return fma(y * e, fma(e, 0.375, 0.5), y);
}

// sqrt(x), and 1 / (sqrt(x) (sqrt(x) + |y|)), for a normal x > 0: FP32 starts
// on the mantissas, third-order Newton for the root, two Newton steps for the
// reciprocal (an FP64 division or root is some 20 operations on the slow pipe).
__device__ __forceinline__ void root_and_beta(double x, double y, double& nrm, double& beta) {
  const int e = (((int)(__double2hiint(x) >> 20) - 1023) & ~1);  // even: x = X 2^e, X in [1, 4)
  const double X = x * __hiloint2double((1023 - e) << 20, 0);
  double r = (double)rsqrtf((float)X);
  const double f = fma(-X * r, r, 1.0);
  r = fma(r * f, fma(f, 0.375, 0.5), r);
  double s = X * r;
  s = fma(0.5 * r, fma(-s, s, X), s);  // one correction of the root itself
  const double half = __hiloint2double((1023 + e / 2) << 20, 0), inv = __hiloint2double((1023 - e / 2) << 20, 0);
  nrm = s * half;
  const double d = s + fabs(y) * inv;  // in [1, 4): |y| <= sqrt(x)
  double q = (double)(1.0f / (float)d);
  q = fma(q, fma(-d, q, 1.0), q);
  q = fma(q, fma(-d, q, 1.0), q);
  beta = r * q * inv * inv;
}

}  // namespace la
}  // namespace tnfa
