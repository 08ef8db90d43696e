// The FP64 roots of roots.cuh against CUDA's over their ranges: x in [1, 2] for
// rsqrt_1_2; x from 1e-300 to 1e300, |y| <= sqrt(x), for root_and_beta, the ends
// of every binade and y = 0, +-sqrt(x) among them.  FP32's root leaves less than
// 2^-21, so the third-order step 2^-63, and two roundings: 3 u of u = 2^-53.
// beta has the root twice, the reciprocal's step and four products, CUDA's form
// three roundings: 12 u.
#include <cstdio>
#include <cmath>

#include "roots.cuh"

__device__ double rel(double a, double b) { return fabs(a - b) / fabs(b); }
__device__ unsigned long long mix(unsigned long long z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__device__ double unit(unsigned long long z) { return (double)(mix(z) >> 11) * 0x1p-53; }

__global__ void check(int n, unsigned long long* worst) {
  double w[3] = {0, 0, 0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double x = i < 64 ? 1.0 + i * 0x1p-52 : i < 128 ? 2.0 - (i - 64) * 0x1p-52 : 1.0 + unit(3ull * i);
    w[0] = fmax(w[0], rel(tnfa::la::rsqrt_1_2(x), 1.0 / sqrt(x)));
    double z = pow(10.0, 600.0 * unit(3ull * i + 1) - 300.0);
    if (i % 8 == 0) z = __longlong_as_double((__double_as_longlong(z) & 0x7FF0000000000000ll) | (i % 16 ? 0xFFFFFFFFFFFFFll : 0));
    const double s = sqrt(z), t = unit(3ull * i + 2), y = i % 5 == 0 ? 0.0 : i % 5 == 1 ? s : i % 5 == 2 ? -s : (2 * t - 1) * s;
    double nrm, beta;
    tnfa::la::root_and_beta(z, y, nrm, beta);
    w[1] = fmax(w[1], rel(nrm, s));
    w[2] = fmax(w[2], rel(beta, 1.0 / (s * (s + fabs(y)))));
  }
  for (int k = 0; k < 3; ++k) atomicMax(worst + k, (unsigned long long)__double_as_longlong(w[k]));
}

int main() {
  unsigned long long* d = nullptr;
  double h[3] = {1, 1, 1};
  if (cudaMalloc(&d, sizeof h) != cudaSuccess || cudaMemset(d, 0, sizeof h) != cudaSuccess) return 2;
  check<<<304, 256>>>(1 << 24, d);
  if (cudaMemcpy(h, d, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  cudaFree(d);
  const double u = 0x1p-53;
  printf("%.3g %.3g %.3g\n", h[0] / u, h[1] / u, h[2] / u);
  return h[0] <= 3 * u && h[1] <= 3 * u && h[2] <= 12 * u ? 0 : 1;
}
